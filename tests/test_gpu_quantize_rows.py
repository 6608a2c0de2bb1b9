"""The row quantiser at the edges of its row widths and on values at and beside rounding ties: bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [1, 4, 1023, 1024, 1028, 2048, 2052, 4096, 4100, 8192, 8196, 16384, 16388])
def test_rows_of_every_width_with_ties(dim):
    import torch
    import karume_b200 as kb
    gpu = kb.acquire_gpu(0)
    rng = np.random.default_rng(dim)
    x = rng.standard_normal((9, dim)).astype(np.float32) * np.float32([[1], [3], [1e30], [1e-30], [1e-38], [1e-44], [0], [127], [1]])
    half = (rng.integers(-254, 255, dim) / 2).astype(np.float32)  # quotients on ties, and one ulp to either side
    x[7] = np.nextafter(half, np.float32(np.inf) * rng.choice([-1, 1], dim).astype(np.float32)) if dim > 4 else half
    x[8] = half
    x[7:, 0] = 127.0
    if dim > 1:
        x[1, 1] = np.inf
    t = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    q, s = gpu.quantize_rows(t)
    gpu.sync()
    want_q, want_s = oracle.quantize_rows(x, *x.shape)
    assert np.array_equal(s.cpu().numpy().view(np.uint32), want_s.view(np.uint32))
    finite = np.isfinite(x).all(axis=1)
    assert np.array_equal(q.cpu().numpy()[finite], want_q[finite])
    gpu.destroy()
