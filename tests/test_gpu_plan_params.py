"""Plans whose ops write the bias and the norm weight of a later op: those are read after the barrier, all
others ahead of it."""
import numpy as np
import pytest

import oracle
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k", [(1, 256), (1, 192), (2, 256)])
@pytest.mark.parametrize("written", ["none", "bias", "norm"])
def test_parameters_written_by_the_plan(m, k, written):
    import torch
    import karume_b200 as kb
    gpu = kb.acquire_gpu(0)
    rng = np.random.default_rng(m * k)
    n = k  # of the op whose outputs serve as parameters
    x = rng.standard_normal((m, k)).astype(np.float32)
    (d0, s0), (d1, s1) = cases.synth_i4(n, k, seed=1), cases.synth_i4(n, k, seed=2)
    b0 = (5 + rng.standard_normal(n)).astype(np.float32)
    w0, w1 = (gpu.upload_weight("i4", d, s, (n, k), 32) for d, s in ((d0, s0), (d1, s1)))
    bias, norm = rng.standard_normal(n).astype(np.float32), (1 + 0.1 * rng.standard_normal(k)).astype(np.float32)
    dev = lambda a: torch.from_numpy(a).cuda()
    xd, b0d, biasd, normd = dev(x), dev(b0), dev(bias), dev(norm)
    first, out = torch.zeros(m, n, device="cuda"), torch.zeros(m, n, device="cuda")
    torch.cuda.synchronize()
    gpu.plan_begin()
    gpu.linear_fused(xd, [w0], [b0d], [first])
    gpu.linear_fused(xd, [w1], [first[0] if written == "bias" else biasd], [out],
                     norm_weight=first[0] if written == "norm" else normd, eps=1e-5)
    plan = gpu.plan_end()
    y0 = oracle.linear_i4(x, d0, s0.astype(np.float32), b0, n, k, 32)
    if written == "bias":
        bias = y0[0].astype(np.float32)
    if written == "norm":
        norm = y0[0].astype(np.float32)
    ref = oracle.linear_i4(oracle.rms_norm(x, norm, 1e-5), d1, s1.astype(np.float32), bias, n, k, 32)
    rms = float(np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    for _ in range(2):  # the second launch would find the first one's values if it read too early
        first.fill_(float("nan"))
        torch.cuda.synchronize()
        gpu.plan_launch(plan)
        gpu.sync()
        rep = oracle.allclose(out.cpu().numpy(), ref, atol=1e-5 * max(1.0, rms), rtol=1e-3)
        assert rep["pass"], rep
    gpu.plan_free(plan)
    for w in (w0, w1):
        w.free()
    gpu.destroy()
