"""Up to sixteen rows over row-major packed weights (kq_qgemv_rows.cu): every storage, activation type and number of
rows at the edges of its steps, groups of threads and passes, against the f64 oracle; a value's arithmetic is an f32
multiply and multiply-adds, sixteen to a chain, so 1e-5 of the result's rms and 1e-4 relative hold with a wide margin.
The smallest shapes stay on the generic kernel (kq_rows_line.h), in one launch as well."""
import numpy as np
import pytest

import oracle
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import karume_b200 as kb
    g = kb.acquire_gpu(0)
    yield g
    g.destroy()


# (storage, group, n, k): one step and a ragged number of them, one channel and odd numbers, groups of sixteen (two to a
# step) up to a whole row, few channels (256 threads to a pair) and many (four)
SHAPES = [("i4", 32, 1, 32), ("i4", 16, 33, 96), ("i4", 64, 130, 320), ("i4", 128, 257, 1152), ("i4", 4096, 50, 4096), ("i4", 32, 30001, 64),
          ("i8", 0, 1, 16), ("i8", 0, 131, 80), ("i8", 0, 17, 8176), ("i8", 0, 20011, 48)]


@pytest.mark.parametrize("xdt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("m", [1, 2, 3, 5, 16])
@pytest.mark.parametrize("storage,group,n,k", SHAPES)
def test_matches_the_f64_oracle(gpu, storage, group, n, k, m, xdt):
    import torch
    rng = np.random.default_rng(n + m)
    x = rng.standard_normal((m, k)).astype(np.float32)
    if xdt == "f32":
        x[m // 2] *= np.float32(1e30)  # a row of another magnitude
    x = {"f32": lambda v: v, "f16": oracle.round_to_f16, "bf16": oracle.round_to_bf16}[xdt](x)
    bias = rng.standard_normal(n).astype(np.float32)
    if storage == "i4":
        data, scale = cases.synth_i4(n, k, seed=n, group_size=group, scale_dtype="f32" if m % 2 else "f16")
        ref = oracle.linear_i4(x, data, scale.astype(np.float32), bias, n, k, group)
    else:
        data, scale = cases.synth_i8(n, k, seed=n)
        ref = oracle.linear_i8(x, data, scale.astype(np.float32), bias, n, k)
    w = gpu.upload_weight(storage, data, scale, (n, k), group)
    xd = torch.from_numpy(x).cuda().to({"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[xdt])
    out = torch.full((m + 1, n), float("nan"), device="cuda")
    bd = torch.from_numpy(bias).cuda()
    torch.cuda.synchronize()
    before = gpu.launch_count
    gpu.linear(xd, w, bd, out=out[:m])
    gpu.sync()
    assert gpu.launch_count - before == 1
    got = out[:m].cpu().numpy()
    assert bool(torch.isnan(out[m]).all())
    for r in range(m):
        rms = float(np.sqrt(np.mean(ref[r].astype(np.float64) ** 2)))
        rep = oracle.allclose(got[r], ref[r], atol=1e-5 * max(1.0, rms), rtol=1e-4)
        assert rep["pass"], (r, rep)
    w.free()


# Groups of sixteen, two scales to a step, and odd channel counts on rows long enough for this kernel
@pytest.mark.parametrize("xdt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("m", [1, 2, 3, 5, 16])
@pytest.mark.parametrize("storage,group,n,k", [("i4", 16, 35, 4128), ("i4", 64, 1, 8192), ("i8", 0, 3, 8208)])
def test_long_rows_of_few_channels(gpu, storage, group, n, k, m, xdt):
    test_matches_the_f64_oracle(gpu, storage, group, n, k, m, xdt)


@pytest.mark.parametrize("k", [96, 4128])
def test_infinities_and_nans_reach_their_channels(gpu, k):
    import torch
    n = 35
    data, scale = cases.synth_i4(n, k, seed=1, group_size=16)
    w = gpu.upload_weight("i4", data, scale, (n, k), 16)
    x = np.zeros((2, k), np.float32)
    x[0, 5], x[1, 70] = np.inf, np.nan
    out = gpu.linear(torch.from_numpy(x).cuda(), w, torch.zeros(n, device="cuda"))
    gpu.sync()
    weights = oracle.decode_i4(data, (n, k), scale.astype(np.float32), (n, k // 16), 16)
    with np.errstate(invalid="ignore"):
        want = np.where(weights[:, 5] == 0, np.nan, np.sign(weights[:, 5]) * np.inf)
    got = out.cpu().numpy()
    assert np.array_equal(got[0], want.astype(np.float32), equal_nan=True)
    assert bool(np.isnan(got[1]).all())
    w.free()


# The norm and the residual go into the linear's own launch and need no scratch, so the first call of a context may be a
# recorded one: rows that take this kernel (one and two rows to a CTA, four, several passes) and some that take the
# many-row kernel.
@pytest.mark.parametrize("neighbours", ["norm", "residual", "both"])
@pytest.mark.parametrize("storage,group,m,n,k", [("i4", 64, 1, 4097, 4096), ("i4", 16, 2, 3001, 4224), ("i8", 0, 1, 3001, 2800), ("i4", 128, 3, 1000, 12288),
                                                 ("i8", 0, 16, 82, 8064), ("i4", 64, 16, 250, 8192), ("i4", 64, 16, 8191, 768), ("i8", 0, 9, 9001, 1152)])
def test_norm_and_residual_in_a_first_call_that_is_recorded(storage, group, m, n, k, neighbours):
    import torch
    import karume_b200 as kb
    rng = np.random.default_rng(n)
    x, bias, res = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (n,), (m, n)))
    norm = (1 + 0.1 * rng.standard_normal(k)).astype(np.float32)
    xn = x if neighbours == "residual" else oracle.rms_norm(x, norm, 1e-5)
    if storage == "i4":
        data, scale = cases.synth_i4(n, k, seed=n, group_size=group)
        ref = oracle.linear_i4(xn, data, scale.astype(np.float32), bias, n, k, group)
    else:
        data, scale = cases.synth_i8(n, k, seed=n)
        ref = oracle.linear_i8(xn, data, scale.astype(np.float32), bias, n, k)
    if neighbours != "norm":
        ref = oracle.add(ref, res)
    fresh = kb.acquire_gpu(0)
    fresh.use_stream(torch.cuda.Stream())
    w = fresh.upload_weight(storage, data, scale, (n, k), group)
    xd, bd, nd, out = (torch.from_numpy(a).cuda() for a in (x, bias, norm, res))  # the residual is the output buffer
    kept = out.clone()
    torch.cuda.synchronize()
    fresh.graph_begin()
    fresh.linear_fused(xd, [w], [bd], [out], norm_weight=None if neighbours == "residual" else nd, eps=1e-5 if neighbours != "residual" else 0.0,
                       residual=None if neighbours == "norm" else out)
    g = fresh.graph_end()
    rms = float(np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    for _ in range(2):
        out.copy_(kept)
        torch.cuda.synchronize()
        fresh.graph_launch(g)
        fresh.sync()
        rep = oracle.allclose(out.cpu().numpy(), ref, atol=1e-5 * max(1.0, rms), rtol=1e-4)
        assert rep["pass"], rep
    fresh.graph_free(g)
    w.free()
    fresh.destroy()
