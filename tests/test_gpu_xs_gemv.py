"""The decode linear with the activations in registers (kq_qgemv_i4_xs.cu): row counts at the edges of
its column forms, k at the edges of a warp's slab, a CTA's slabs, a cluster's and a second pass, several weights in
one launch, with and without the neighbours of a decoder layer, against the oracle."""
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


def dev(a):
    import torch
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    torch.cuda.synchronize()
    return t


def check(got, ref):
    rms = float(np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    rep = oracle.allclose(got.cpu().numpy(), ref, atol=1e-5 * max(1.0, rms), rtol=1e-3)
    assert rep["pass"], rep


@pytest.mark.parametrize("xdt,m", [("f32", 3), ("f32", 4), ("f32", 5), ("f32", 8), ("f32", 9), ("f32", 16), ("bf16", 4), ("bf16", 13),
                                   ("f16", 5), ("f16", 8), ("f16", 16)])
@pytest.mark.parametrize("n,k", [(16, 64), (48, 192), (272, 2048), (80, 2112), (32, 16448)])
def test_rows_and_k_at_the_edges(gpu, xdt, m, n, k):
    import torch
    rng = np.random.default_rng(m * k)
    rnd = {"f32": lambda v: v, "f16": oracle.round_to_f16, "bf16": oracle.round_to_bf16}[xdt]
    x = rnd(rng.standard_normal((m, k)).astype(np.float32))
    data, scale = cases.synth_i4(n, k, seed=n + m, scale_dtype="f32" if m % 2 else "f16")
    bias = rng.standard_normal(n).astype(np.float32)
    w = gpu.upload_weight("i4", data, scale, (n, k), 32)
    out = torch.full((m, n), float("nan"), device="cuda")
    xd = dev(x).to({"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[xdt])
    torch.cuda.synchronize()
    gpu.linear(xd, w, dev(bias), out=out)
    gpu.sync()
    check(out, oracle.linear_i4(x, data, scale.astype(np.float32), bias, n, k, 32))
    again = gpu.linear(xd, w, dev(bias))
    gpu.sync()
    assert torch.equal(out, again)
    w.free()


@pytest.mark.parametrize("m", [1, 2, 4, 7, 16])
@pytest.mark.parametrize("k", [128, 4096])
def test_neighbours_in_the_same_launch(gpu, m, k):
    rng = np.random.default_rng(m + k)
    ns = [4096, 32, 1040]
    x = rng.standard_normal((m, k)).astype(np.float32) * np.float32(3.0)
    g = (1 + 0.1 * rng.standard_normal(k)).astype(np.float32)
    xn = oracle.rms_norm(x, g, 1e-5)
    ws, refs, biases = [], [], []
    for i, n in enumerate(ns + [ns[2]]):
        data, scale = cases.synth_i4(n, k, seed=i + 5)
        b = rng.standard_normal(n).astype(np.float32)
        ws.append(gpu.upload_weight("i4", data, scale, (n, k), 32))
        biases.append(dev(b))
        refs.append(oracle.linear_i4(xn, data, scale.astype(np.float32), b, n, k, 32))
    res = rng.standard_normal((m, ns[2])).astype(np.float32)
    before = gpu.launch_count
    xd, gd = dev(x), dev(g)
    outs = [dev(np.zeros((m, n), np.float32)) for n in ns]
    gpu.linear_fused(xd, ws[:3], biases[:3], outs, norm_weight=gd, eps=1e-5)
    (act,) = gpu.linear_fused(xd, ws[2:], biases[2:], norm_weight=gd, eps=1e-5, swiglu=True)
    hidden = dev(res)  # the residual is the output buffer
    gpu.linear_fused(xd, [ws[2]], [biases[2]], [hidden], norm_weight=gd, eps=1e-5, residual=hidden)
    gpu.sync()
    assert gpu.launch_count - before == 3
    for got, ref in zip(outs, refs):
        check(got, ref)
    check(act, oracle.silu_mul(refs[2], refs[3]))
    check(hidden, oracle.add(refs[2], res))
    for w in ws:
        w.free()
