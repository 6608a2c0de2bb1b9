"""The many-row linear with weights as exact integers (kq_qgemm_exact.cu): every packed layout,
activation type and accumulator-chain length at the edges of its tiles, against the f64 oracle;
the integer-dot form bit for bit."""
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


# (storage, group, m, n, k): one and several row tiles, ragged rows and channels, k tails of half a
# k-step, groups of one k16 slice up to longer than an accumulator chain, K slices
SHAPES = [("i4", 32, 17, 16, 64), ("i4", 32, 257, 272, 512), ("i4", 32, 40, 130, 96), ("i4", 16, 65, 304, 1152),
          ("i4", 64, 33, 250, 320), ("i4", 128, 300, 512, 4096), ("i4", 2048, 18, 144, 4096), ("i8", 0, 40, 64, 96),
          ("i8", 0, 257, 512, 1536), ("i8", 0, 66, 131, 80), ("i8", 0, 600, 784, 4096),
          # a few rows of an untiled weight, on both sides of the amount of work that brings them here
          ("i4", 64, 1, 3072, 4096), ("i4", 16, 3, 1001, 4224), ("i4", 128, 16, 250, 256), ("i8", 0, 2, 1501, 2800)]


@pytest.mark.parametrize("xdt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("storage,group,m,n,k", SHAPES)
def test_matches_the_f64_oracle(gpu, xdt, storage, group, m, n, k):
    import torch
    if xdt == "bf16" and n % 16 == 0 and k % 64 == 0 and group in (0, 32):
        pytest.skip("the bf16 GEMM's case")
    rng = np.random.default_rng(m + n)
    x = rng.standard_normal((m, k)).astype(np.float32)
    x[m // 2] *= np.float32(1e30) if xdt != "f16" else np.float32(1e3)  # a row of another magnitude
    x[m - 1] *= np.float32(1e-30) if xdt != "f16" else np.float32(1e-3)
    x = {"f32": lambda v: v, "f16": oracle.round_to_f16, "bf16": oracle.round_to_bf16}[xdt](x)
    bias = rng.standard_normal(n).astype(np.float32)
    bias[n // 2:] = 0.0
    if storage == "i4":
        data, scale = cases.synth_i4(n, k, seed=n, group_size=group, scale_dtype="f32" if m % 2 else "f16")
        ref = oracle.linear_i4(x, data, scale.astype(np.float32), bias, n, k, group)
    else:
        data, scale = cases.synth_i8(n, k, seed=n)
        ref = oracle.linear_i8(x, data, scale.astype(np.float32), bias, n, k)
    w = gpu.upload_weight(storage, data, scale, (n, k), group)
    xd = dev(x).to({"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[xdt])
    out = torch.full((m, n), float("nan"), device="cuda")
    torch.cuda.synchronize()
    gpu.linear(xd, w, dev(bias), out=out)
    gpu.sync()
    got = out.cpu().numpy()
    for rows in (slice(m // 2, m // 2 + 1), slice(m - 1, m), np.setdiff1d(np.arange(m), [m // 2, m - 1])):
        if ref[rows].size == 0:
            continue
        rms = float(np.sqrt(np.mean(ref[rows].astype(np.float64) ** 2)))
        rep = oracle.allclose(got[rows], ref[rows], atol=1e-5 * max(1.0, rms), rtol=1e-4)
        assert rep["pass"], rep
    again = gpu.linear(xd, w, dev(bias))
    gpu.sync()
    assert torch.equal(out, again)
    w.free()


@pytest.mark.parametrize("storage,group,m,n,k", [s for s in SHAPES if s[1] <= 1024] + [("i4", 16, 129, 67, 48), ("i8", 0, 300, 528, 8960),
                         # few rows, on both sides of the lines between this kernel and the mma.sync one
                         ("i8", 0, 3, 64, 32), ("i8", 0, 8, 49152, 96), ("i8", 0, 8, 49168, 96), ("i8", 0, 16, 49168, 448), ("i8", 0, 16, 49168, 512),
                         ("i4", 32, 8, 144, 512), ("i4", 32, 1, 18944, 64), ("i4", 32, 8, 18960, 64), ("i4", 32, 16, 49168, 448), ("i4", 32, 16, 49168, 512)])
def test_integer_dot_is_bit_exact(gpu, storage, group, m, n, k):
    rng = np.random.default_rng(m)
    x = rng.standard_normal((m, k)).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    if storage == "i4":
        data, scale = cases.synth_i4(n, k, seed=n, group_size=group, scale_dtype="f32" if m % 2 else "f16")
        u = np.stack([data & 15, data >> 4], axis=1).reshape(n, k).astype(np.int16) - 8
        want = oracle.linear_w4a8(x, u.astype(np.int8), scale.astype(np.float32), bias, group)
    else:
        data, scale = cases.synth_i8(n, k, seed=n)
        want = oracle.linear_w8a8(x, data, scale.astype(np.float32), bias)
    w = gpu.upload_weight(storage, data, scale, (n, k), group)
    xq, xs = gpu.quantize_rows(dev(x))
    out = gpu.linear_a8(xq, xs, w, dev(bias))
    gpu.sync()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), np.asarray(want, np.float32).view(np.uint32))
    w.free()


# K slices that meet in a cluster (two or four, the last one short), next to ragged channels and rows, on tiles of 32 and 64 rows
@pytest.mark.parametrize("xdt", ["f32", "f16"])
@pytest.mark.parametrize("storage,group,m,n,k", [("i4", 32, 20, 272, 576), ("i4", 16, 33, 100, 1152), ("i4", 128, 97, 513, 1408),
                                                 ("i4", 32, 160, 1040, 1088), ("i4", 32, 223, 528, 960), ("i8", 0, 50, 300, 1616),
                                                 ("i8", 0, 225, 1008, 1120)])
def test_slices_that_meet_in_a_cluster(gpu, xdt, storage, group, m, n, k):
    test_matches_the_f64_oracle(gpu, xdt, storage, group, m, n, k)


# Rows whose values stay in the splitting kernel's registers (2,048 a unit, up to eight units), and one beyond that
@pytest.mark.parametrize("m,n,k", [(17, 40, 2048), (18, 40, 2064), (17, 40, 4112), (17, 24, 16384), (18, 24, 16400)])
def test_rows_of_any_length_are_split(gpu, m, n, k):
    test_matches_the_f64_oracle(gpu, "f32", "i8", 0, m, n, k)


@pytest.mark.parametrize("m,n,k", [(20, 272, 4096), (150, 528, 2176), (97, 259, 1136)])
def test_integer_sums_that_meet_in_a_cluster(gpu, m, n, k):
    test_integer_dot_is_bit_exact(gpu, "i8", 0, m, n, k)


# ... and on tiles of 32 to 256 rows; no launch adds the slices
@pytest.mark.parametrize("xdt,storage,group,m,n,k,nt,slices", [s for s in cases.EXACT_SLICED if s[0] != "i8"])
def test_slices_of_wide_tiles_meet_in_a_cluster(gpu, xdt, storage, group, m, n, k, nt, slices):
    before = gpu.launch_count
    test_matches_the_f64_oracle(gpu, xdt, storage, group, m, n, k)
    repacked = 1 if group in (0, 32) and n % 16 == 0 and k % (32 if storage == "i8" else 64) == 0 else 0
    assert gpu.launch_count - before - repacked == 2 * (1 if xdt == "f16" else 2)


def test_residual_and_several_weights_of_slices_in_a_cluster(gpu):
    import torch
    rng = np.random.default_rng(5)
    xdt, storage, group, m, n, k, _, _ = cases.EXACT_SLICED[3]
    x, res = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((m, n)).astype(np.float32)
    norm, bias = (1 + 0.1 * rng.standard_normal(k)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    data, scale = cases.synth_i4(n, k, seed=n)
    w = gpu.upload_weight(storage, data, scale, (n, k), group)
    out = dev(res)  # the residual is the output buffer
    before = gpu.launch_count
    gpu.linear_fused(dev(x), [w], [dev(bias)], [out], norm_weight=dev(norm), eps=1e-5, residual=out)
    gpu.sync()
    assert gpu.launch_count - before == 2
    want = oracle.add(oracle.linear_i4(oracle.rms_norm(x, norm, 1e-5), data, scale.astype(np.float32), bias, n, k, group), res)
    rep = oracle.allclose(out.cpu().numpy(), want, atol=1e-5 * float(np.sqrt(np.mean(want.astype(np.float64) ** 2))), rtol=1e-4)
    assert rep["pass"], rep
    w.free()
    # 512, 256 and 272 channels are the column pairs of the 1,040 of this case
    xdt, storage, group, m, n, k, _, _ = cases.EXACT_SLICED[1]
    x = oracle.round_to_f16(rng.standard_normal((m, k)).astype(np.float32))
    ws, biases, wants = [], [], []
    for each in (512, 256, n - 768):
        data, scale = cases.synth_i4(each, k, seed=each)
        ws.append(gpu.upload_weight(storage, data, scale, (each, k), group))
        biases.append(rng.standard_normal(each).astype(np.float32))
        wants.append(oracle.linear_i4(x, data, scale.astype(np.float32), biases[-1], each, k, group))
    before = gpu.launch_count
    outs = gpu.linear_multi(dev(x).to(torch.float16), ws, [dev(b) for b in biases])
    gpu.sync()
    assert gpu.launch_count - before == 1
    for got, want in zip(outs, wants):
        rep = oracle.allclose(got.cpu().numpy(), want, atol=1e-5 * max(1.0, float(np.sqrt(np.mean(want.astype(np.float64) ** 2)))), rtol=1e-4)
        assert rep["pass"], rep
    for w in ws:
        w.free()


@pytest.mark.parametrize("m,n,k,nt,slices", [s[3:] for s in cases.EXACT_SLICED if s[0] == "i8"])
def test_integer_sums_of_wide_tiles_meet_in_a_cluster(gpu, m, n, k, nt, slices):
    before = gpu.launch_count
    test_integer_dot_is_bit_exact(gpu, "i8", 0, m, n, k)
    assert gpu.launch_count - before == 3  # the weight's repacking, the quantiser, the matmul


# A resident pair takes several tiles in turn: bit for bit on every channel of the rows at the edges of the row tiles (of the
# multiples of 32 that they may have)
@pytest.mark.parametrize("m,n,k", cases.EXACT_RESIDENT)
def test_several_tiles_to_a_pair_are_bit_exact(gpu, m, n, k):
    rng = np.random.default_rng(m)
    x = rng.standard_normal((m, k)).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    data, scale = cases.synth_i8(n, k, seed=n)
    rows = sorted({r for edge in range(0, m + 32, 32) for r in (edge - 1, edge) if 0 <= r < m} | {m - 1})
    want = np.asarray(oracle.linear_w8a8(x[rows], data, scale.astype(np.float32), bias), np.float32)
    w = gpu.upload_weight("i8", data, scale, (n, k), 0)
    xq, xs = gpu.quantize_rows(dev(x))
    outs = [gpu.linear_a8(xq, xs, w, dev(bias)) for _ in range(2)]
    gpu.sync()
    got = outs[0].cpu().numpy()
    assert np.array_equal(got[rows].view(np.uint32), want.view(np.uint32))
    assert np.array_equal(got.view(np.uint32), outs[1].cpu().numpy().view(np.uint32))
    w.free()


def test_every_form_behind_the_other_in_a_recording(gpu):
    """Launches that overlap (each starts while the one before ends) replay with the bits of the same calls one at a time: a
    gated pair, slices in a cluster that read its output, several tiles to a pair, and few rows over row-major weights."""
    import torch
    rng = np.random.default_rng(9)
    m, k, n, n8 = 300, 256, 4752, 9488
    gate, up = (gpu.upload_weight("i4", *cases.synth_i4(n, k, seed=s), (n, k), 32) for s in (1, 2))
    w8 = gpu.upload_weight("i8", *cases.synth_i8(n8, n, seed=3), (n8, n), 0)
    down = gpu.upload_weight("i4", *cases.synth_i4(1056, n, seed=4, group_size=16), (1056, n), 16)
    few = gpu.upload_weight("i4", *cases.synth_i4(4097, 1056, seed=5, group_size=16), (4097, 1056), 16)
    x, norm = dev(rng.standard_normal((m, k)).astype(np.float32)), dev((1 + 0.1 * rng.standard_normal(k)).astype(np.float32))
    zero = torch.zeros(16384, device="cuda")
    xq, xs = gpu.quantize_rows(dev(rng.standard_normal((m, n)).astype(np.float32)))
    gpu.sync()

    def step(into, fence):
        act, y, z, last = into
        gpu.linear_fused(x, [gate, up], [zero[:n], zero[:n]], [act], norm_weight=norm, eps=1e-5, swiglu=True)
        fence()
        gpu.linear(act, down, zero[:1056], out=y)
        fence()
        gpu.linear_a8(xq, xs, w8, zero[:n8], out=z)
        fence()
        gpu.linear(y[:3], few, zero[:4097], out=last)
        fence()

    def outputs():
        return [torch.zeros(s, device="cuda") for s in ((m, n), (m, 1056), (m, n8), (3, 4097))]

    stream = torch.cuda.Stream()
    gpu.use_stream(stream)
    gpu.set_overlap(True)
    try:
        with torch.cuda.stream(stream):
            want, got = outputs(), outputs()
            torch.cuda.synchronize()
            step(want, gpu.sync)
            step(got, lambda: None)
            gpu.sync()
            assert all(torch.equal(a, b) for a, b in zip(want, got))
            gpu.graph_begin()
            step(got, lambda: None)
            g = gpu.graph_end()
            for _ in range(3):
                for t in got:
                    t.zero_()
                gpu.graph_launch(g)
                gpu.sync()
                assert all(torch.equal(a, b) for a, b in zip(want, got))
            gpu.graph_free(g)
    finally:
        gpu.use_stream(torch.cuda.current_stream())
    for w in (gate, up, w8, down, few):
        w.free()


# The gate in the matmul's epilogue (its tiles fill half of the device): ragged rows and channels, every storage; out on top
# of x takes the separate kernels
@pytest.mark.parametrize("storage,group,xdt,m,n,k", [("i4", 32, "f32", 513, 2416, 128), ("i4", 32, "f16", 300, 4752, 64), ("i4", 16, "f32", 270, 2401, 96),
                                                     ("i8", 0, "f32", 257, 4736, 96), ("i8", 0, "f16", 800, 2440, 80), ("i4", 64, "bf16", 1030, 3333, 192)])
def test_gate_in_the_epilogue(gpu, storage, group, xdt, m, n, k):
    import torch
    rng = np.random.default_rng(m)
    x = {"f32": lambda v: v, "f16": oracle.round_to_f16, "bf16": oracle.round_to_bf16}[xdt](rng.standard_normal((m, k)).astype(np.float32))
    norm = (1 + 0.1 * rng.standard_normal(k)).astype(np.float32) if xdt == "f32" else None
    xn = oracle.rms_norm(x, norm, 1e-5) if xdt == "f32" else x
    ws, biases, refs = [], [], []
    for seed in (1, 2):
        data, scale = cases.synth_i4(n, k, seed=seed, group_size=group) if storage == "i4" else cases.synth_i8(n, k, seed=seed)
        ws.append(gpu.upload_weight(storage, data, scale, (n, k), group))
        biases.append(rng.standard_normal(n).astype(np.float32))
        args = (xn, data, scale.astype(np.float32), biases[-1], n, k)
        refs.append(oracle.linear_i4(*args, group) if storage == "i4" else oracle.linear_i8(*args))
    want = (refs[0] / (1 + np.exp(-refs[0].astype(np.float64))) * refs[1]).astype(np.float32)
    xd = dev(x).to({"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[xdt])
    out = torch.full((m, n), float("nan"), device="cuda")
    torch.cuda.synchronize()
    before = gpu.launch_count
    gpu.linear_fused(xd, ws, [dev(b) for b in biases], [out], norm_weight=dev(norm) if norm is not None else None, eps=1e-5, swiglu=True)
    gpu.sync()
    assert gpu.launch_count - before == (1 if xdt == "f16" else 2)
    rms = float(np.sqrt(np.mean(want.astype(np.float64) ** 2)))
    rep = oracle.allclose(out.cpu().numpy(), want, atol=1e-5 * max(1.0, rms), rtol=1e-4)
    assert rep["pass"], rep
    over = torch.zeros(m * max(n, k), device="cuda")  # x and out share their first bytes
    xo = over.view(xd.dtype)[: m * k].view(m, k)
    xo.copy_(xd)
    torch.cuda.synchronize()
    gpu.linear_fused(xo, ws, [dev(b) for b in biases], [over[: m * n].view(m, n)], norm_weight=dev(norm) if norm is not None else None, eps=1e-5, swiglu=True)
    gpu.sync()
    rep = oracle.allclose(over[: m * n].view(m, n).cpu().numpy(), want, atol=1e-5 * max(1.0, rms), rtol=1e-4)
    assert rep["pass"], rep
    for w in ws:
        w.free()


@pytest.mark.parametrize("m,n,k", [(17, 64, 128), (130, 544, 1536)])
def test_norm_gate_and_residual_around_it(gpu, m, n, k):
    import torch
    rng = np.random.default_rng(k)
    x = rng.standard_normal((m, k)).astype(np.float32)
    g = (1 + 0.1 * rng.standard_normal(k)).astype(np.float32)
    ws, refs = [], []
    xn = oracle.rms_norm(x, g, 1e-5)
    zero = np.zeros(n, np.float32)
    for s in (1, 2):
        data, scale = cases.synth_i4(n, k, seed=s)
        ws.append(gpu.upload_weight("i4", data, scale, (n, k), 32))
        refs.append(oracle.linear_i4(xn, data, scale.astype(np.float32), zero, n, k, 32))
    bias = dev(zero)
    res = rng.standard_normal((m, n)).astype(np.float32)
    (act,) = gpu.linear_fused(dev(x), ws, [bias, bias], norm_weight=dev(g), eps=1e-5, swiglu=True)
    (added,) = gpu.linear_fused(dev(x), ws[:1], [bias], norm_weight=dev(g), eps=1e-5, residual=dev(res))
    both = gpu.linear_multi(dev(xn), ws, [bias, bias])
    gpu.sync()
    for got, want in ((act, oracle.silu_mul(refs[0], refs[1])), (added, oracle.add(refs[0], res)), (both[0], refs[0]), (both[1], refs[1])):
        rep = oracle.allclose(got.cpu().numpy(), want, atol=1e-5, rtol=1e-3)
        assert rep["pass"], rep
    for w in ws:
        w.free()


# Magnitudes that lie side by side in k: an f32 multiply-add gives a channel the sum of its own products
# whatever else the row holds, so no value may be resolved relative to a larger one of its row.
DECADES = (1e-9, 1.0, 1e9)


@pytest.mark.parametrize("xdt", ["f32", "bf16"])
@pytest.mark.parametrize("storage,group,m,n,k", [("i4", 32, 40, 144, 512), ("i4", 32, 300, 528, 2048), ("i4", 16, 65, 301, 1152), ("i4", 2048, 18, 202, 4096),
                                                 ("i8", 0, 33, 330, 2800), ("i8", 0, 257, 130, 1536), ("i8", 0, 40, 144, 1056), ("i4", 64, 3, 3000, 4096)])
def test_channels_that_only_see_the_small_values_of_a_row(gpu, xdt, storage, group, m, n, k):
    """Channel c has weights only where k % 3 == c % 3, and those activations are 1e-9, 1 or 1e9 times
    N(0, 1).  Each third of the channels has to meet the tolerance on its own scale: f32 sums of up to
    4096 / 3 terms, 1e-5 of their rms (sqrt(k) 2^-24 is 4e-6) and 1e-4 relative."""
    import torch
    rng = np.random.default_rng(m + n)
    which = np.arange(k) % 3
    x = rng.standard_normal((m, k)).astype(np.float32) * np.asarray(DECADES, np.float32)[which]
    x = {"f32": lambda v: v, "bf16": oracle.round_to_bf16}[xdt](x)
    live = which[None, :] == (np.arange(n) % 3)[:, None]
    bias = np.zeros(n, np.float32)
    if storage == "i4":
        if xdt == "bf16" and group == 32:
            pytest.skip("the bf16 GEMM's case")
        nibbles = np.where(live, rng.integers(0, 16, size=(n, k)), 8).astype(np.uint8)
        data = cases.pack_nibbles(nibbles.reshape(-1))
        scale = (np.abs(rng.standard_normal((n, k // group))) * 0.02 / 7 + 1e-6).astype(np.float32)
        ref = oracle.linear_i4(x, data, scale, bias, n, k, group)
    else:
        if xdt == "f32" and n % 16 == 0 and k % 32 == 0:
            pytest.skip("tiled int8 weights: resolved relative to the row's largest value, as in the int8 GEMV")
        data = np.where(live, rng.integers(-127, 128, size=(n, k)), 0).astype(np.int8)
        scale = (np.abs(rng.standard_normal(n)) * 0.02 / 127 + 1e-8).astype(np.float32)
        ref = oracle.linear_i8(x, data, scale, bias, n, k)
    w = gpu.upload_weight(storage, data, scale, (n, k), group)
    got = gpu.linear(dev(x).to({"f32": torch.float32, "bf16": torch.bfloat16}[xdt]), w, dev(bias))
    gpu.sync()
    got = got.cpu().numpy()
    for c in range(3):
        mine, want = got[:, c::3], ref[:, c::3]
        rep = oracle.allclose(mine, want, atol=1e-5 * float(np.sqrt(np.mean(want.astype(np.float64) ** 2))), rtol=1e-4)
        assert rep["pass"], (DECADES[c], rep)
    w.free()


def test_an_infinite_activation_reaches_the_channels_that_multiply_it(gpu):
    """Inf times a weight is an infinity of the product's sign, times a zero weight a NaN, and stays in its row."""
    n, k, m = 144, 256, 20
    rng = np.random.default_rng(2)
    x = rng.standard_normal((m, k)).astype(np.float32)
    q = rng.integers(-127, 128, size=(n, k)).astype(np.int8)
    q[:, 100] = np.where(np.arange(n) % 3 == 0, 5, np.where(np.arange(n) % 3 == 1, -7, 0))
    scale = np.full(n, 1e-3, np.float32)
    clean = oracle.linear_i8(np.where(np.arange(m)[:, None] == 3, 0, x).astype(np.float32), q, scale, np.zeros(n, np.float32), n, k)
    x[3, 100] = np.inf
    w = gpu.upload_weight("i8", q, scale, (n, k), 0)
    got = gpu.linear(dev(x), w, dev(np.zeros(n, np.float32)))
    gpu.sync()
    got = got.cpu().numpy()
    assert np.all(got[3, 0::3] == np.inf) and np.all(got[3, 1::3] == -np.inf) and np.all(np.isnan(got[3, 2::3]))
    rest = np.arange(m) != 3
    assert oracle.allclose(got[rest], clean[rest], atol=1e-5, rtol=1e-4)["pass"]
    w.free()


@pytest.mark.parametrize("xdt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("storage,group,n", [("i8", 0, 515), ("i8", 0, 512), ("i4", 1024, 512), ("i4", 128, 512)])
def test_long_sums_do_not_drift(gpu, xdt, storage, group, n):
    """2-norm error against f64 of sums over 8192 k.  The tensor core truncates each accumulation of 16 k, half a unit of
    2^-24 on average; chains of at most 256 k have 16: 16 x 2^-25 = 4.8e-7, and the rounding of 32 to 128 chains' sums,
    sqrt(128) x 2^-25 at the most = 3.4e-7: together (at right angles) 6e-7.  (One chain of 1024 k: 1 to 2.6e-6.)"""
    import torch
    if xdt == "bf16" and storage == "i8" and n % 16 == 0:
        pytest.skip("the bf16 GEMM's case")
    m, k = 70, 8192
    rng = np.random.default_rng(n + group)
    x = {"f32": lambda v: v, "f16": oracle.round_to_f16, "bf16": oracle.round_to_bf16}[xdt](rng.standard_normal((m, k)).astype(np.float32))
    bias = np.zeros(n, np.float32)
    if storage == "i4":
        data, scale = cases.synth_i4(n, k, seed=n, group_size=group, scale_dtype="f32")
        ref = oracle.linear_i4(x, data, scale, bias, n, k, group)
    else:
        data, scale = cases.synth_i8(n, k, seed=n)
        ref = oracle.linear_i8(x, data, scale.astype(np.float32), bias, n, k)
    w = gpu.upload_weight(storage, data, scale, (n, k), group)
    got = gpu.linear(dev(x).to({"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[xdt]), w, dev(bias))
    gpu.sync()
    diff = got.cpu().numpy().astype(np.float64) - ref
    assert np.linalg.norm(diff) <= 6e-7 * np.linalg.norm(ref.astype(np.float64)), np.linalg.norm(diff) / np.linalg.norm(ref.astype(np.float64))
    w.free()
