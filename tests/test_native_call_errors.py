"""The native form of the serving calls (csrc/kq_torch.cpp): a C++ exception inside one (an output that
cannot be allocated, a tensor without memory) is the Python exception that torch raises for it, and the
process lives on."""
import os
import subprocess
import sys

import numpy as np
import pytest

from tests import cases

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# CUDA tensors of a fake mode have a device, sizes and strides; torch sees no GPU here, so that no output
# can be allocated.  A sparse tensor has no address.
CALLS = """
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from karume_b200 import _kqtorch
with FakeTensorMode():
    x = torch.empty(3, 64, device="cuda")
    bias = torch.empty(32, device="cuda")
    out = torch.empty(3, 32, device="cuda")
    xq = torch.empty(3, 64, device="cuda", dtype=torch.int8)
    xs = torch.empty(3, device="cuda")
    index = torch.empty(3, device="cuda", dtype=torch.int32)
sparse = torch.ones(32).to_sparse()
for name, args in (("linear", (8, 1, 32, 64, x, bias, None)), ("linear", (8, 1, 32, 64, x, sparse, out)),
                   ("linear_fused", (8, [1], 64, x, [sparse], [out], None, 0.0, None, 0)), ("quantize_rows", (8, x)),
                   ("linear_a8", (8, 1, 32, 64, xq, xs, bias, None)), ("embedding", (8, 1, 64, index, None))):
    try:
        getattr(_kqtorch, name)(*args)
    except RuntimeError as e:
        print("raised", name)
"""


def test_a_failure_inside_a_native_call_is_an_exception():
    # in a process of its own: an exception that leaves through CPython ends it
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="", PYTHONPATH=ROOT)
    done = subprocess.run([sys.executable, "-c", CALLS], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, (done.returncode, done.stdout, done.stderr[-2000:])
    assert done.stdout.split() == "raised linear raised linear raised linear_fused raised quantize_rows raised linear_a8 raised embedding".split()


@pytest.mark.gpu
def test_an_output_that_does_not_fit_raises_out_of_memory_and_the_next_call_runs():
    import torch
    import karume_b200 as kb
    gpu = kb.acquire_gpu(0)
    n, k, m = 65536, 64, 4096
    data, scale = cases.synth_i4(n, k, seed=1)
    w = gpu.upload_weight("i4", data, scale, (n, k), 32)
    x, bias = torch.zeros(m, k, device="cuda"), torch.ones(n, device="cuda")
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved(0) + (256 << 20)) / total)  # the output is 1 GiB
    try:
        with pytest.raises(torch.cuda.OutOfMemoryError):
            gpu.linear(x, w, bias)
        got = gpu.linear(x[:2], w, bias)
        gpu.sync()
        assert np.array_equal(got.cpu().numpy(), np.ones((2, n), np.float32))
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    w.free()
    gpu.destroy()
