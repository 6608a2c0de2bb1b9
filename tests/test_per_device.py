"""Limits that a launcher learns from the device (how many clusters it holds) choose K splits, and with them the order of
sums: a thread that saw them half filled would get other bits.  A host program around karume_b200/csrc/kq_per_device.h
asks for them from many threads at once, and no launcher keeps such state outside it."""
import glob
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "karume_b200", "csrc")


def test_entries_are_complete_before_anybody_sees_them(tmp_path):
    gxx = shutil.which("g++")
    cuda = next((p for p in (os.path.join(os.path.dirname(os.path.dirname(shutil.which("nvcc") or "")), "include"), "/usr/local/cuda/include")
                 if os.path.exists(os.path.join(p, "cuda_runtime.h"))), None)
    if gxx is None or cuda is None:
        pytest.skip("no host C++ compiler or no CUDA headers")
    exe = tmp_path / "per_device_check"
    subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", CSRC, "-isystem", cuda,
                    os.path.join(ROOT, "tests", "native", "per_device_check.cpp"), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout + done.stderr


def test_no_launcher_fills_a_shared_entry_in_place():
    for name in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(name) as fh:
            text = fh.read()
        assert not re.search(r"(->|\.)slot\(\)|->done\b.*=\s*true", text), os.path.basename(name)
