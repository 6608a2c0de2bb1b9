"""Which kernel runs few rows over a row-major weight (karume_b200/csrc/kq_rows_line.h): timed calls of which one side is at least
a tenth faster go to that side."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# (storage, group, m, k, n, activations, us of the kernel for row-major weights, us of the generic or the many-row kernel)
TIMED = [("i4", 16, 2, 256, 64, "f32", 3.6, 2.1), ("i4", 128, 1, 512, 600, "f16", 3.1, 2.6), ("i4", 16, 3, 512, 600, "f32", 4.6, 3.6),
         ("i4", 128, 3, 256, 1024, "f16", 4.6, 2.6), ("i4", 128, 1, 8064, 82, "f32", 5.2, 12.8), ("i8", 0, 1, 8064, 82, "f32", 4.2, 15.6),
         ("i4", 128, 1, 768, 36699, "f32", 9.8, 21.0), ("i4", 128, 4, 768, 36699, "f32", 16.3, 20.5), ("i4", 128, 2, 4096, 4090, "f32", 12.0, 15.4),
         ("i4", 128, 4, 4096, 4090, "f32", 18.5, 14.9), ("i8", 0, 1, 4096, 4090, "f32", 8.7, 16.9), ("i4", 128, 1, 4096, 4090, "f16", 8.7, 11.6),
         ("i8", 0, 1, 4096, 4090, "f16", 7.7, 10.8), ("i8", 0, 2, 4096, 2841, "f16", 12.3, 10.8), ("i8", 0, 4, 2048, 3571, "f16", 13.3, 8.7),
         ("i8", 0, 16, 8064, 82, "f16", 10.8, 8.2), ("i8", 0, 8, 768, 36699, "f32", 29.5, 24.6)]


def test_timed_calls_go_to_the_faster_side(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "rows_line_check"
    subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "karume_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "rows_line_check.cpp"), "-o", str(exe)], check=True)
    lines = []
    for storage, group, m, k, n, x, _, _ in TIMED:
        many_row = m * n * k >= ((12 << 20) if storage == "i4" else (8 << 20))  # the amount of work at which the generic kernel is behind
        lines.append(f"{int(storage == 'i4')} {n} {k} {m} {int(x == 'f16')} {int(many_row)} {group}")
    done = subprocess.run([str(exe)], input="\n".join(lines), capture_output=True, text=True, check=True)
    for case, taken in zip(TIMED, done.stdout.split(), strict=True):
        assert (taken == "1") == (case[6] < case[7]), case
