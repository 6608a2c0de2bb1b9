"""How a many-row call is cut into tiles and K slices (karume_b200/csrc/kq_exact_geometry.h) is host arithmetic: a host program
checks it over a grid of shapes, and that the shapes which the GPU tests run for a form of the kernel are cut that way."""
import os
import shutil
import subprocess

import pytest

from tests import cases

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path_factory.mktemp("geometry") / "exact_geometry_check"
    subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "karume_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "exact_geometry_check.cpp"), "-o", str(exe)], check=True)
    return str(exe)


def cut(program, shapes):
    """(rows per tile, row tiles, slices, slices in a cluster) of (x, storage, group, m, n, k) each."""
    lines = []
    for x, storage, group, m, n, k in shapes:
        tiled_i8 = storage == "i8" and n % 16 == 0 and k % 32 == 0
        math = {"f16": 0, "bf16": 2, "i8": 4}.get(x, 1 if tiled_i8 else 3)
        lines.append(f"{m} {n} {k} {math} {group}")
    done = subprocess.run([program, "shapes"], input="\n".join(lines), capture_output=True, text=True, check=True)
    return [tuple(map(int, line.split())) for line in done.stdout.splitlines()]


def test_tiles_and_slices_cover_a_call(program):
    done = subprocess.run([program], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout + done.stderr
    assert done.stdout.startswith("ok "), done.stdout


def test_the_shapes_of_the_cluster_tests_are_cut_in_clusters(program):
    shapes = [s[:6] for s in cases.EXACT_SLICED]
    for shape, (nt, tiles, slices, in_cluster) in zip(cases.EXACT_SLICED, cut(program, shapes), strict=True):
        assert (nt, slices, in_cluster) == (shape[6], shape[7], shape[7]), (shape, nt, tiles, slices, in_cluster)


def test_the_shapes_of_the_resident_pair_tests_are_more_tiles_than_pairs(program):
    shapes = [("i8", "i8", 0, m, n, k) for m, n, k in cases.EXACT_RESIDENT]
    for (_, _, _, m, n, k), (nt, tiles, slices, _) in zip(shapes, cut(program, shapes), strict=True):
        assert slices == 1 and (n + 255) // 256 * tiles > 74, (m, n, k, nt, tiles, slices)


# Cuts that were timed against their neighbours, with those that came within 3 % of the fastest: (rows a tile, slices, slices
# in a cluster)
MEASURED = [(("f32", "i4", 32, 2048, 4096, 14336), {(256, 1, 1)}), (("f32", "i4", 32, 1905, 4608, 1600), {(256, 1, 1)}),
            (("f16", "i8", 0, 153, 5280, 1152), {(64, 1, 1)}), (("f16", "i4", 32, 675, 432, 640), {(32, 1, 1)}),
            (("f32", "i4", 32, 1788, 400, 640), {(64, 1, 1)}), (("f16", "i4", 64, 422, 832, 640), {(32, 1, 1)}),
            (("f32", "i4", 32, 804, 6144, 4096), {(160, 1, 1)}), (("f16", "i4", 32, 87, 1152, 1792), {(32, 4, 4)})]


def test_measured_shapes_are_cut_as_was_fastest(program):
    for (shape, fast), (nt, _, slices, in_cluster) in zip(MEASURED, cut(program, [s for s, _ in MEASURED]), strict=True):
        assert (nt, slices, in_cluster) in fast, (shape, nt, slices, in_cluster)
