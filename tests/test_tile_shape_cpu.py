"""The rules for a single tile with full outputs (csrc/tile_shape.cuh, compiled
for the host)."""
import ctypes as ct
import os
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
SRC = r"""
#include "tile_shape.cuh"
extern "C" int on_cluster(int32_t R, int32_t W, int steps, int std_steps, double n) {
    return pfx::full_tile_on_cluster(R, W, steps, std_steps != 0, n);
}
extern "C" int ctas(int strips, int cw, int most) {
    return pfx::full_tile_ctas(strips, cw, [&](int n) { return n <= most; });
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("tile_shape")
    src, lib = str(d / "t.cpp"), str(d / "t.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "parflexdtw_b200", "csrc"), src, "-o", lib])
    h = ct.CDLL(lib)
    h.on_cluster.argtypes = [ct.c_int32, ct.c_int32, ct.c_int, ct.c_int, ct.c_double]
    return h


def cluster_steps(R, W, warps=32):
    """Pipeline steps of an R x W tile on a cluster's warps."""
    span = -(-(W + 63) // 16) * 16
    lag = max(80, -(-(-(-span // warps)) // 16) * 16)
    return (-(-R // 64) - 1) * max(lag, 120) + span


# (R, W): whether the cluster was the faster one with one step, two, three in
# another order (measured; None: within 6 %), and with the standard steps
FASTER = {(16, 256): (0, 0, 0, 1), (64, 64): (0, 0, 0, 1), (100, 120): (0, 0, 0, 1),
          (300, 310): (0, 0, 0, 1), (450, 450): (None, 0, 0, 1), (500, 600): (1, None, 0, 1),
          (700, 600): (1, None, None, 1), (1000, 1000): (1, 1, 1, 1), (1500, 1801): (1, 1, 1, 1),
          (30, 3000): (0, 0, 0, 1), (3000, 30): (0, 0, 0, 1), (65, 3000): (0, 0, 0, 1),
          (200, 3000): (None, 0, 0, 1), (3000, 200): (0, 0, 0, 1), (300, 3000): (1, 1, None, 1),
          (500, 3000): (1, 1, 1, 1), (9000, 20): (0, 0, 0, 1), (9000, 100): (0, 0, 0, 1),
          (300, 1000): (1, 0, 0, 1), (1000, 300): (0, 0, 0, 1), (15, 700): (0, 0, 0, 0),
          (63, 65): (0, 0, 0, 0)}


@pytest.mark.parametrize("R,W", sorted(FASTER))
def test_the_faster_kernel(host, R, W):
    n = cluster_steps(R, W)
    for steps, std, want in zip((1, 2, 3, 3), (0, 0, 0, 1), FASTER[R, W]):
        if want is not None:
            assert host.on_cluster(R, W, steps, std, n) == want


@pytest.mark.parametrize("strips,cw,want", [(1, 4, 1), (4, 4, 1), (5, 4, 2), (16, 4, 4), (17, 4, 8),
                                            (48, 4, 8), (49, 8, 8), (500, 8, 8)])
def test_ctas(host, strips, cw, want):
    """As many CTAs as the strips ask for, or what can be resident at once; 0
    (the other kernel) where no cluster can."""
    for most in (0, 1, 2, 3, 4, 7, 8, 16):
        got = host.ctas(strips, cw, most)
        fits = [n for n in (1, 2, 4, 8) if n <= min(want, most)]
        assert got == (max(fits) if fits else 0)
