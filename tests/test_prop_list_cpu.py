"""Entries of the propagation's lists (csrc/prop_list.cuh, compiled for the
host): slots and sources beyond 2^31 come back as they went in, and the
geometries whose places or distances would not fit are told apart."""
import ctypes as ct
import os
import random
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
SRC = r"""
#include "prop_list.cuh"
extern "C" void pack(int32_t n2, int32_t L2, int32_t a, int32_t i, int64_t k, int64_t src,
                     int32_t copy, int32_t* out) {
    out[0] = pfx::prop_place(n2, L2, a, i, k);
    out[1] = pfx::prop_back(k, src, copy != 0);
}
extern "C" void unpack(int32_t n2, int32_t L2, int32_t a, const int32_t* v, int32_t* i,
                       int64_t* out) {
    out[0] = pfx::prop_slot(n2, L2, a, v[0], i);
    out[1] = pfx::prop_src(out[0], v[1]);
    out[2] = v[1] < 0;
}
extern "C" int fits(int64_t n1, int64_t n2, int64_t L) { return pfx::prop_list_fits(n1, n2, L); }
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("prop_list")
    src, lib = str(d / "p.cpp"), str(d / "p.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "parflexdtw_b200", "csrc"), src, "-o", lib])
    h = ct.CDLL(lib)
    h.pack.argtypes = [ct.c_int32] * 4 + [ct.c_int64] * 2 + [ct.c_int32, ct.c_void_p]
    h.fits.argtypes = [ct.c_int64] * 3
    return h


# tiles of 64 rows of 258,100 x 258,100 cells: 2.15e9 slots
@pytest.mark.parametrize("n1,n2,L", [(1, 1, 2), (1, 7, 3), (7, 1, 100), (5, 9, 33),
                                     (4097, 4097, 64), (16, 16777200, 64), (2, 1 << 20, 500),
                                     (1, 1 << 26, 17), (1 << 26, 1, 17), (300000, 300, 12)])
def test_round_trip(host, n1, n2, L):
    assert host.fits(n1, n2, L)
    rng = random.Random(n1 + n2)
    L2 = 2 * L
    v, back, row = (ct.c_int32 * 2)(), (ct.c_int64 * 3)(), ct.c_int32()
    tiles = [(n1 - 1, n2 - 1), (n1 - 1, 0), (0, n2 - 1)]
    tiles += [(rng.randrange(n1), rng.randrange(n2)) for _ in range(300)]
    for i, j in tiles:
        for q in (0, L2 - 1, rng.randrange(L2)):
            k = (i * n2 + j) * L2 + q
            for di, dj in ((1, 0), (0, 1)):
                if i < di or j < dj:
                    continue
                for s in (0, L2 - 1, rng.randrange(L2)):
                    src = ((i - di) * n2 + j - dj) * L2 + s
                    for copy in (0, 1):
                        host.pack(n2, L2, i + j, i, k, src, copy, v)
                        assert v[0] >= 0
                        host.unpack(n2, L2, i + j, v, ct.byref(row), back)
                        assert (row.value, list(back)) == (i, [k, src, copy])


@pytest.mark.parametrize("n1,n2,L,ok", [
    (1 << 20, 1 << 20, 1023, True), (1 << 20, 1 << 20, 1024, False),  # places
    (1 << 20, (1 << 20) - 1, 1024, True), (2, (1 << 24) - 1, 64, True),  # distances
    (2, 1 << 24, 64, False), (1, 1 << 24, 64, True)])
def test_what_fits(host, n1, n2, L, ok):
    assert bool(host.fits(n1, n2, L)) == ok
