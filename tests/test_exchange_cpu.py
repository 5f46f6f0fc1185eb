"""The entries through which lanes pass pairs (csrc/exchange.cuh, compiled for
the host): every store and load of an entry that matter to each other are
ordered by program order and the barriers, whatever the lanes' pace."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
SRC = r"""
#include "exchange.cuh"
extern "C" int store(int lane, int t) { return pfx::exchange_store(lane, t); }
extern "C" int load(int lane, int t) { return pfx::exchange_load(lane, t); }
extern "C" int entries() { return pfx::kXch; }
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("exchange")
    src, lib = str(d / "e.cpp"), str(d / "e.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "parflexdtw_b200", "csrc"), src, "-o", lib])
    return ct.CDLL(lib)


def unordered(store, load, steps, second):
    """Pairs of accesses of an entry by two lanes, one a store, that nothing
    orders, and loads that do not see the previous lane's store of their step.
    second(t): whether a barrier follows step t's loads."""
    clocks = np.zeros((32, 32), int)  # lane's view of every lane's time
    last = {}  # entry -> list of (lane, time, store) since its last store
    seen, bad = {}, 0

    def tick(lane):
        clocks[lane, lane] += 1
        return clocks[lane, lane]

    def access(lane, e, store_):
        nonlocal bad
        for other, time, was_store in last.get(e, []):
            if other != lane and (store_ or was_store) and clocks[lane, other] < time:
                bad += 1
        now = (lane, tick(lane), store_)
        last[e] = [now] if store_ else last.get(e, []) + [now]

    def barrier():
        clocks[:] = clocks.max(axis=0)

    for t in range(steps):
        for lane in range(31):  # lane 31 stores into the ring
            access(lane, store(lane, t), True)
            seen[store(lane, t)] = (t, lane)
        barrier()
        for lane in range(1, 32):  # lane 0 loads from the ring
            access(lane, load(lane, t), False)
            if seen.get(load(lane, t)) != (t, lane - 1):
                bad += 1
        if second(t):
            barrier()
    return bad


def test_every_access_is_ordered(host):
    n = host.entries()
    for t in range(2):
        for lane in range(32):
            assert 0 <= host.store(lane, t) < n and 0 <= host.load(lane, t) < n
    assert unordered(host.store, host.load, 40, lambda t: t % 2 == 0) == 0


def test_the_check_sees_what_is_not(host):
    """Without the barrier after even steps, or with one after odd steps."""
    assert unordered(host.store, host.load, 40, lambda t: False) > 0
    assert unordered(host.store, host.load, 40, lambda t: t % 2 == 1) > 0
