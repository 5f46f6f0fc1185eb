"""Copies of a batch's paths: any offsets, and with no device memory left."""
import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

import parflexdtw_b200 as pf  # noqa: E402
from parflexdtw_b200 import _lib, plan, workloads as W  # noqa: E402

SHAPES = [(900, 700), (300, 410), (64, 64), (257, 511)]


@pytest.fixture(scope="module")
def batch():
    rng = np.random.default_rng(8)
    b = pf.Batch(SHAPES, 100, [(1, 1), (1, 2), (2, 1)], (2.0, 3.0, 3.0), 12)
    b.load([W.warped_pair(rng, n, m) for n, m in SHAPES])
    b.run(0.1)
    lens = b.results()[2]
    yield b, lens, [b.plan(i).path(int(k)) for i, k in enumerate(lens)]
    b.close()


def copy(fn, b, offsets, cap, lens=None):
    out = np.full((cap, 2), -7, np.int64)
    i64 = ct.POINTER(ct.c_int64)
    args = [out.ctypes.data_as(i64), np.asarray(offsets, np.int64).ctypes.data_as(i64)]
    if lens is not None:
        args.append(np.asarray(lens, np.int64).ctypes.data_as(i64))
    _lib.check(getattr(_lib.load(), fn)(b.handle, plan.current_stream_ptr(), *args, cap))
    return out


@pytest.mark.parametrize("gap,first", [(0, 0), (0, 11), (3, 0), (100000, 5)])
@pytest.mark.parametrize("order", [(0, 1, 2, 3), (2, 0, 3, 1)])
def test_offsets(batch, gap, first, order):
    b, lens, paths = batch
    offs, at = [0] * 4, first
    for i in order:
        offs[i] = at
        at += int(lens[i]) + gap
    out = copy("pfx_batch_copy_paths", b, offs, at)
    rows = copy("pfx_batch_copy_paths_rows", b, offs, at, lens).reshape(-1)
    for o, k, p in zip(offs, lens, paths):
        assert np.array_equal(out[o:o + k], p)
        assert np.array_equal(rows[2 * o:2 * (o + int(k))].reshape(2, -1), p.T)


def test_no_device_memory_left(batch):
    b, lens, paths = batch
    b.paths(lens), b.paths_rows(lens)  # their kernels are loaded
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    pf.clear_plan_cache()
    hogs = []
    for step in (1 << 30, 1 << 25, 1 << 21):
        try:
            while len(hogs) < 1000:
                hogs.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            pass
    try:
        for got in (b.paths(lens), [r.T for r in b.paths_rows(lens)]):
            assert all(np.array_equal(g, p) for g, p in zip(got, paths))
    finally:
        hogs.clear()
        torch.cuda.empty_cache()
