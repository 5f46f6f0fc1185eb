"""Scratch of the single-tile call: backpointers of the tile's own shape."""
import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parflexdtw_b200.parflex import _tile_full  # noqa: E402
from test_zz_no_alloc import _pool_used_high, _reset_pool_high  # noqa: E402

STD = [(1, 1), (1, 2), (2, 1)]


@pytest.mark.parametrize("R,W", [(300, 8000), (8000, 300), (64, 65), (16, 2000)])
def test_backpointer_scratch(R, W, oracle_mod):
    C = np.random.default_rng(R).random((R, W))
    Cd = torch.from_numpy(C).cuda()
    rt = ct.CDLL("libcudart.so.12")
    pool = ct.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(ct.byref(pool), torch.cuda.current_device()) == 0
    torch.cuda.synchronize()
    _reset_pool_high(rt, pool)
    base = _pool_used_high(rt, pool)
    D, P, B = _tile_full(Cd, 0, R, 0, W, STD, (2.0, 3.0, 3.0))
    cells = -(-R // 64) * 64 * (-(-(W + 63) // 16) * 16)
    assert 0 < _pool_used_high(rt, pool) - base <= cells // 4 + 24 * max(R, W) + 4096
    _, _, Do, Po, Bo = oracle_mod.flexdtw(C, STD, (2.0, 3.0, 3.0))
    assert np.array_equal(D, Do) and np.array_equal(P, Po) and np.array_equal(B, Bo)
