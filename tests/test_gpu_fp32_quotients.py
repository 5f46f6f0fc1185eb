"""The FP32 form's rounded quotients against the C oracle, bit for bit: costs
whose quotients lie within a few units in the last place of each other, and
magnitudes at and beyond the ends of the range the fast division covers."""
import numpy as np
import pytest

from test_gpu_stage1_blocks import check

pytestmark = pytest.mark.gpu


def near_ties(R, W, seed):
    """1 plus up to three last places: neighbouring paths' means nearly agree."""
    rng = np.random.default_rng(seed)
    return 1.0 + rng.integers(0, 4, (R, W)) * 2.0 ** -23


@pytest.mark.parametrize("R,W,warps", [(400, 600, 4), (1500, 1300, 0), (1300, 1500, 8)])
def test_near_ties(R, W, warps, oracle_mod):
    check(near_ties(R, W, R), warps, oracle_mod, precision="fp32")


@pytest.mark.parametrize("e", [-149, -126, -92, -82, -80, -78, 100, 109, 118, 125])
def test_range_ends(e, oracle_mod):
    C = np.random.default_rng(7).random((230, 250)) * 2.0 ** e
    check(C.astype(np.float32).astype(np.float64), 4, oracle_mod, precision="fp32")


@pytest.mark.parametrize("warps", [0, 4])
def test_zero_regions(warps, oracle_mod):
    rng = np.random.default_rng(11)
    C = rng.random((420, 380))
    C[100:, 60:300] = 0.0
    C[rng.random(C.shape) < 0.2] = 0.0
    C[rng.random(C.shape) < 0.01] *= 2.0 ** -100
    check(C.astype(np.float32).astype(np.float64), warps, oracle_mod, precision="fp32")
