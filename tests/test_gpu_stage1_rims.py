"""Stage 1's loops for blocks at a tile's rim against the C oracle, bit for
bit: lone strips, two strips and more, on both sides of the width (800 columns)
from which strip 0 and the last strip have one, last columns at every place in
a block, and costs that leave the loop."""
import numpy as np
import pytest

from test_gpu_stage1_blocks import check, cost

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,W", [(3, 900), (2, 800), (40, 799), (63, 816), (64, 800), (65, 801),
                                 (100, 1500), (128, 807), (129, 799), (190, 80), (200, 81),
                                 (193, 63), (260, 15), (300, 2), (300, 3), (257, 831)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_rims(R, W, precision, oracle_mod):
    C = cost("random", R, W, R + W)
    if precision == "fp32":
        C = C.astype(np.float32).astype(np.float64)
    for warps in (0, 4):
        check(C, warps, oracle_mod, precision=precision)


@pytest.mark.parametrize("kind", ["ties", "zeros", "inf", "nan", "negative"])
@pytest.mark.parametrize("R,W", [(60, 830), (180, 820), (200, 100)])
def test_values_at_rims(kind, R, W, oracle_mod):
    check(cost(kind, R, W, 3), 4, oracle_mod)
