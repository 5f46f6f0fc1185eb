"""The single-tile call with other step sets than the standard one, on both
sides of the rule that gives them to the cluster kernel, and with values that
cross from CTA to CTA, against the C oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parflexdtw_b200.parflex import _tile_full  # noqa: E402

SETS = [([(1, 1)], (2.0,)), ([(1, 2), (2, 1)], (3.0, 3.0)), ([(2, 1), (1, 1), (1, 2)], (3.0, 2.0, 3.0))]


def check(C, steps, weights, oracle_mod):
    D, P, B = _tile_full(torch.from_numpy(C).cuda(), 0, C.shape[0], 0, C.shape[1], steps, weights)
    with np.errstate(all="ignore"):
        _, _, Do, Po, Bo = oracle_mod.flexdtw(C, steps, weights)
    assert np.array_equal(D, Do, equal_nan=True)
    assert np.array_equal(P, Po) and np.array_equal(B, Bo)


@pytest.mark.parametrize("steps,weights", SETS)
@pytest.mark.parametrize("R,W", [(16, 256), (300, 310), (500, 600), (700, 600), (1000, 300),
                                 (300, 1000), (900, 1000), (513, 1200)])
def test_other_steps(R, W, steps, weights, oracle_mod):
    check(np.random.default_rng(R + W).random((R, W)) ** 2, steps, weights, oracle_mod)


@pytest.mark.parametrize("kind", ["ties", "inf", "nan", "negative"])
@pytest.mark.parametrize("steps,weights", [([(1, 1), (1, 2), (2, 1)], (2.0, 3.0, 3.0))] + SETS[:2])
def test_values(kind, steps, weights, oracle_mod):
    rng = np.random.default_rng(6)
    C = rng.random((900, 1000))
    if kind == "ties":
        C = rng.integers(1, 3, C.shape) * 0.5
    elif kind == "negative":
        C -= 0.5
    else:
        C[rng.random(C.shape) < 0.05] = np.inf if kind == "inf" else np.nan
    check(C, steps, weights, oracle_mod)
