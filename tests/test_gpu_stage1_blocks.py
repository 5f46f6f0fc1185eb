"""The stage-1 kernel's fast and careful loops against the C oracle, bit for
bit: tiles around the strip (64 rows) and block (16 steps) boundaries, and
costs that make cells undecided (ties, zeros), negative or not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

import parflexdtw_b200 as pf  # noqa: E402

STD = [(1, 1), (1, 2), (2, 1)]
KINDS = ("random", "ties", "zeros", "negative", "inf", "nan", "tiny", "huge")


def cost(kind, R, W, seed):
    rng = np.random.default_rng(seed)
    C = rng.random((R, W)) ** 2
    if kind == "ties":  # few distinct values: equal and nearly equal quotients
        C = rng.integers(1, 4, (R, W)) * 0.25
        C[:, W // 2:] *= 1 + 2.0 ** -50
    elif kind == "zeros":
        C[rng.random((R, W)) < 0.5] = 0.0
    elif kind == "negative":
        C -= 0.5
    elif kind == "inf":
        C[rng.random((R, W)) < 0.3] = np.inf
        C[R // 2, :W // 2] = -np.inf
    elif kind == "nan":
        C[rng.random((R, W)) < 0.01] = np.nan
    elif kind == "tiny":  # subnormal quotients
        C *= 2.0 ** -1000
    elif kind == "huge":  # cross products overflow
        C *= 2.0 ** 1008
    return C


def codes(plan, R, W):
    """(R, W) step codes (-1: none) from the plan's packed backpointers."""
    w = plan.host("BACKPTR").view(np.uint32)
    nP = -(-(W + 63) // 16)
    r, c = np.arange(R)[:, None], np.arange(W)[None, :]
    rho = r & 63
    tau = c + rho
    word = w[(((r >> 6) * nP + (tau >> 4)) * 32 + (rho >> 1)) * 2 + (rho & 1)]
    b = ((word >> (2 * (tau & 15)).astype(np.uint32)) & 3).astype(np.int64)
    return np.where(b == 3, -1, b)


def run_tile(C, warps, steps=STD, weights=(2.0, 3.0, 3.0), precision="fp64"):
    R, W = C.shape
    p = pf.Plan(R, W, max(R, W), steps, weights, precision=precision)
    if warps:
        p.set_warps(warps)
    p.load_cost(torch.from_numpy(C).cuda())
    p.stage1()
    D, P, B = p.host("EDGE_D")[0, 0], p.host("EDGE_P")[0, 0], codes(p, R, W)
    p.close()
    return D, P, B


def check(C, warps, oracle_mod, steps=STD, weights=(2.0, 3.0, 3.0), precision="fp64"):
    R, W = C.shape
    D, P, B = run_tile(C, warps, steps, weights, precision)
    with np.errstate(all="ignore"):
        _, _, Do, Po, Bo = oracle_mod.flexdtw(C, steps, weights, fp32=precision == "fp32")
    assert np.array_equal(D[0, :W], Do[-1], equal_nan=True)
    assert np.array_equal(D[1, :R], Do[:, -1], equal_nan=True)
    assert np.array_equal(P[0, :W], Po[-1]) and np.array_equal(P[1, :R], Po[:, -1])
    assert np.array_equal(B, Bo)


# warps 0: the plan's own choice (for one tile, a cluster of CTAs)
@pytest.mark.parametrize("warps", [0, 4, 8])
@pytest.mark.parametrize("R,W", [(2, 2), (3, 200), (200, 3), (64, 97), (65, 96), (127, 129),
                                 (128, 128), (193, 241), (320, 65), (700, 655)])
def test_tile_shapes(R, W, warps, oracle_mod):
    check(cost("random", R, W, R * 1000 + W), warps, oracle_mod)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("warps", [0, 4])
def test_cost_values(kind, precision, warps, oracle_mod):
    C = cost(kind, 333, 290, 5)
    if precision == "fp32":
        if kind in ("tiny", "huge"):
            C *= 2.0 ** (890 if kind == "tiny" else -890)
        C = C.astype(np.float32).astype(np.float64)
    check(C, warps, oracle_mod, precision=precision)


@pytest.mark.parametrize("steps,weights", [([(1, 1), (1, 2), (2, 1)], (1.1, 3.0, 2.7)),
                                           ([(2, 1), (1, 1), (1, 2)], (3.0, 2.0, 3.0)),
                                           ([(1, 2), (2, 1)], (3.0, 3.0)), ([(1, 1)], (2.0,))])
@pytest.mark.parametrize("kind", ["random", "ties", "inf"])
def test_step_sets(steps, weights, kind, oracle_mod):
    check(cost(kind, 150, 219, 9), 4, oracle_mod, steps, weights)


@pytest.mark.parametrize("L,warps", [(257, 4), (320, 8), (1000, 0), (1000, 4), (2000, 0),
                                     (2000, 4), (2000, 16), (2600, 0)])
def test_long_tiles_share_rings(L, warps, oracle_mod):
    """Several rounds of strips per warp, last strips full or not: no strip
    overwrites ring slots another one still reads."""
    check(cost("random", L, L - 3, L), warps, oracle_mod)
