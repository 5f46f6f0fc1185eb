"""Stage 1 on the kernel each call asks for: set_warps keeps a tile on one CTA,
whatever the plan would take, and the kernels that the plan takes by itself --
clusters of several CTAs and the 16-warp queue -- against the C oracle, bit for
bit, with every kind of cost and step set."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

import parflexdtw_b200 as pf  # noqa: E402
from test_gpu_stage1_blocks import KINDS, check, cost  # noqa: E402

STD, WEIGHTS = [(1, 1), (1, 2), (2, 1)], (2.0, 3.0, 3.0)


@pytest.mark.parametrize("N,M,L", [(420, 400, 420), (2000, 2000, 2000), (2000, 2400, 500),
                                   (5000, 5100, 1000)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_chosen_warps_are_used(N, M, L, precision):
    p = pf.Plan(N, M, L, STD, WEIGHTS, precision=precision)
    own, rule = p.stage1_shape(), p.warps
    for nw in (4, 8, 16):
        p.set_warps(nw)
        assert p.warps == nw
        shape = p.stage1_shape()
        assert shape == (0, nw, 0) if nw < 16 else shape in ((0, 16, 0), own)
    p.default_warps()
    assert p.stage1_shape() == own and p.warps == rule
    p.close()


def cluster_of(L, M, steps=STD, weights=WEIGHTS, precision="fp64"):
    p = pf.Plan(L, M, L, steps, weights, precision=precision)
    shape = p.stage1_shape()
    p.close()
    return shape[0]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_values_on_clusters(kind, precision, oracle_mod):
    L, M = 1100, 1093
    assert cluster_of(L, M, precision=precision) >= 2
    C = cost(kind, L, M, 5)
    if precision == "fp32":
        if kind in ("tiny", "huge"):
            C *= 2.0 ** (890 if kind == "tiny" else -890)
        C = C.astype(np.float32).astype(np.float64)
    check(C, 0, oracle_mod, precision=precision)


@pytest.mark.parametrize("steps,weights", [([(1, 1), (1, 2), (2, 1)], (1.1, 3.0, 2.7)),
                                           ([(2, 1), (1, 1), (1, 2)], (3.0, 2.0, 3.0)),
                                           ([(1, 2), (2, 1)], (3.0, 3.0)), ([(1, 1)], (2.0,))])
@pytest.mark.parametrize("kind", ["random", "ties", "inf"])
@pytest.mark.parametrize("L", [1100, 2000])
def test_step_sets_on_clusters(L, steps, weights, kind, oracle_mod):
    assert cluster_of(L, L - 5, steps, weights) >= 2
    check(cost(kind, L, L - 5, 9), 0, oracle_mod, steps, weights)


@pytest.mark.parametrize("steps,weights", [(STD, WEIGHTS), ([(1, 2), (1, 1)], (3.0, 2.0))])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_sixteen_warp_queue(steps, weights, precision, oracle_mod):
    """More tiles than SMs on 16 warps each: the same edges and codes as on 4,
    and the oracle's alignment."""
    N, M, L = 2700, 2900, 200
    C = np.random.default_rng(3).random((N, M)) ** 2
    if precision == "fp32":
        C = C.astype(np.float32).astype(np.float64)
    p = pf.Plan(N, M, L, steps, weights, precision=precision)
    got = {}
    for nw in (4, 16):
        p.set_warps(nw)
        assert p.n1 * p.n2 > 148 and p.stage1_shape() == (0, nw, 0)
        p.run(torch.from_numpy(C).cuda(), 0.1)
        best, end, found, n = p.result()
        got[nw] = [p.host(x) for x in ("EDGE_D", "EDGE_P", "BACKPTR")] + [np.float64(best),
                                                                        p.path(n)]
    for a, b in zip(got[4], got[16]):
        assert np.array_equal(a, b)
    if precision == "fp64":
        ref = oracle_mod.parflex_full(C, steps, weights, 0.1, L)
        assert got[16][3] == ref["best_cost"] and np.array_equal(got[16][4].T, ref["wp"])
    p.close()
