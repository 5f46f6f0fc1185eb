"""Stage 2 against the C oracle, bit for bit, where its launches differ: edge
lengths that are no multiple of a warp, one tile to many anti-diagonals, more
dependent slots on a diagonal than the cluster has threads, walks through many
strips, undecidable and non-finite costs (steps that are none), and the same
pairs as a batch (one launch for all of them)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

import parflexdtw_b200 as pf  # noqa: E402
from parflexdtw_b200 import workloads as W  # noqa: E402

STEPS, WEIGHTS, BETA = [(1, 1), (1, 2), (2, 1)], (2.0, 3.0, 3.0), 0.1


def same(a, b):
    return np.array_equal(np.asarray(a), np.asarray(b), equal_nan=True)


def check_plan(plan, best, ref):
    for name, key in (("EDGE_CF", "edge_Cf_olap"), ("D_ARR", "D_arr"), ("L_ARR", "L_arr"),
                      ("TOP_D", "top_D"), ("TOP_L", "top_L"), ("RIGHT_D", "right_D"),
                      ("RIGHT_L", "right_L")):
        assert same(plan.host(name), ref[key]), name
    n_top, n_right = (-(-x // plan.L) for x in (plan.M, plan.N))
    norm = plan.host("SEG_NORM")
    assert same(norm[0, :n_top], ref["seg_best_norm"][0, :n_top])
    assert same(norm[1, :n_right], ref["seg_best_norm"][1, :n_right])
    assert best == ref["best_cost"]


@pytest.mark.parametrize("kind", ["chroma", "ties", "inf"])
@pytest.mark.parametrize("N,M,L", [(40, 50, 60), (61, 47, 7), (300, 410, 33), (515, 290, 100),
                                   (1500, 1700, 1000), (3000, 3300, 3001), (2600, 2500, 301)])
def test_stage2_vs_oracle(N, M, L, kind, oracle_mod):
    rng = np.random.default_rng(N + M + L)
    if kind == "chroma":
        C = W.cost_matrix_det(*W.warped_pair(rng, N, M))
    else:
        C = rng.integers(1, 4, (N, M)) * 0.25
    if kind == "inf":
        C[rng.random((N, M)) < 0.05] = np.inf
        C[N // 3:N // 3 + 3, :M // 2] = np.inf  # no step wins behind it
    try:
        with np.errstate(all="ignore"):
            ref = oracle_mod.parflex_full(C, STEPS, WEIGHTS, BETA, L)
    except ValueError:
        ref = None
    plan = pf.Plan(N, M, L, STEPS, WEIGHTS)
    for _ in range(2):  # the second run finds the first one's lists and counts
        plan.run(torch.from_numpy(C).cuda(), BETA)
        if ref is None:
            with pytest.raises(ValueError):
                plan.result()
            continue
        best, end, _, n = plan.result()
        check_plan(plan, best, ref)
        assert end == ref["best_end"]
        assert same(plan.path(n).T, ref["wp"])
    plan.close()


def test_batch_of_uneven_pairs_is_one_launch_per_step(oracle_mod):
    rng = np.random.default_rng(3)
    shapes = [(700, 90), (90, 700), (257, 511), (64, 64), (1200, 1100)]
    pairs = [W.warped_pair(rng, n, m) for n, m in shapes]
    b = pf.Batch(shapes, [100, 33, 64, 200, 500], STEPS, WEIGHTS, 12)
    b.load(pairs)
    for beta in (0.1, 0.3, 0.1):
        b.run(beta)
        best, end, lens = b.results()
        paths, rows = b.paths(lens), b.paths_rows(lens)
        for i, (F1, F2) in enumerate(pairs):
            ref = oracle_mod.parflex_full(W.cost_matrix_det(F1, F2), STEPS, WEIGHTS, beta, b.L[i])
            check_plan(b.plan(i), best[i], ref)
            assert same(paths[i].T, ref["wp"]) and same(rows[i], ref["wp"])
    b.close()
