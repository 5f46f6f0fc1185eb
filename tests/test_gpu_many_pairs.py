"""A wave of more pairs than one grid's second dimension holds (65535)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

import parflexdtw_b200 as pf  # noqa: E402
from parflexdtw_b200 import workloads as W  # noqa: E402

STEPS, WEIGHTS, BETA, L = [(1, 1), (1, 2), (2, 1)], (2.0, 3.0, 3.0), 0.1, 12


def test_66000_pairs(oracle_mod):
    rng = np.random.default_rng(2)
    kinds = [W.warped_pair(rng, int(n), int(m)) for n, m in rng.integers(20, 30, (61, 2))]
    refs = [oracle_mod.parflex_full(W.cost_matrix_det(*p), STEPS, WEIGHTS, BETA, L) for p in kinds]
    dev = [tuple(torch.from_numpy(f).cuda() for f in p) for p in kinds]
    n = 66000
    shapes = [(kinds[i % 61][0].shape[1], kinds[i % 61][1].shape[1]) for i in range(n)]
    b = pf.Batch(shapes, L, STEPS, WEIGHTS, 12)
    assert b.waves == 1
    b.load([dev[i % 61] for i in range(n)])
    b.run(BETA, use_graph=False)
    best, end, lens = b.results()
    paths = b.paths(lens)
    for i in range(n):
        ref = refs[i % 61]
        assert best[i] == ref["best_cost"] and np.array_equal(paths[i].T, ref["wp"]), i
    b.close()
