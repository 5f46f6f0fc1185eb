"""A plan made and run on a stream of its own while the default stream is busy:
its buffers' first fills come before its first work."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

import parflexdtw_b200 as pf  # noqa: E402
from parflexdtw_b200 import workloads as W  # noqa: E402

STEPS, WEIGHTS, BETA = [(1, 1), (1, 2), (2, 1)], (2.0, 3.0, 3.0), 0.1


@pytest.mark.parametrize("ranged", [False, True])
def test_first_run_beside_a_busy_default_stream(ranged, oracle_mod):
    F1, F2 = W.warped_pair(np.random.default_rng(4), 900, 1100)
    ref = oracle_mod.parflex_full(W.cost_matrix_det(F1, F2), STEPS, WEIGHTS, BETA, 100)
    dev = [torch.from_numpy(f).cuda() for f in (F1, F2)]
    for _ in range(3):
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)  # about 10 ms
        with torch.cuda.stream(torch.cuda.Stream()):
            p = pf.Plan(900, 1100, 100, STEPS, WEIGHTS)
            if ranged:  # every tile, but no cost slabs made by the first load
                p.set_tile_range(0, p.n1 * p.n2)
            p.load_features(*dev)
            p.run(None, BETA)
            best, _, _, n = p.result()
            assert best == ref["best_cost"] and np.array_equal(p.path(n).T, ref["wp"])
            p.close()
