"""A batch's stage-2 table is written with its waves, not by a run: a first run
can be captured, a captured run keeps its beta whatever runs in between, and a
run on another stream than the default one finds the table there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

import parflexdtw_b200 as pf  # noqa: E402
from parflexdtw_b200 import workloads as W  # noqa: E402

STEPS, WEIGHTS = [(1, 1), (1, 2), (2, 1)], (2.0, 3.0, 3.0)
SHAPES, LENGTHS = [(300, 410), (90, 700), (257, 511)], [100, 64, 200]


def pairs():
    rng = np.random.default_rng(5)
    return [W.warped_pair(rng, n, m) for n, m in SHAPES]


def make(data, **kw):
    b = pf.Batch(SHAPES, LENGTHS, STEPS, WEIGHTS, 12, **kw)
    b.load(data)
    return b


def outputs(b):
    best, end, lens = b.results()
    return best, end, b.paths(lens)


def check(got, data, beta, oracle_mod):
    best, end, paths = got
    for i, (F1, F2) in enumerate(data):
        ref = oracle_mod.parflex_full(W.cost_matrix_det(F1, F2), STEPS, WEIGHTS, beta, LENGTHS[i])
        assert best[i] == ref["best_cost"]
        assert np.array_equal(paths[i].T, ref["wp"])


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a[:2], b[:2])) and \
        all(np.array_equal(x, y) for x, y in zip(a[2], b[2]))


@pytest.mark.parametrize("cost", ["slabs", "tile"])
@pytest.mark.parametrize("masked", [False, True])
def test_first_run_captured(cost, masked, oracle_mod):
    data = pairs()
    warm = make(data, cost=cost)  # the kernels are loaded
    b = make(data, cost=cost)
    if masked:
        keep = torch.ones(b.tiles, dtype=torch.uint8, device="cuda")
        keep[1::7] = 0
        warm.set_masks(keep)
        b.set_masks(keep)
    want = {}
    for beta in (0.1, 0.35):
        warm.run(beta, use_graph=False)
        want[beta] = outputs(warm)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        b.run(0.1, use_graph=False)
    for other in (None, 0.35, 0.35):
        if other is not None:
            b.run(other)
            assert same(outputs(b), want[other])
        g.replay()
        assert same(outputs(b), want[0.1])
    if not masked:
        check(want[0.1], data, 0.1, oracle_mod)
        check(want[0.35], data, 0.35, oracle_mod)
    torch.cuda.synchronize()
    del g
    warm.close()
    b.close()


def test_first_run_on_a_stream_of_its_own(oracle_mod):
    data = pairs()
    for k in range(8):
        with torch.cuda.stream(torch.cuda.Stream()):
            b = make(data)
            for beta in (0.1, 0.2, 0.35):
                b.run(beta, use_graph=k % 2 == 0)
                check(outputs(b), data, beta, oracle_mod)
            b.set_masks(torch.ones(b.tiles, dtype=torch.uint8, device="cuda"))
            b.run(0.2, use_graph=k % 2 == 1)
            check(outputs(b), data, 0.2, oracle_mod)
            b.close()


@pytest.mark.parametrize("beta", [0.0, 0.1, 0.37, 0.5, 0.99, -0.5, 3.0, 1e300, float("nan")])
def test_scan_buffer_from_beta(beta, oracle_mod):
    """The scan's buffer is computed on the device: of any beta, the columns and
    rows before it are left out, and no others."""
    data = pairs()
    b = make(data)
    b.run(beta)
    b.results()
    for i, (n, m) in enumerate(SHAPES):
        mn, mx = float(min(n, m)), float(max(n, m))
        bg = mn * (1 - (1 - beta) * mn / mx)
        buf = int(bg) if abs(bg) < 2.0 ** 63 else 0
        C = W.cost_matrix_det(*data[i])
        ref = oracle_mod.parflex_full(C, STEPS, WEIGHTS, 0.1, LENGTHS[i])
        D = ref["D_arr"]
        hop = LENGTHS[i] - 1
        for name, size, row in (("TOP_D", m, 0), ("RIGHT_D", n, 1)):
            got = b.plan(i).host(name)
            for g in range(size):
                t = 0 if g == 0 else (g - 1) // hop
                want = D[-1, t, 0, g - t * hop] if row == 0 else D[t, -1, 1, g - t * hop]
                if g < buf or not np.isfinite(want):
                    assert np.isnan(got[g]), (name, g)
                else:
                    assert got[g] == want or np.isnan(got[g]) and g == 0, (name, g)
    b.close()
