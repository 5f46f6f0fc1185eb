"""The cost slabs built from features against the row-major cost kernel, bit
for bit: tile widths around the chunks of steps a block takes (64 to 576), odd
row counts, feature counts on both sides of the 12 and 16 special forms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

import parflexdtw_b200 as pf  # noqa: E402


@pytest.mark.parametrize("d", [1, 2, 12, 13, 16])
@pytest.mark.parametrize("N,M,L", [(2, 2, 40), (64, 65, 100), (129, 512, 513), (127, 513, 640),
                                   (256, 514, 514), (191, 1091, 1200), (1300, 1700, 600),
                                   (3000, 3100, 230)])
def test_slabs_are_the_cost(N, M, L, d):
    rng = np.random.default_rng(N + M + d)
    F1, F2 = (torch.from_numpy(rng.random((d, n))).cuda() for n in (N, M))
    p = pf.Plan(N, M, L, [(1, 1), (1, 2), (2, 1)], (2.0, 3.0, 3.0))
    p.load_features(F1, F2)
    got = p.cost_matrix()
    p.close()
    assert np.array_equal(got, pf.cost_matrix_from_features_gpu(F1, F2).cpu().numpy())
