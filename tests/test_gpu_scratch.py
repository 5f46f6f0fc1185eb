"""The scratch memory that the library keeps between calls is given back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

import parflexdtw_b200 as pf  # noqa: E402
from parflexdtw_b200.parflex import _tile_full  # noqa: E402


def test_clear_plan_cache_gives_it_back(oracle_mod):
    C = torch.rand((3000, 3100), dtype=torch.float64, device="cuda")

    def call():
        return _tile_full(C, 0, 3000, 0, 3100, [(1, 1), (1, 2), (2, 1)], (2.0, 3.0, 3.0))
    D = call()[0]  # 12 bytes per cell of scratch: 112 MB
    torch.cuda.synchronize()
    kept = torch.cuda.mem_get_info()[0]
    pf.clear_plan_cache()
    assert torch.cuda.mem_get_info()[0] - kept >= 100 << 20
    assert np.array_equal(call()[0], D)  # and is taken again when it is needed
    pf.clear_plan_cache()
    pf.clear_plan_cache()
