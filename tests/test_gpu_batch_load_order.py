"""Batch.load copies in the order given: a buffer of the batch that is a source
of a later pair has its new contents by then, whatever kind each source is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

import parflexdtw_b200 as pf  # noqa: E402


@pytest.mark.parametrize("kinds", [("host", "own"), ("device", "own"), ("f32", "own"),
                                   ("own", "host"), ("own", "device")])
def test_own_buffers_as_sources(kinds):
    d, n, m = 3, 700, 900
    b = pf.Batch([(n, m), (n, m), (n, m)], 200, [(1, 1), (1, 2), (2, 1)], (2.0, 3.0, 3.0), d)
    rng = np.random.default_rng(1)
    old, new, last = ([rng.integers(0, 99, (d, x)) * 0.5 for x in (n, m)] for _ in range(3))
    b.load([old, old, old])

    def source(kind, data, own):
        if kind == "own":
            return b.feature_views(own)
        if kind == "host":
            return data
        t = [torch.from_numpy(x).cuda() for x in data]
        return [x.float() for x in t] if kind == "f32" else t

    # "own" second: pair 0's buffers after they were given `new`; "own" first:
    # pair 1's buffers before they are
    own = 0 if kinds[1] == "own" else 1
    b.load([source(kinds[0], new, own), source(kinds[1], new, own), last])
    want = [new, new, last] if own == 0 else [old, new, last]
    for i in range(3):
        for got, x in zip(b.feature_views(i), want[i]):
            assert np.array_equal(got.cpu().numpy(), x)
    b.close()
