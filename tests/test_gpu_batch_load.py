"""Batch.load: every form of input ends up in the batch's buffers unchanged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

import parflexdtw_b200 as pf  # noqa: E402

STEPS, W = [(1, 1), (1, 2), (2, 1)], (2.0, 3.0, 3.0)


def form(x, k):
    """x (d, n) as the k-th kind of input."""
    t = torch.from_numpy(x).cuda()
    d, n = x.shape
    if k == 0:
        return t
    if k == 1:  # base off a 16-byte boundary
        flat = torch.empty(d * n + 1, dtype=torch.float64, device="cuda")
        flat[1:] = t.reshape(-1)
        return flat[1:].view(d, n)
    if k == 2:  # strided
        return torch.cat([t, t], 1)[:, :n]
    if k == 3:
        return t.t().contiguous().t()
    if k == 4:
        return t.to(torch.float32)
    if k == 5:
        return x
    return t.clone().requires_grad_()


@pytest.mark.parametrize("pairs,lo,hi,d", [(1, 2, 3, 1), (3, 300, 400, 5), (70, 40, 90, 3),
                                           (5, 4000, 5001, 12)])
def test_load_forms(pairs, lo, hi, d):
    rng = np.random.default_rng(pairs)
    shapes = [tuple(int(v) for v in rng.integers(lo, hi, 2)) for _ in range(pairs)]
    b = pf.Batch(shapes, 200, STEPS, W, d)
    data = [tuple(rng.integers(0, 1 << 20, (d, n)) / 8.0 for n in s) for s in shapes]
    with torch.no_grad():
        b.load([tuple(form(x, (2 * i + j) % 7) for j, x in enumerate(p))
                for i, p in enumerate(data)])
    for i, p in enumerate(data):
        for got, x in zip(b.feature_views(i), p):
            assert np.array_equal(got.cpu().numpy(), x.astype(np.float64))
    # its own buffers as the source
    b.load([b.feature_views(i) for i in range(pairs)])
    for i, p in enumerate(data):
        assert np.array_equal(b.feature_views(i)[1].cpu().numpy(), p[1])
    with pytest.raises(ValueError):
        b.load([(x[:, :-1], y) for x, y in data])
    b.close()
