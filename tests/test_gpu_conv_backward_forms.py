"""The convolutions' backward kernels beyond the shapes and values of
test_gpu_conv_backward.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import cnn_oracle as CO  # noqa: E402
from parflexdtw_b200 import _lib, plan  # noqa: E402


def backward(x, w, stride, y, relu, dy, dx, dw, db):
    _lib.check(_lib.load().pfx_conv3x3_backward(
        x.data_ptr(), *x.shape, w.data_ptr(), w.shape[0], stride, y.data_ptr(), relu,
        dy.data_ptr(), None if dx is None else dx.data_ptr(), dw.data_ptr(), db.data_ptr(),
        plan.current_stream_ptr()))


def test_more_than_2_31_pixels():
    """Listed pixels in every part of a map of more than 2^31 (about 38 GB in
    all): the sums are small integers, so exact in FP32."""
    H, W = 46500, 46400
    if torch.cuda.mem_get_info()[0] < 40e9:
        pytest.skip("needs 40 GB")
    x, y, dy = (torch.zeros((1, H, W), device="cuda") for _ in range(3))
    rng = np.random.default_rng(1)
    rows = np.concatenate([rng.integers(1, H - 1, 40), [1, H - 2]])
    cols = np.concatenate([rng.integers(1, W - 1, 40), [1, W - 2]])
    assert rows.max() * W > 1 << 31
    want = np.zeros((3, 3))
    for k, (r, c) in enumerate(zip(rows, cols)):  # one value of x next to each
        ky, kx = k % 3, k // 3 % 3
        x[0, r + ky - 1, c + kx - 1] = k + 1.0
        y[0, r, c] = 1.0
        dy[0, r, c] = 2.0
    xh = [(int(r), int(c)) for r, c in zip(rows, cols)]
    for r, c in set(xh):
        want += 2.0 * x[0, r - 1:r + 2, c - 1:c + 2].cpu().numpy()
    w = torch.ones((1, 1, 3, 3), device="cuda")
    dx, dw = torch.empty_like(x), torch.zeros((1, 1, 3, 3), device="cuda")
    db = torch.zeros(1, device="cuda")
    backward(x, w, 1, y, 1, dy, dx, dw, db)
    assert np.array_equal(dw.cpu().numpy()[0, 0], want) and db.item() == 2.0 * len(set(xh))
    for r, c in xh:
        assert dx[0, r, c].item() >= 2.0
    assert dx.sum(dtype=torch.float64).item() == 18.0 * len(set(xh))
    del x, y, dy, dx
    torch.cuda.empty_cache()


@pytest.mark.parametrize("where", ["x", "w", "both", "dy"])
@pytest.mark.parametrize("cin,cout,stride,H,W", [(32, 32, 2, 41, 60), (1, 32, 4, 70, 61),
                                                 (32, 1, 1, 19, 33), (40, 36, 1, 20, 17)])
def test_values_that_are_not_finite(cin, cout, stride, H, W, where):
    """An infinite or NaN weight or activation makes NaN of every product it is
    in, those with a gradient of 0 among them, as a dense sum has it."""
    rng = np.random.default_rng(cin + H)
    Ho, Wo = (H - 1) // stride + 1, (W - 1) // stride + 1
    x = rng.standard_normal((cin, H, W)).astype(np.float32)
    w = rng.standard_normal((cout, cin, 3, 3)).astype(np.float32)
    y = np.ones((cout, Ho, Wo), np.float32)
    dy = (rng.standard_normal(y.shape) * (rng.random((1, Ho, Wo)) < 0.05)).astype(np.float32)
    dy[:, 2:, :] = 0  # far from what follows
    if where in ("x", "both"):
        x[0, H - 3, W // 2], x[cin - 1, H - 2, 1] = np.inf, np.nan
    if where in ("w", "both"):
        w[0, 0, 1, 1], w[cout - 1, cin - 1, 2, 0] = -np.inf, np.nan
    if where == "dy":
        dy[0, Ho - 1, Wo - 1], dy[cout - 1, Ho // 2, 0] = np.inf, np.nan
    d = [torch.from_numpy(a).cuda() for a in (x, w, y, dy)]
    dx, dw = torch.full((cin, H, W), 7.0, device="cuda"), torch.zeros((cout, cin, 3, 3), device="cuda")
    db = torch.zeros(cout, device="cuda")
    backward(d[0], d[1], stride, d[2], 1, d[3], dx, dw, db)
    with np.errstate(all="ignore"):
        ref = CO.conv3x3_backward(x, w, stride, y, 1, dy)
    assert any(np.isnan(r).any() for r in ref)
    for got, want in zip((dx, dw, db), ref):
        got = got.cpu().numpy()
        assert np.array_equal(np.isnan(got), np.isnan(want))
        assert np.array_equal(np.isinf(got), np.isinf(want))
        ok = np.isfinite(want)
        # sums of at most 9 cout or Ho Wo products of standard normals
        assert np.allclose(got[ok], want[ok], rtol=1e-4, atol=1e-3)
