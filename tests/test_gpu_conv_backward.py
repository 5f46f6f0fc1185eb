"""The convolutions' backward kernels on sparse and dense output gradients
against the numpy oracle.  A sum of n products in FP32, in any order, is within
(n + 2) 2^-24 (1 + small) of exact relative to the sum of the products'
magnitudes; the bound used is 1.1 (n + 2) 2^-24 times that sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import cnn_oracle as CO  # noqa: E402
from parflexdtw_b200 import _lib, plan  # noqa: E402


@pytest.mark.parametrize("density", [0.0, 0.004, 0.3, 1.0])
@pytest.mark.parametrize("cin,cout,stride,relu,H,W", [(32, 32, 2, 1, 95, 131), (1, 32, 4, 1, 70, 61),
                                                      (32, 1, 1, 0, 33, 65), (40, 36, 1, 1, 20, 17),
                                                      (5, 3, 2, 0, 16, 1), (64, 64, 4, 1, 9, 30)])
def test_backward(cin, cout, stride, relu, H, W, density):
    rng = np.random.default_rng(cin + cout + H)
    x = rng.standard_normal((cin, H, W)).astype(np.float32)
    w = (rng.standard_normal((cout, cin, 3, 3)) * 0.3).astype(np.float32)
    Ho, Wo = (H - 1) // stride + 1, (W - 1) // stride + 1
    y = rng.standard_normal((cout, Ho, Wo)).astype(np.float32)
    dy = rng.standard_normal((cout, Ho, Wo)).astype(np.float32)
    dy *= rng.random((1, Ho, Wo)) < density
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, w, y, dy)]
    dx = torch.full((cin, H, W), 7.0, device="cuda")  # every value is stored
    dw = torch.full((cout, cin, 3, 3), 0.5, device="cuda")  # added to
    db = torch.full((cout,), -0.25, device="cuda")
    _lib.check(_lib.load().pfx_conv3x3_backward(
        d[0].data_ptr(), cin, H, W, d[1].data_ptr(), cout, stride, d[2].data_ptr(), relu,
        d[3].data_ptr(), dx.data_ptr(), dw.data_ptr(), db.data_ptr(), plan.current_stream_ptr()))
    ref = CO.conv3x3_backward(x, w, stride, y, relu, dy)
    mag = CO.conv3x3_backward(np.abs(x), np.abs(w), stride, y, relu, np.abs(dy))
    n = Ho * Wo
    for got, want, size, terms, start in ((dx, ref[0], mag[0], 9 * cout, 0.0),
                                          (dw, ref[1], mag[1], n, 0.5), (db, ref[2], mag[2], n, -0.25)):
        err = np.abs(got.cpu().numpy().astype(np.float64) - (want + start))
        assert (err <= 1.1 * (terms + 2) * 2.0 ** -24 * (size + abs(start))).all()
