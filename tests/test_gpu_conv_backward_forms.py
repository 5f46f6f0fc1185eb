"""The convolutions' backward kernels beyond the shapes and values of
test_gpu_conv_backward.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

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
