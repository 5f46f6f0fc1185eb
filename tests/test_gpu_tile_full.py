"""The single-tile call with full D, P and B outputs against the C oracle, bit
for bit, around the size from which it runs on a cluster (4096 cells), strip
and chunk boundaries, cost rows apart, and undecidable or non-finite costs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

import parflexdtw_b200 as pf  # noqa: E402

STD = [(1, 1), (1, 2), (2, 1)]


def check(C, oracle_mod, steps=STD, weights=(2.0, 3.0, 3.0), pad=0):
    R, W = C.shape
    full = torch.zeros((R, W + pad), dtype=torch.float64, device="cuda")
    full[:, :W] = torch.from_numpy(C)
    with np.errstate(all="ignore"):
        _, _, D, P, B, _ = pf.flexdtw_chunk_from_global_C(full, W + pad, 0, R, 0, W, steps,
                                                          list(weights))
        _, _, Do, Po, Bo = oracle_mod.flexdtw(C, steps, weights)
    assert np.array_equal(D, Do, equal_nan=True)
    assert np.array_equal(P, Po) and np.array_equal(B, Bo)


@pytest.mark.parametrize("R,W", [(63, 65), (64, 64), (16, 256), (15, 700), (300, 16), (65, 200), (257, 190),
                                 (512, 577), (1500, 1801), (3100, 900)])
def test_shapes(R, W, oracle_mod):
    check(np.random.default_rng(R + W).random((R, W)) ** 2, oracle_mod, pad=R % 7)


@pytest.mark.parametrize("kind", ["ties", "inf", "nan", "negative"])
@pytest.mark.parametrize("steps,weights", [(STD, (2.0, 3.0, 3.0)), ([(2, 1), (1, 1)], (3.0, 2.0))])
def test_values(kind, steps, weights, oracle_mod):
    rng = np.random.default_rng(4)
    C = rng.random((200, 230))
    if kind == "ties":
        C = rng.integers(1, 3, C.shape) * 0.5
    elif kind == "negative":
        C -= 0.5
    else:
        C[rng.random(C.shape) < 0.05] = np.inf if kind == "inf" else np.nan
    best = np.isfinite(C).all()
    if best:
        check(C, oracle_mod, steps, weights)
        return
    from parflexdtw_b200.parflex import _tile_full  # no endpoint to search for
    D, P, B = _tile_full(torch.from_numpy(C).cuda(), 0, 200, 0, 230, steps, weights)
    with np.errstate(all="ignore"):
        _, _, Do, Po, Bo = oracle_mod.flexdtw(C, steps, weights)
    assert np.array_equal(D, Do, equal_nan=True)
    assert np.array_equal(P, Po) and np.array_equal(B, Bo)


@pytest.mark.parametrize("n", [1, 1023, (1 << 20) - 1, 1 << 20, (1 << 20) + 1, 3 * (1 << 20) + 17])
def test_host_copies(n):
    """Uploads and downloads in pieces of 8 MB return what went in."""
    from parflexdtw_b200.parflex import _download, cost_matrix_to_gpu
    C = np.random.default_rng(n).random((1, n))
    up = cost_matrix_to_gpu(C)
    codes = torch.arange(n, device="cuda").to(torch.int8)
    D, B = _download(up, codes)
    assert up.shape == C.shape and np.array_equal(D, C)
    assert B.dtype == np.int8 and np.array_equal(B, codes.cpu().numpy())
