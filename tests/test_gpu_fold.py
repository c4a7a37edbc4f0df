"""Tall operands of at most 64 columns, whose packed rows the tensor products
read in pairs: odd and even row counts around the tiles, dense and strided
rows, narrow and full outputs.

Tolerances: a product of 22-bit operands errs by at most 2^-21 of |A| |B| per
element, its FP32 accumulation by the K = 64 terms' rounding: 1e-6 (|A| |B|).
QR factors: the mixed form's 1e-5."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

ROWS = [1, 2, 3, 127, 128, 129, 255, 256, 257, 511, 4097, 40001]


@pytest.mark.parametrize("m", ROWS)
@pytest.mark.parametrize("n,k", [(1, 1), (7, 64), (32, 5), (63, 63), (64, 64), (64, 65), (65, 64)])
def test_products(m, n, k):
    import pyloworder_gb300 as P
    rng = np.random.default_rng(m * 100 + n + k)
    A = rng.standard_normal((m, n)).astype(np.float32) * 10.0 ** rng.uniform(-6, 6, n).astype(np.float32)
    B = (rng.standard_normal((n, k)) * 10.0 ** rng.uniform(-6, 6, k)).astype(np.float32)
    C = P.math.matmul(A, B).astype(np.float64)
    A64, B64 = A.astype(np.float64), B.astype(np.float64)
    assert np.all(np.abs(C - A64 @ B64) <= 1e-6 * (np.abs(A64) @ np.abs(B64)))


@pytest.mark.parametrize("m", [64, 65, 127, 128, 129, 255, 256, 257, 4097, 40001])
@pytest.mark.parametrize("n", [1, 33, 62, 64])
@pytest.mark.parametrize("ld", [0, 5])
def test_factors(m, n, ld):
    import pyloworder_gb300 as P
    if m < n:
        pytest.skip("tall matrices")
    rng = np.random.default_rng(m + n)
    W = rng.standard_normal((m, n + ld)).astype(np.float32)
    A = torch.from_numpy(W).cuda()[:, ld:]
    Q, R = (x.double().cpu().numpy() for x in P.math.tsqr(A))
    A64 = W[:, ld:].astype(np.float64)
    assert np.max(np.abs(Q.T @ Q - np.eye(n))) < 1e-5
    assert np.linalg.norm(Q @ R - A64) < 1e-5 * np.linalg.norm(A64)
    assert np.linalg.norm(R - np.linalg.qr(A64)[1]) < 1e-4 * np.linalg.norm(R)
