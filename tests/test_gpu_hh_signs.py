"""Householder QR's column signs at the edges of the one-CTA elimination (200
columns) and of its warps: the signs of LAPACK's R, for tall and square matrices."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 96, 128, 199, 200, 201, 230])
@pytest.mark.parametrize("extra", [0, 1, 300])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_signs(n, extra, dt):
    import pyloworder_gb300 as P
    A = np.random.default_rng(n + extra).standard_normal((n + extra, n)).astype(dt)
    Q, R = (x.cpu().numpy().astype(np.float64) for x in P.math.tsqr(torch.from_numpy(A).cuda()))
    Qn, Rn = np.linalg.qr(A.astype(np.float64))
    assert np.array_equal(np.sign(np.diag(R)), np.sign(np.diag(Rn)))
    # (a square random matrix may be ill-conditioned: its own condition number)
    tol = (1e-5 if dt == np.float32 else 1e-12) * (1 if extra == 300 else np.linalg.cond(A))
    assert np.linalg.norm(Q @ R - A) < (1e-5 if dt == np.float32 else 1e-12) * np.linalg.norm(A)
    assert np.linalg.norm(R - Rn) < tol * np.linalg.norm(Rn)
