"""FP64 products from digits on the tensor cores (the FP64 form's Grams and
applies): column counts around the 64-column tiles, row counts around the
32-row stages and the chunks, strided, FP32 and complex operands, graded and
spiky ones.

Tolerances.  A product is exact to 2^-58 of its operands' scales per row and
rounded once, so CholeskyQR3 keeps the FP64 form's bounds: 10 n u on
orthogonality and on the columns' backward error (u = 2^-53, n <= 200: 2.2e-13;
the shift of the first pass is undone by the later ones)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu
TOL = 2.2e-13


def check(A64, Q, R, tol=TOL):
    n = A64.shape[1]
    assert np.max(np.abs(Q.T @ Q - np.eye(n))) < tol
    assert np.max(np.linalg.norm(Q @ R - A64, axis=0) / np.linalg.norm(A64, axis=0)) < tol


@pytest.mark.parametrize("m", [200, 255, 256, 257, 288, 289, 511, 4097, 20011])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 127, 129, 200])
@pytest.mark.parametrize("ld", [0, 3])
def test_factors(m, n, ld):
    import pyloworder_gb300 as P
    rng = np.random.default_rng(m * 7 + n)
    W = rng.standard_normal((m, n + ld))
    Q, R = (x.cpu().numpy() for x in P.math.tsqr(torch.from_numpy(W).cuda()[:, ld:]))
    check(W[:, ld:], Q, R)


@pytest.mark.parametrize("kind", ["columns", "rows", "spikes", "tiny", "huge", "zero column"])
def test_scales(kind):
    import pyloworder_gb300 as P
    rng = np.random.default_rng(3)
    m, n = 5000, 70
    A = rng.standard_normal((m, n))
    if kind == "columns":
        A *= 10.0 ** rng.uniform(-3, 3, n)
    elif kind == "rows":
        A *= 10.0 ** rng.uniform(-6, 0, m)[:, None]
    elif kind == "spikes":
        A[rng.integers(0, m, n), np.arange(n)] = 1e5
    elif kind == "tiny":
        A *= 1e-140
    elif kind == "huge":
        A *= 1e140
    elif kind == "zero column":
        A[:, 5] = 0
        U, S, V = P.math.tsqr_svd(torch.from_numpy(A).cuda())
        U, S, V = (x.cpu().numpy() for x in (U, S, V))
        assert np.linalg.norm((U * S) @ V - A) < TOL * np.linalg.norm(A)
        assert np.max(np.abs(S - np.linalg.svd(A, compute_uv=False))) < TOL * S[0]
        return
    Q, R = (x.cpu().numpy() for x in P.math.tsqr(torch.from_numpy(A).cuda()))
    check(A, Q, R)


@pytest.mark.parametrize("m,n", [(3000, 20), (1111, 65)])
@pytest.mark.parametrize("dt", [np.float32, np.complex128, np.float64])
def test_svd(m, n, dt):
    import pyloworder_gb300 as P
    rng = np.random.default_rng(n)
    A = rng.standard_normal((m, n))
    if dt == np.complex128:
        A = A + 1j * rng.standard_normal((m, n))
    A = A.astype(dt)
    U, S, V = P.vmmath.tsqr_svd(torch.from_numpy(A).cuda(), precision="fp64")
    U, S, V = (x.cpu().numpy() for x in (U, S, V))
    tol = 1e-6 if dt == np.float32 else TOL
    ex = np.linalg.svd(A.astype(np.complex128 if dt == np.complex128 else np.float64), compute_uv=False)
    assert np.max(np.abs(S - ex)) < tol * ex[0]
    assert np.linalg.norm((U * S) @ V - A) < tol * np.linalg.norm(A)


def test_not_finite():
    import pyloworder_gb300 as P
    A = np.random.default_rng(1).standard_normal((500, 9))
    for v in (np.nan, np.inf, -np.inf):
        B = A.copy()
        B[77, 4] = v
        with pytest.raises(Exception):
            P.math.tsqr_svd(torch.from_numpy(B).cuda())
