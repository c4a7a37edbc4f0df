"""The reduced DMD stage at the sizes where its matrices leave shared memory (the
eigenvectors of T above r = 79, P and both matrices above 112), and at the smallest.

A is normal (rotations of distinct angles and radii in an orthogonal basis), so
its eigenvalues, its unitary eigenvectors and the amplitudes (P is diagonal) are
perfectly conditioned: errors of r eps each, 1e-12 up to r = 130 with the
amplitudes' sums over the snapshots."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 31, 32, 33, 40, 41, 64, 79, 80, 81, 111, 112, 113, 114, 130])
def test_reduced(N):
    from pyloworder_gb300 import _lib as L
    rng = np.random.default_rng(N)
    nt = 2 * N + 17
    D = np.zeros((N, N))
    for k in range(N // 2):
        th, r = np.pi * (k + 0.5) / (N // 2 + 1), 1.0 - 0.2 * rng.random()
        D[2 * k:2 * k + 2, 2 * k:2 * k + 2] = r * np.array([[np.cos(th), -np.sin(th)], [np.sin(th), np.cos(th)]])
    if N % 2:
        D[-1, -1] = 0.95
    Q = np.linalg.qr(rng.standard_normal((N, N)))[0]
    A = Q @ D @ Q.T
    S = np.sort(rng.uniform(1, 2, N))[::-1].copy()
    VT = np.linalg.qr(rng.standard_normal((nt, N)))[0].T.copy()
    aux1 = A @ (S[:, None] * VT)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    muR, muI = torch.empty(N, dtype=torch.float64, device="cuda"), torch.empty(N, dtype=torch.float64, device="cuda")
    b = torch.empty(2 * N, dtype=torch.float64, device="cuda")
    Mphi = torch.empty((nt, 2 * N), dtype=torch.float64, device="cuda")
    ws, info = L.workspace(L.load().plom_dmd_reduced_workspace(N, nt)), L.new_info()
    a1, s1, v1 = d(aux1), d(S), d(VT)
    L.call("plom_dmd_reduced", L.ptr(a1), L.ptr(s1), L.ptr(v1), N, nt, L.ptr(muR), L.ptr(muI), L.ptr(b),
           L.ptr(Mphi), L.ptr(ws), ws.numel(), L.ptr(info), L.stream_ptr())
    L.check_info(info, "DMD reduced stage")
    mu = muR.cpu().numpy() + 1j * muI.cpu().numpy()
    bj = b.cpu().numpy().view(np.complex128)
    M = Mphi.cpu().numpy().view(np.complex128)
    ex = np.linalg.eigvals(A)
    dist = np.abs(mu[:, None] - ex[None])
    assert dist.min(1).max() < 1e-12 and dist.min(0).max() < 1e-12
    assert np.all(np.diff(np.abs(bj)) < 1e-10)
    # the modes: (S VT)^T-weighted eigenvectors, A w = mu w, |w| = 1
    W = (S[:, None] * VT) @ M * mu
    assert np.max(np.abs(A @ W - W * mu)) < 1e-11
    assert np.max(np.abs(np.linalg.norm(W, axis=0) - 1)) < 1e-11
    # the amplitudes reproduce the projected snapshots: sum_k w_k b_k mu_k^t, least squares
    V = mu[:, None] ** np.arange(nt)
    P = (W.conj().T @ W) * (V @ V.conj().T).conj()
    q = np.diag(V @ (S[:, None] * VT).conj().T @ W).conj()
    assert np.max(np.abs(P @ bj - q)) < 1e-10 * np.max(np.abs(q))
