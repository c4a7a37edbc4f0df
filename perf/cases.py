"""The work that a user of this package has it do, as cases that can be timed and compared.

A case is a dict of plain values; `kind` names the public call and the sizes
are those of the snapshot matrix (m points x n snapshots, one snapshot per
column).  Sizes come from the package's own workloads: 16,384 to 4,194,304
points and 32 to 1,024 snapshots for POD and DMD (the serving mix), the
16,384 x 200 FP64 field of the plain form, 2,097,152 x 512 with r = 32 for
DMD, rank 64 + 16 with two power iterations for the randomized SVD, 256-point
windows with half overlap for SPOD.  Odd and ragged sizes are among them.

What is returned.  A singular vector has an arbitrary sign (a phase, if
complex), and the vectors of a noise floor are an arbitrary basis of it, so a
program that uses the factors does not depend on either: it truncates, and
reconstructs.  The SVD and DMD cases return the singular values (eigenvalues)
whole and the reconstructed field whole; QR factors, whose signs are fixed,
and products come back as they are; SPOD returns all energies and
frequencies and the leading modes, which are the ones that the data
determines.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import pyloworder_gb300 as plom

ROWS = 1 << 18  # rows generated at a time


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def listed():
    return [
        # the smallest job of the serving mix: launches and the n x n stage
        {"name": "pod_16384x32", "kind": "pod", "m": 16384, "n": 32, "dtype": "float32"},
        # the plain form: FP64 POD of a 128 x 128 grid, 200 snapshots
        {"name": "pod_f64_16384x200", "kind": "pod", "m": 16384, "n": 200, "dtype": "float64"},
        # an ordinary unstructured-mesh POD: neither size is a multiple of anything
        {"name": "pod_250001x301", "kind": "pod", "m": 250001, "n": 301, "dtype": "float32"},
        # the largest job of the serving mix
        {"name": "pod_4194304x1024", "kind": "pod", "m": 4194304, "n": 1024, "dtype": "float32"},
        # tsqr_svd of a long, narrow field in which every mode is resolved
        {"name": "svd_2097152x64", "kind": "svd", "m": 2097152, "n": 64, "dtype": "float32"},
        # an orthonormal basis of a ragged field (Q and R)
        {"name": "tsqr_1000003x96", "kind": "tsqr", "m": 1000003, "n": 96, "dtype": "float32"},
        # a few leading modes of a large field by the randomized range finder
        {"name": "rpod_2097152x512", "kind": "rpod", "m": 2097152, "n": 512, "dtype": "float32",
         "r": 80, "q": 2},
        # DMD at full size: 16 conjugate pairs, and the field they give back
        {"name": "dmd_2097152x512", "kind": "dmd", "m": 2097152, "n": 512, "dtype": "float32",
         "r": 32, "remove_mean": False},
        # a small DMD with the default mean removal
        {"name": "dmd_65537x129", "kind": "dmd", "m": 65537, "n": 129, "dtype": "float32",
         "r": 10, "remove_mean": True},
        # SPOD with 256-point windows and half overlap (31 blocks, 129 frequencies)
        {"name": "spod_262144x4096", "kind": "spod", "m": 262144, "n": 4096, "dtype": "float32",
         "ndft": 256, "nolap": 128},
        # a small SPOD with every parameter left at its default
        {"name": "spod_20011x600", "kind": "spod", "m": 20011, "n": 600, "dtype": "float32",
         "ndft": 0, "nolap": 0},
        # projection of a field onto given modes and back (matmulp, matmul)
        {"name": "project_1048577x200", "kind": "project", "m": 1048577, "n": 200,
         "dtype": "float32", "r": 50},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pod", "pod", "pod", "pod64", "svd", "tsqr", "rpod", "dmd", "dmd", "spod",
                       "spod", "project"])
    if kind == "pod64":
        n = _log(rng, 32, 256)
        return {"kind": "pod", "m": _log(rng, 16384, min(262144, 5.0e9 / n ** 2)), "n": n,
                "dtype": "float64"}
    if kind == "spod":
        n = _log(rng, 256, 8192)
        ndft = rng.choice([0] + [d for d in (64, 128, 256) if 8 * d <= n <= 32 * d])  # at most 63 blocks
        return {"kind": "spod", "m": _log(rng, 8192, min(1048576, 2 ** 30 / n)), "n": n,
                "dtype": "float32", "ndft": ndft, "nolap": ndft // 2}
    m = _log(rng, 16384, 2097152)
    case = {"kind": kind, "m": m, "dtype": "float32"}
    if kind == "pod":
        return dict(case, n=_log(rng, 32, 1024))
    if kind in ("svd", "tsqr"):
        return dict(case, n=_log(rng, 32, 128))
    if kind == "rpod":
        r = rng.randrange(20, 81)
        return dict(case, n=_log(rng, 4 * r, 1024), r=r, q=rng.choice([1, 2, 3]))
    if kind == "dmd":
        r = 2 * rng.randrange(3, 17)
        return dict(case, n=_log(rng, 4 * r, 512), r=r, remove_mean=rng.random() < 0.5)
    return dict(case, n=_log(rng, 32, 1024), r=rng.randrange(8, 97))


# --------------------------------------------------------------------------
# seeded fields, made on the device
# --------------------------------------------------------------------------

def _dt(case):
    return getattr(torch, case["dtype"])


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _modes(case):
    """Coherent modes of a POD field: a quarter of the snapshots, 64 at most;
    of a randomized one, what the rank leaves besides the oversampling."""
    return case["r"] * 4 // 5 if case["kind"] == "rpod" else max(4, min(64, case["n"] // 4))


def _pod_field(case, seed):
    """sum_k k^-1.5 sin(kx x) sin(ky y) cos(w_k t + th_k) + 1e-5 N(0, 1) on a
    two-dimensional grid: distinct spatial modes, frequencies over [0.1, 2]."""
    m, n, dt, K = case["m"], case["n"], _dt(case), _modes(case)
    rng = np.random.default_rng([seed, 1])
    pairs = rng.choice(256, size=K, replace=False)
    w = 0.1 + 1.9 * (rng.permutation(K) + rng.uniform(0.25, 0.75, K)) / K
    th = rng.uniform(0, 2 * np.pi, K)
    amp = np.arange(1, K + 1) ** -1.5
    T = torch.tensor(amp[:, None] * np.cos(w[:, None] * np.arange(n) + th[:, None]), dtype=dt,
                     device="cuda")
    kx = torch.tensor(pairs // 16 + 1, dtype=dt, device="cuda")
    ky = torch.tensor(pairs % 16 + 1, dtype=dt, device="cuda")
    ny = math.isqrt(m)
    hx, hy = 2 * math.pi / max(1, -(-m // ny) - 1), 2 * math.pi / (ny - 1)
    g, X = _gen(seed), torch.empty((m, n), dtype=dt, device="cuda")
    for r0 in range(0, m, ROWS):
        i = torch.arange(r0, min(m, r0 + ROWS), device="cuda")
        xs, ys = (i // ny).to(dt) * hx, (i % ny).to(dt) * hy
        phi = torch.sin(xs[:, None] * kx) * torch.sin(ys[:, None] * ky)
        X[r0:r0 + ROWS] = phi @ T
        X[r0:r0 + ROWS].add_(torch.randn((len(i), n), dtype=dt, device="cuda", generator=g), alpha=1e-5)
    return X


def _decaying_field(m, n, dt, seed, last=1e-2):
    """A field whose n modes are all resolved: random spatial modes, energies
    falling geometrically from 1 to `last`, an orthogonal temporal basis."""
    rng = np.random.default_rng([seed, 2])
    V = np.linalg.qr(rng.standard_normal((n, n)))[0]
    A = torch.tensor((last ** (np.arange(n) / max(1, n - 1)))[:, None] * V.T, dtype=dt, device="cuda")
    g, X = _gen(seed), torch.empty((m, n), dtype=dt, device="cuda")
    for r0 in range(0, m, ROWS):
        X[r0:r0 + ROWS] = torch.randn((min(ROWS, m - r0), n), dtype=dt, device="cuda", generator=g) @ A
    return X


def _smooth_shapes(m, k, dt, rng, scale=None):
    """m x k smooth random spatial shapes (64 waves each), made row chunk by row chunk."""
    C = torch.tensor(rng.standard_normal((64, k)) / 8 * (1 if scale is None else scale), dtype=dt, device="cuda")
    ph = torch.tensor(rng.uniform(0, 2 * np.pi, 64), dtype=dt, device="cuda")
    wave = torch.arange(1, 65, dtype=dt, device="cuda") * (2 * math.pi / m)
    for r0 in range(0, m, ROWS):
        i = torch.arange(r0, min(m, r0 + ROWS), dtype=dt, device="cuda")
        yield r0, torch.sin(i[:, None] * wave + ph) @ C


def _dmd_field(case, seed):
    """r / 2 conjugate pairs exp((s + i w) dt), s in [-0.05, 0], w over
    [0.05, 3], dt = 0.1, on smooth random spatial modes, plus 1e-4 noise."""
    m, n, dt, p = case["m"], case["n"], _dt(case), case["r"] // 2
    rng = np.random.default_rng([seed, 3])
    om = 0.05 + 2.95 * (np.arange(p) + rng.uniform(0.3, 0.7, p)) / p
    if n < 256:  # a short record still has to hold some periods of each mode
        om *= 256 / n
    lam = np.exp((rng.uniform(-0.05, 0.0, p) + 1j * om) * 0.1)
    V = lam[:, None] ** np.arange(n)
    T = torch.tensor(2 * np.concatenate([V.real, -V.imag]), dtype=dt, device="cuda")
    g, X = _gen(seed), torch.empty((m, n), dtype=dt, device="cuda")
    for r0, phi in _smooth_shapes(m, 2 * p, dt, rng):
        X[r0:r0 + ROWS] = phi @ T
        X[r0:r0 + ROWS].add_(torch.randn((len(phi), n), dtype=dt, device="cuda", generator=g), alpha=1e-4)
    return X


def _spod_field(case, seed):
    """Three coherent broadband structures (each a third of the last) on smooth
    shapes, plus AR(1) red noise (coefficient 0.9) at every point."""
    m, n, dt = case["m"], case["n"], _dt(case)
    rng, g = np.random.default_rng([seed, 4]), _gen(seed)
    H = 1 / (1 - 0.9 * torch.exp(-2j * math.pi * torch.fft.rfftfreq(n, device="cuda")))

    def red(rows):
        e = torch.randn((rows, n), dtype=dt, device="cuda", generator=g)
        return torch.fft.irfft(torch.fft.rfft(e, dim=1) * H, n=n, dim=1)

    S, X = red(3), torch.empty((m, n), dtype=dt, device="cuda")
    rows = max(1, (1 << 28) // n)
    for r0, phi in _smooth_shapes(m, 3, dt, rng, scale=np.array([1.0, 0.3, 0.1])):
        X[r0:r0 + ROWS] = phi @ S
    for r0 in range(0, m, rows):
        X[r0:r0 + rows].add_(red(min(rows, m - r0)), alpha=1e-2)
    return X


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------

def prepare(case, seed):
    kind, m, n = case["kind"], case["m"], case["n"]
    state = {"case": case}
    if kind in ("pod", "rpod"):
        state["X"] = _pod_field(case, seed)
    elif kind == "dmd":
        state["X"] = _dmd_field(case, seed)
        state["t"] = torch.arange(n - 1, dtype=torch.float64, device="cuda")
    elif kind == "spod":
        state["X"] = _spod_field(case, seed)
        state["t"] = np.arange(n, dtype=np.float64)
    else:
        state["X"] = _decaying_field(m, n, _dt(case), seed)
        if kind == "project":
            U = torch.randn((m, case["r"]), dtype=_dt(case), device="cuda", generator=_gen(seed + 1))
            state["U"] = U.div_(math.sqrt(m))
    return state


def run(state):
    case, X = state["case"], state["X"]
    kind = case["kind"]
    if kind == "pod":
        U, S, V = plom.POD.run(X)
        return S, plom.POD.reconstruct(*plom.POD.truncate(U, S, V, r=_modes(case)))
    if kind == "rpod":
        U, S, V = plom.POD.run(X, randomized=True, r=case["r"], q=case["q"], seed=7)
        return S, plom.POD.reconstruct(*plom.POD.truncate(U, S, V, r=_modes(case)))
    if kind == "svd":
        U, S, V = plom.math.tsqr_svd(X)
        return S, plom.POD.reconstruct(U, S, V)
    if kind == "tsqr":
        return plom.math.tsqr(X)
    if kind == "dmd":
        muR, muI, Phi, b = plom.DMD.run(X, case["r"], remove_mean=case["remove_mean"])
        return muR, muI, plom.DMD.reconstruction_jovanovic(Phi, muR, muI, state["t"], b)
    if kind == "spod":
        L, P, f = plom.SPOD.run(X, state["t"], nDFT=case["ndft"], nolap=case["nolap"])
        return L, P[:3 * case["m"]], f  # rows i + m b: the three leading modes b
    if kind == "project":
        A = plom.math.matmulp(state["U"].T, X)
        return A, plom.math.matmul(state["U"], A)
    raise ValueError(kind)


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------

def _welch(case):
    n, ndft, nolap = case["n"], case["ndft"], case["nolap"]
    ndft = ndft or 2 ** int(math.floor(math.log2(n / 10)))
    nolap = nolap or ndft // 2
    return ndft, nolap, (n - nolap) // (ndft - nolap), -(-ndft // 2) + 1


def work(case):
    m, n, s = case["m"], case["n"], 8 if case["dtype"] == "float64" else 4
    kind, r = case["kind"], case.get("r", 0)
    if kind in ("pod", "svd"):
        K = _modes(case) if kind == "pod" else n
        # X in; U, V and the reconstruction out; Gram + U, then the reconstruction
        return {"bytes": s * (3 * m * n + n * n), "flops": 4 * m * n * n + 2 * m * n * K}
    if kind == "tsqr":
        return {"bytes": s * (2 * m * n + n * n), "flops": 4 * m * n * n}
    if kind == "rpod":
        return {"bytes": s * (2 * m * n + m * r + r * n),
                "flops": 4 * m * n * r * (case["q"] + 1) + 4 * m * r * r * (case["q"] + 1) + 2 * m * n * _modes(case)}
    if kind == "dmd":
        # X in; Phi and the reconstruction out; Gram, U_r, its projection, Phi, reconstruction
        return {"bytes": s * (2 * m * n + 2 * m * r), "flops": 2 * m * n * n + 2 * m * n * r * 6}
    if kind == "spod":
        ndft, _, nb, nf = _welch(case)
        return {"bytes": s * (m * n + m * nb * nf),
                "flops": int(2.5 * ndft * math.log2(ndft)) * m * nb + 12 * m * nb * nb * nf}
    return {"bytes": s * (2 * m * n + m * r), "flops": 4 * m * n * r}


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------

def _chunks(X):
    rows = max(1, (1 << 26) // X.shape[1])
    return (X[r0:r0 + rows].double() for r0 in range(0, X.shape[0], rows))


def _gram_svd(X, remove_mean, cols=None):
    """Singular values and right vectors of X (mean removed), from its Gram matrix."""
    G = 0
    for c in _chunks(X):
        c = c - c.mean(1, keepdim=True) if remove_mean else c
        c = c[:, :cols]
        G = G + c.T @ c
    lam, V = torch.linalg.eigh(G)
    return lam.clamp_min(0).sqrt().flip(0), V.flip(1)


def _dmd_order(mu, b):
    """Descending |b|; of a conjugate pair the positive imaginary part first."""
    order = np.flip(np.abs(b).argsort())
    mu = mu[order].copy()
    i = 0
    while i < len(mu) - 1:
        if mu[i].imag != 0:
            if mu[i].imag < 0:
                mu[i], mu[i + 1] = mu[i].conj(), mu[i]
            i += 1
        i += 1
    return mu


def exact(case, seed):
    state = prepare(case, seed)
    X, kind, n = state["X"], case["kind"], case["n"]
    if kind != "spod" and case["m"] * n * n > 1.2e12:  # the 64-bit Gram matrix alone takes seconds
        return None
    if kind in ("pod", "rpod"):
        S, V = _gram_svd(X, True)
        Vk, K = V[:, :_modes(case)], case["r"] if kind == "rpod" else n
        rec = torch.cat([(c - c.mean(1, keepdim=True)) @ Vk @ Vk.T for c in _chunks(X)])
        return S[:K], rec
    if kind == "svd":
        return _gram_svd(X, False)[0], X.double()
    if kind == "tsqr":
        return tuple(torch.linalg.qr(X.double()))
    if kind == "project":
        A = sum(u.T @ x for u, x in zip(state["U"].double().split(1 << 20), X.double().split(1 << 20)))
        return A, state["U"].double() @ A
    if kind == "dmd":
        r, nt = case["r"], n - 1
        rm = case["remove_mean"]
        S, V = _gram_svd(X, rm, nt)
        S, V = S[:r], V[:, :r]
        A = 0  # U^T Y2
        for c in _chunks(X):
            c = c - c.mean(1, keepdim=True) if rm else c
            A = A + ((c[:, :nt] @ V) / S).T @ c[:, 1:]
        Sn, Vn = S.cpu().numpy(), V.cpu().numpy()
        mu, W = np.linalg.eig(A.cpu().numpy() @ (Vn / Sn))
        vand = mu[:, None] ** np.arange(nt)
        P = (W.conj().T @ W) * (vand @ vand.conj().T).conj()
        q = np.diag(vand @ (Sn[:, None] * Vn.T).conj().T @ W).conj()
        b = np.linalg.solve(P, q)
        M = torch.tensor(((Vn / Sn) @ W / mu) @ (b[:, None] * vand), device="cuda").real.contiguous()
        rec = torch.cat([(c - c.mean(1, keepdim=True) if rm else c)[:, 1:] @ M for c in _chunks(X)])
        mu = _dmd_order(mu, b)
        return mu.real.copy(), mu.imag.copy(), rec
    ndft, nolap, nb, nf = _welch(case)
    i = np.arange(ndft)
    win = 0.54 - 0.46 * np.cos(2 * np.pi * i / (ndft - 1))
    scale = np.full(nf, 2.0)
    scale[[0, -1]] = 1.0
    wt = torch.tensor(win, device="cuda")
    sc = torch.tensor(scale / win.mean() / ndft / math.sqrt(nb), device="cuda")
    G = torch.zeros((nf, nb, nb), dtype=torch.complex128, device="cuda")
    rows = max(1, (1 << 25) // (nb * ndft))
    for r0 in range(0, case["m"], rows):
        c = X[r0:r0 + rows].double()
        c = c - c.mean(1, keepdim=True)
        Q = (torch.fft.fft(c.unfold(1, ndft, ndft - nolap)[:, :nb] * wt)[:, :, :nf] * sc).permute(2, 0, 1)
        G += Q.mH @ Q
    L = torch.linalg.eigvalsh(G).flip(1)
    order = torch.argsort(L[:, 0], descending=True)
    f = order.cpu().numpy() / float(ndft)  # unit time step
    return L[order], None, f
