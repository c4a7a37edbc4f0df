"""The register FFT of the SPOD stage at every size it takes (32 to 1,024) and at
window counts around its pairs and the window pairs of one pass of a CTA.

Tolerance: log2(N) <= 10 butterfly levels round by half a unit each, of numbers up
to the largest bin: 10 x 2^-24 x 2 (products and sums), 1.2e-6 of the largest
coefficient."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nDFT", [32, 64, 128, 256, 512, 1024])
@pytest.mark.parametrize("nBlks", [1, 2, 3, 15, 16, 17, 31, 32, 33, 34])
@pytest.mark.parametrize("M", [1, 5])
def test_fft(nDFT, nBlks, M):
    import pyloworder_gb300 as P
    rng = np.random.default_rng(nDFT + nBlks)
    step = nDFT // 2 + 1  # windows start at odd samples too
    N = (nBlks - 1) * step + nDFT
    Y = rng.standard_normal((M, N + 3)).astype(np.float32)
    mu = rng.standard_normal(M).astype(np.float32)
    win = 0.54 - 0.46 * np.cos(2 * np.pi * np.arange(nDFT) / (nDFT - 1))
    nf = nDFT // 2 + 1
    Yd = torch.from_numpy(Y).cuda()[:, 1:1 + N]
    Q = P.SPOD.spod_fft_device(Yd, Yd.stride(0), nDFT, nDFT - step, nBlks, nf, win, 0.25,
                               mean=torch.from_numpy(mu).cuda()).cpu().numpy()
    for b in range(nBlks):
        y = (Y[:, 1 + b * step:1 + b * step + nDFT] - mu[:, None]).astype(np.float64)
        F = np.fft.fft(y * win, axis=1)[:, :nf] * 0.25
        F[:, 1:nf - 1] *= 2
        assert np.max(np.abs(Q[:, :, b].T - F)) < 1.2e-6 * np.abs(F).max()


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 9, 1500])
@pytest.mark.parametrize("nBlks,nf", [(1, 1), (2, 2), (3, 17), (31, 31), (31, 32), (31, 33), (7, 129), (2, 4097), (70, 129)])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_gather(M, nBlks, nf, dt):
    # a copy: every value exact, whole points and parts of one per tile
    from pyloworder_gb300 import _lib as L
    if M * nBlks * nf > 5e6:
        pytest.skip("small cases")
    rng = np.random.default_rng(M + nBlks)
    pad = 3  # matrices need not be back to back
    U = rng.standard_normal((nf, M * nBlks + pad, 2)).astype(dt)
    order = rng.permutation(nf).astype(np.int32)
    Ud, od = torch.from_numpy(U).cuda(), torch.from_numpy(order).cuda()
    P = torch.zeros((M * nBlks, nf), dtype=Ud.dtype, device="cuda")
    L.call("plom_spod_gather", L.dtype_code(P), L.ptr(Ud), M, nBlks, nf, M * nBlks + pad, L.ptr(od), L.ptr(P),
           L.stream_ptr())
    ex = U[order, :M * nBlks, 0].reshape(nf, M, nBlks).transpose(2, 1, 0).reshape(M * nBlks, nf)
    assert np.array_equal(P.cpu().numpy(), ex)
