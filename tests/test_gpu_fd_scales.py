"""The drop-in frequency-domain residual where the polarisations and the
patterns differ in size, the smaller of one on the larger of the other: a
detector at the null of one pattern with a source seen near edge-on.  Every
bin's error has to stay a rounding of |F+ h+| + |Fx hx|, as in FP64,
whatever the sizes of the other products' factors.

The data are the template, in extended precision and rounded, and each bin is
weighted by 1 / (|F+ h+| + |Fx hx|)^2, so that the root mean square of a block
is the relative error: the data's rounding 2^-53 / sqrt(3) and the kernel's unit of at
most 2^-54 a few times over, together 2e-16; 1e-15 allowed, beside the delay phase's
own two roundings in the reference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Fp,Fx", [(0.0, 1.0), (1e-9, 0.7), (0.6, 0.0), (0.9, -1e-12), (-0.3, 0.8), (1e-30, 1e-31), (1e-5, 1e5)])
@pytest.mark.parametrize("ratio", [1.0, 1e-3, 1e-6, 1e-12, 1e6, 1e9, 0.0, "mixed"])
@pytest.mark.parametrize("tau", [0.0, 0.013])
def test_relative_error(Fp, Fx, ratio, tau):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300.eob import pytdinterp
    n, df, LD = 2048, 0.25, np.longdouble
    rng = np.random.default_rng(5)
    size = 10.0 ** rng.uniform(-12, 12, n) if ratio == "mixed" else ratio
    hp = 1e-22 * (rng.normal(size=n) + 1j * rng.normal(size=n))
    hx = 1e-22 * size * (rng.normal(size=n) + 1j * rng.normal(size=n))
    turn = (df * np.arange(n)) * tau
    turn -= np.round(turn)
    ph = -2 * LD(np.pi) * turn.astype(LD) - 2 * LD(1.2246467991473532e-16) * turn.astype(LD)  # pi to 107 bits
    c, s = np.cos(ph), np.sin(ph)
    gr = LD(Fp) * hp.real.astype(LD) + LD(Fx) * hx.real.astype(LD)
    gi = LD(Fp) * hp.imag.astype(LD) + LD(Fx) * hx.imag.astype(LD)
    data = (gr * c - gi * s).astype(np.float64) + 1j * (gr * s + gi * c).astype(np.float64)
    scale = np.abs(Fp * hp) + np.abs(Fx * hx)
    scale[scale == 0] = 1.0
    d = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")
    out = torch.zeros(-(-n // 1024), dtype=torch.complex128, device="cuda")
    pytdinterp.all_in_one_likelihood(out, d(hp), d(hx), d(data), d(scale ** 2), d(np.array([Fp])), d(np.array([Fx])),
                                     d(np.array([tau])), df, 1, 1, n)
    rms = np.sqrt(out.cpu().numpy().real / 1024)
    # f tau is rounded twice in the reference here: 2^-53 of up to 42 rad
    allowed = 1e-15 + (2 * 2.0 ** -53 * 2 * np.pi * df * n * tau)
    assert rms.max() <= allowed, rms.max()


@pytest.mark.parametrize("nch", [1, 3, 8])
def test_split_fft(nch):
    """The same from the FFT of h_+ + i h_x, patterns of very different sizes beside ordinary ones.
    FP64 rounds H itself to 2^-53 of |h_+|, which is the template's error here: with data of
    the template's size, 1e-3 |h_+|, 2^-53 1e3 of it twice over: 1e-12."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300 import fd
    B, N, df = 3, 4096, 0.25
    n = N // 2 + 1
    rng = np.random.default_rng(nch)
    c = lambda *k: rng.normal(size=k) + 1j * rng.normal(size=k)
    hp, hx = c(B, n), 1e-3 * c(B, n)
    for a in (hp, hx):
        a[:, 0], a[:, -1] = a[:, 0].real, a[:, -1].real
    H = np.zeros((B, N), dtype=complex)
    H[:, :n] = hp + 1j * hx
    H[:, n:] = (np.conj(hp) + 1j * np.conj(hx))[:, -2:0:-1]
    Fp, Fx, tau = rng.uniform(-1, 1, (nch, B)), rng.uniform(-1, 1, (nch, B)), rng.uniform(-0.02, 0.02, (nch, B))
    Fp[0] = [0.0, 1e-9, 1e-3]
    data, psd = 1e-3 * c(nch, n), rng.uniform(0.5, 2.0, (nch, n))
    k = (N - np.arange(n)) % N
    p, x = 0.5 * (H[:, :n] + np.conj(H[:, k])), (H[:, :n] - np.conj(H[:, k])) / 2j
    e = np.exp(-2j * np.pi * df * np.arange(n) * tau[:, :, None])
    r = data[:, None, :] - (Fp[:, :, None] * p + Fx[:, :, None] * x) * e
    ref = -2.0 * df * np.sum(np.abs(r) ** 2 / psd[:, None, :], axis=(0, 2))
    d = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")
    got = fd.fd_lnl_from_fft(torch.view_as_real(d(H)).contiguous(), d(data), d(psd), d(Fp), d(Fx), d(tau), df)
    np.testing.assert_allclose(got.cpu().numpy(), ref, rtol=1e-12)
