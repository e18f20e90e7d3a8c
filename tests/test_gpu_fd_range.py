"""The integer path of the frequency-domain residual (drop-in
all_in_one_likelihood and the split-FFT likelihood) against the oracle over the
ranges of strain, noise and delay it has to take: geometric units and physical
strain, far above and below the noise, near the ends of FP64, zero data, zero
templates and zero patterns, delays of many turns;
one bin block and the first bin of the next; and what it hands to FP64:
infinities, NaN, infinite and negative PSDs.

Relative 1e-12 on sums of squares: each residual carries a few eps of
|d| + |h| and of its phase (up to 2 pi 8000 x 0.03 turns, 2e-13 rad)."""
import numpy as np
import pytest

from oracle import td_oracle as T

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")


def _case(n, nch, B, hscale, dscale, pscale, seed):
    rng = np.random.default_rng(seed)
    c = lambda k, s: s * (rng.normal(size=k) + 1j * rng.normal(size=k))
    return dict(hp=c(B * n, hscale), hc=c(B * n, hscale), data=c(nch * n, dscale),
                psd=pscale * rng.uniform(0.3, 3.0, nch * n), Fp=rng.uniform(-1, 1, nch * B),
                Fc=rng.uniform(-1, 1, nch * B), tau=rng.uniform(-0.03, 0.03, nch * B), df=0.25, n=n, nch=nch, B=B)


def _run(dev, k):
    import torch
    from eobgpu_gb300.eob import pytdinterp
    out = torch.zeros(-(-k["n"] // 1024) * k["B"] * k["nch"], dtype=torch.complex128, device="cuda")
    pytdinterp.all_in_one_likelihood(out, dev(k["hp"]), dev(k["hc"]), dev(k["data"]), dev(k["psd"]), dev(k["Fp"]),
                                     dev(k["Fc"]), dev(k["tau"]), k["df"], k["B"], k["nch"], k["n"])
    return out.cpu().numpy()


def _ref(k):
    return T.all_in_one_likelihood(k["hp"], k["hc"], k["data"], k["psd"], k["Fp"], k["Fc"], k["tau"], k["df"], k["B"],
                                   k["nch"], k["n"])


@pytest.mark.parametrize("scales", [(1, 1, 1), (1e-23, 1e-23, 1e-46), (1e-18, 1e-23, 1e-46), (1e-29, 1e-23, 1e-46),
                                    (1e140, 1e140, 1e280), (1e-140, 1e-140, 1e-280), (1e-5, 1.0, 1e300), (1, 1e-30, 1)])
@pytest.mark.parametrize("shape", [(1, 1, 1), (1025, 3, 2), (2600, 2, 19), (700, 5, 1)])
def test_scales(dev, scales, shape):
    k = _case(*shape, *scales, 3)
    ref, got = _ref(k).real, _run(dev, k)
    assert np.all(got.imag == 0)
    np.testing.assert_allclose(got.real, ref, rtol=1e-12, atol=0)


@pytest.mark.parametrize("what", ["data", "template", "patterns", "delay", "turns"])
def test_special_values(dev, what):
    k = _case(1500, 2, 3, 1.0, 1.0, 1.0, 5)
    if what == "data":
        k["data"][:] = 0
    elif what == "template":
        k["hp"][:], k["hc"][:] = 0, 0
    elif what == "patterns":
        k["Fp"][:], k["Fc"][:] = 0, 0
    elif what == "delay":
        k["tau"][:] = 0
    else:
        k["tau"] *= 1e3  # phases of 1e5 rad: eps of them in the oracle's own reduction
    np.testing.assert_allclose(_run(dev, k).real, _ref(k).real, rtol=1e-9 if what == "turns" else 1e-12, atol=0)


def test_bins_handed_to_fp64(dev):
    k = _case(1500, 2, 2, 1.0, 1.0, 1.0, 7)
    plain = _ref(k).real.reshape(-1, 2, 2)
    for name, at, value in (("psd", 5, np.inf), ("psd", 7, -2.0), ("psd", 9, 1e-310), ("data", 11, 1e300),
                            ("hp", 13, 1e-320)):
        k[name][at] = value
    with np.errstate(all="ignore"):
        ref = _ref(k).real
    np.testing.assert_allclose(_run(dev, k).real, ref, rtol=1e-12, atol=0)
    for name, at, value in (("data", 11, np.inf), ("hp", 20, np.nan), ("psd", 1501, 0.0)):
        q = _case(1500, 2, 2, 1.0, 1.0, 1.0, 7)
        q[name][at] = value
        got = _run(dev, q).real.reshape(-1, 2, 2)
        bad = ~np.isfinite(got)
        want = np.zeros_like(bad)
        if name == "data":
            want[0, :, 0] = True
        elif name == "hp":
            want[0, 0, :] = True
        else:
            want[0, :, 1] = True
        assert np.array_equal(bad, want), name
        np.testing.assert_allclose(got[~bad], plain[~bad], rtol=1e-12)


@pytest.mark.parametrize("N,nch,start", [(2, 1, 0), (8190, 1, 0), (8192, 4, 40), (8194, 8, 0)])
def test_split_fft_edges(dev, N, nch, start):
    """Bins at the block's edges and every detector count's limits, data far
    below and above the template."""
    import torch
    from eobgpu_gb300 import fd
    rng = np.random.default_rng(N)
    B, n = 3, N // 2 + 1
    h = 1e-22 * (rng.normal(size=(B, N)) + 1j * rng.normal(size=(B, N)))
    H = np.fft.fft(h)
    psd = 1e-46 * rng.uniform(0.5, 2.0, (nch, n))
    psd[:, :2] = 1e300
    data = 1e-21 * rng.choice([1e-6, 1.0, 1e3], size=(nch, n)) * (rng.normal(size=(nch, n)) + 1j * rng.normal(size=(nch, n)))
    Fp, Fx, tau = rng.uniform(-1, 1, (nch, B)), rng.uniform(-1, 1, (nch, B)), rng.uniform(-.02, .02, (nch, B))
    df = 0.125
    got = fd.fd_lnl_from_fft(torch.view_as_real(dev(H)).contiguous(), dev(data), dev(psd), dev(Fp), dev(Fx), dev(tau), df,
                             start).cpu().numpy()
    k = (N - np.arange(n)) % N
    hp, hx = 0.5 * (H[:, :n] + np.conj(H[:, k])), (H[:, :n] - np.conj(H[:, k])) / 2j
    hp[:, :start], hx[:, :start] = 0, 0
    e = np.exp(-2j * np.pi * df * np.arange(n) * tau[:, :, None])  # [nch, B, n]
    r = data[:, None, :] - (Fp[:, :, None] * hp + Fx[:, :, None] * hx) * e
    ref = -0.5 * 4 * df * np.sum(np.abs(r) ** 2 / psd[:, None, :], axis=(0, 2))
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=1e-300)
