"""The delay phase of the frequency-domain likelihoods on long data at small
delays: the data are the template itself, e^{-2 pi i f tau} at unit size with
the phase reduced exactly (integers), so the residual is the rounding alone.

Bound on its rms per bin: the data's own rounding (sine and cosine of a
reduced angle up to pi: 2^-53 pi / sqrt(3) / 2 from the angle, 2^-53 / sqrt(6)
from the values: 1.1e-16 together) and the kernel's (its unit, 2^-54 of the
template or below, a few of them: 2e-16), 1e-15 allowed.  df is a power of two, so
that df tau itself is exact."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(2.0 ** -10, 1.234e-3, 2 ** 20), (2.0 ** -7, -3.1e-4, 2 ** 18), (2.0 ** -5, 7.3e-3, 32768), (0.125, 0.0213, 8192),
         (2.0 ** -10, 1e-9, 2 ** 19)]


@pytest.fixture(scope="module")
def dev():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")


def _rotated(df, tau, n):
    u = Fraction(df) * Fraction(tau)
    num, den = u.numerator, u.denominator
    turn = np.array([(i * num % den) / den for i in range(n)])
    turn -= np.round(turn)
    return np.exp(-2j * np.pi * turn)


@pytest.mark.parametrize("df,tau,bins", CASES)
def test_dropin(dev, df, tau, bins):
    import torch
    from eobgpu_gb300.eob import pytdinterp
    n = bins + 1
    one, zero = dev(np.ones(n, dtype=complex)), dev(np.zeros(n, dtype=complex))
    out = torch.zeros(-(-n // 1024), dtype=torch.complex128, device="cuda")
    pytdinterp.all_in_one_likelihood(out, one, zero, dev(_rotated(df, tau, n)), dev(np.ones(n)), dev(np.ones(1)),
                                     dev(np.zeros(1)), dev(np.array([tau])), df, 1, 1, n)
    rms = np.sqrt(out.cpu().numpy().real / np.minimum(1024, n - 1024 * np.arange(len(out))))
    assert rms.max() <= 1e-15, rms.max()


@pytest.mark.parametrize("df,tau,bins", CASES)
def test_split_fft(dev, df, tau, bins):
    import torch
    from eobgpu_gb300 import fd
    n, N = bins + 1, 2 * bins
    H = np.zeros((1, N, 2))
    H[0, 1:bins, 0] = 2.0  # h_+ = 1, and 1 / i in h_x, which the second pattern (0) leaves out
    H[0, 0, 0] = H[0, bins, 0] = 1.0
    H = dev(H)
    pat = [dev(np.array([[v]])) for v in (1.0, 0.0, tau)]
    lnl = fd.fd_lnl_from_fft(H, dev(_rotated(df, tau, n)[None]), dev(np.ones((1, n))), *pat, df).cpu().numpy()[0]
    rms = np.sqrt(-lnl / (2.0 * df) / n)
    assert rms <= 1e-15, rms
