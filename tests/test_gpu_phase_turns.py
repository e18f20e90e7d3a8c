"""Multiples of the integer phase (PhaseTurns), which every call of several
modes takes, read through TDInterp_wrap2: three modes of amplitude 1, one at
a time, with constant phase splines return e^{-i m phi}, against extended
precision of the exact product m phi: around zero, at the table's steps and
quadrants, at phases of long inspirals, and on both sides of 2^40, where the library
takes over.

Bound below 2^40: the turn is cut off at 2^-64 (times m, 2 pi m 2^-64), the integer
steps are within 2^-59.6, the result is rounded (2^-54 for values up to 1, 2^-53
at 1); the sum of the modes adds exact zeros.  Above: the product m phi rounds in
the library's argument, m phi 2^-53."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BELOW = [0.0, 1e-300, 5e-39, 1e-20, 1e-8, 2.0 ** 39, 2.0 ** 40 - 0.25, 3.0e11]
ABOVE = [2.0 ** 40, 2.0 ** 40 + 3.0, 2.0 ** 41, 1e15]


def _run(phi, ms, which):
    import torch
    from eobgpu_gb300.eob import pytdinterp
    n, K = len(phi), len(ms)
    d = lambda a, t=torch.float64: torch.tensor(np.ascontiguousarray(a), dtype=t, device="cuda")
    y = np.zeros((2 * K + 1, n))
    y[which] = 1.0
    y[2 * K] = phi
    zero = d(np.zeros(y.size))
    one = lambda v: d([v], torch.int32)
    out = torch.zeros(n, dtype=torch.complex128, device="cuda")
    pytdinterp.TDInterp_wrap2(out, d(np.zeros(n)), d(np.zeros(n)), d(y.ravel()), zero, zero, zero, n, one(n), n, 1, K,
                              d([8] * K, torch.int32), d(ms, torch.int32), d(np.arange(n), torch.int32), one(n), n)
    return out.cpu().numpy()


@pytest.mark.parametrize("ms", [(2, 1, 3), (5, 5, 4), (8, -2, 7)])
def test_multiples_against_extended_precision(ms):
    torch = pytest.importorskip("torch")
    mp = pytest.importorskip("mpmath")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(sum(ms))
    step = 2 * np.pi / 2048
    k = np.arange(0, 2049, 9) * step
    phi = np.concatenate([BELOW, ABOVE, k, np.nextafter(k + 0.5 * step, 10), np.arange(17) * np.pi / 4,
                          rng.uniform(0, 2e4, 600), rng.uniform(0, 1e9, 200)])
    phi = np.concatenate([phi, -phi])
    mp.mp.prec = 200
    for which, m in enumerate(ms):
        got = _run(phi, ms, which)
        ref = np.array([complex(mp.expj(-m * mp.mpf(float(p)))) for p in phi])
        big = np.abs(phi) >= 2.0 ** 40
        bound = np.where(big, 2.0 ** -52 + abs(m) * np.abs(phi) * 2.0 ** -53,
                         2.0 ** -53 + 2.0 ** -59.6 + 2 * np.pi * abs(m) * 2.0 ** -64)
        assert np.all(np.abs(got.real - ref.real) <= bound), m
        assert np.all(np.abs(got.imag - ref.imag) <= bound), m


def test_phases_that_are_no_numbers():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    got = _run(np.array([np.inf, -np.inf, np.nan, 1.0]), (2, 1), 0)
    assert np.array_equal(np.isnan(got.real), [True, True, True, False])
