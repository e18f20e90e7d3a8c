"""The waveform path's table-driven sincos, read through TDInterp_wrap2 (one
mode of amplitude 1 with constant phase splines returns e^{-i m phi}), against
extended precision: around zero, on both sides of the table's steps and of the
quadrants, at phases of long inspirals, and where it turns to the library.

Bound: two table roundings (5.6e-17 each) and three of the sums (1.1e-16 / 2 each at
values up to 1), single-precision terms 1e-16: 3.3e-16 absolute."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 5])
def test_sincos_against_extended_precision(m):
    torch = pytest.importorskip("torch")
    mp = pytest.importorskip("mpmath")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300.eob import pytdinterp
    rng = np.random.default_rng(m)
    step = 2 * np.pi / 2048
    k = np.arange(0, 2049, 3) * step / m
    phi = np.concatenate([[0.0, 1e-300, 1e-40, 5e-39, 1e-20, 1e-8], k, np.nextafter(k + 0.5 * step / m, 10),
                          np.nextafter(k + 0.5 * step / m, 0), np.arange(17) * np.pi / 4, rng.uniform(0, 2e4, 4000),
                          rng.uniform(0, 1e9, 500), 2.0 ** 40 + np.arange(5.0), [2.0 ** 39, 2.0 ** 41, 1e15]])
    phi = np.concatenate([phi, -phi])
    n = len(phi)
    d = lambda a, t=torch.float64: torch.tensor(np.ascontiguousarray(a), dtype=t, device="cuda")
    y = np.concatenate([np.ones(n), np.zeros(n), phi])
    zero = d(np.zeros(3 * n))
    one = lambda v: d([v], torch.int32)
    out = torch.zeros(n, dtype=torch.complex128, device="cuda")
    pytdinterp.TDInterp_wrap2(out, d(np.zeros(n)), d(np.zeros(n)), d(y), zero, zero, zero, n, one(n), n, 1, 1, one(2),
                              one(m), d(np.arange(n), torch.int32), one(n), n)
    got = out.cpu().numpy()
    ph = np.float64(m) * phi  # the product is rounded once on either side
    mp.mp.prec = 200
    ref = np.array([complex(mp.expj(-mp.mpf(float(p)))) for p in ph])
    assert np.max(np.abs(got.real - ref.real)) <= 3.3e-16
    assert np.max(np.abs(got.imag - ref.imag)) <= 3.3e-16


def test_sincos_of_non_finite_phases():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from eobgpu_gb300.eob import pytdinterp
    phi = np.array([np.inf, -np.inf, np.nan, 1.0])
    n = len(phi)
    d = lambda a, t=torch.float64: torch.tensor(np.ascontiguousarray(a), dtype=t, device="cuda")
    one = lambda v: d([v], torch.int32)
    zero = d(np.zeros(3 * n))
    out = torch.zeros(n, dtype=torch.complex128, device="cuda")
    pytdinterp.TDInterp_wrap2(out, d(np.zeros(n)), d(np.zeros(n)), d(np.concatenate([np.ones(n), np.zeros(n), phi])),
                              zero, zero, zero, n, one(n), n, 1, 1, one(2), one(2), d(np.arange(n), torch.int32),
                              one(n), n)
    assert np.array_equal(np.isnan(out.cpu().numpy().real), [True, True, True, False])
