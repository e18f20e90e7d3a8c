"""Points at which the multipoles of every (l, m), l <= 8, are compared with
the oracle: spinning binaries of equal and unequal masses, both coefficient
settings (use_hm = 0 keeps the test-particle spin terms of the higher modes,
odd powers of v among them), from a wide orbit to v = 0.6.

h_lm is a product of sums; the largest rounding is that of (rho_lm^l + f_lm):
rho's terms reach ~10 at v = 0.6 and the power 8 multiplies their relative
rounding, so each side is good to 8 x 20 terms x 2^-53 x 10 = 2e-13: 1e-12 of each
mode's peak over the points is allowed."""
import numpy as np

LM = [(l, m) for l in range(2, 9) for m in range(1, l + 1)]
BINARIES = [(0.5, 0.4, 0.4), (0.5, 0.6, -0.3), (0.75, 0.7, -0.5), (0.8571428571428571, -0.8, 0.3)]  # m1, chi1, chi2


def params(m1, chi1, chi2):
    m2 = 1.0 - m1
    eta = m1 * m2
    chiS, chiA = (chi1 + chi2) / 2, (chi1 - chi2) / 2
    return np.array([m1, m2, eta, (1 - 2 * eta) * chiS + (m1 - m2) * chiA, chiS, chiA])


def rows():
    """(r, phi, pphi, v, Hreal, vPhi input) on orbits of increasing frequency."""
    v = np.array([0.15, 0.25, 0.33, 0.4, 0.5, 0.6])
    r = 1.0 / v ** 2
    return np.ascontiguousarray(np.stack([r, np.linspace(0.0, 30.0, len(v)), 1.0 / v * (1 + 1.5 * v * v), v,
                                          1.0 - 0.02 * v, 1.0 + 0.1 * v * v], axis=1))


def oracle_modes(oracle, m1, chi1, chi2, use_hm, h22=0.3):
    """h_lm [35][n] with unit prefix."""
    ctx = oracle.context(np.array([m1]), np.array([1.0 - m1]), np.array([chi1]), np.array([chi2]), use_hm)
    q = rows()
    eta = params(m1, chi1, chi2)[2]
    return np.array([ctx.waveform(q[:, 0], q[:, 1], 0 * q[:, 0], q[:, 2], q[:, 3], q[:, 4], eta, q[:, 5], l, m, 1.0, h22)
                     for l, m in LM])
