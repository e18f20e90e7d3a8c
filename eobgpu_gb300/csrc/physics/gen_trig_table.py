"""Write trig_table.h: the tables of eob_sincos and of the Gamma phase.

kSinFix[i] = sin(2 pi i / 2048) in units of 2^-61, i = 0..512 (a quarter wave;
the cosine is read backwards).

kArgGamma[l - 2][k]: coefficients, in z = (y / (l + 1))^2, of a polynomial for
arg Gamma(l + 1 + i y) / y on 0 <= z <= 0.81, l = 2..8.  The function is
analytic there (nearest singularity z = -1, the pole of Gamma at 0), so the
Chebyshev interpolant of degree 19 is within 3e-17 of it, relative to its
value; it is converted to powers of z at 60 digits.  kArgGammaLow: the same on
0 <= z <= 0.125, where most of an inspiral lies, of degree 10.

Values come from mpmath; the output is hexadecimal floating point, so the
header is the same on every machine.

    python gen_trig_table.py > trig_table.h
"""
import mpmath as mp

mp.mp.dps = 60
DEG, ZMAX = 19, mp.mpf("0.81")
DEG_LOW, ZLOW = 10, mp.mpf("0.125")


def arg_gamma_over_y(l, z):
    y = mp.sqrt(z) * (l + 1)
    if y < mp.mpf("1e-20"):
        return mp.psi(0, l + 1)
    return mp.im(mp.loggamma(mp.mpc(l + 1, y))) / y


def fit(f, n, zmax, tol):
    """Coefficients in powers of z of the Chebyshev interpolant of f on [0, zmax] at n nodes."""
    nodes = [mp.cos(mp.pi * (2 * j + 1) / (2 * n)) for j in range(n)]
    fv = [f((x + 1) / 2 * zmax) for x in nodes]
    cheb = [mp.mpf(2 if k else 1) / n * sum(fv[j] * mp.cos(k * mp.pi * (2 * j + 1) / (2 * n)) for j in range(n))
            for k in range(n)]
    # Chebyshev series in x -> powers of x -> powers of z, x = 2 z / zmax - 1
    t0, t1 = [mp.mpf(1)], [mp.mpf(0), mp.mpf(1)]
    px = [mp.mpf(0)] * n
    for k in range(n):
        t = t0 if k == 0 else t1
        for i, c in enumerate(t):
            px[i] += cheb[k] * c
        if k >= 1:
            t2 = [mp.mpf(0)] + [2 * c for c in t1]
            for i, c in enumerate(t0):
                t2[i] -= c
            t0, t1 = t1, t2
    pz = [mp.mpf(0)] * n
    for i, c in enumerate(px):  # c (2 z / zmax - 1)^i
        for j in range(i + 1):
            pz[j] += c * mp.binomial(i, j) * (2 / zmax) ** j * (-1) ** (i - j)
    err = max(abs(mp.polyval(pz[::-1], z) / f(z) - 1) for z in [zmax * q / 200 for q in range(201)])
    assert err < tol, err
    return pz


def coefficients(l, deg, zmax):
    return fit(lambda z: arg_gamma_over_y(l, z), deg + 1, zmax, mp.mpf("3e-17"))


def row(v, per=4):
    v = [x if isinstance(x, str) else float(x).hex() for x in v]
    return ",\n    ".join(", ".join(v[i:i + per]) for i in range(0, len(v), per))


def main():
    print("// Written by gen_trig_table.py: quarter-wave sine table and Gamma-phase polynomials.")
    print("#pragma once")
    step = 2 * mp.pi / 2048
    print("#define EOB_SINFIX_INIT { \\\n    "
          + row([hex(int(mp.nint(mp.sin(step * i) * 2 ** 61))) + "ll" for i in range(513)]).replace("\n", " \\\n") + "}")
    for tag, deg, zmax in (("", DEG, ZMAX), ("_LOW", DEG_LOW, ZLOW)):
        rows = ["{" + row(coefficients(l, deg, zmax)).replace("\n", " \\\n") + "}" for l in range(2, 9)]
        print(f"#define EOB_ARG_GAMMA{tag}_N {deg + 1}")
        print(f"#define EOB_ARG_GAMMA_Z{tag[1:] or 'MAX'} {float(zmax)!r}")
        print(f"#define EOB_ARG_GAMMA{tag}_INIT {{ \\\n    " + ", \\\n    ".join(rows) + "}")


main()
