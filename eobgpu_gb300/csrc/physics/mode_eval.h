// Factorized waveform multipole h_lm on a trajectory point.
//
// Restates EOBGetSpinFactorizedWaveform (src/EOB.cu:1235-1613):
//   h_lm = T_lm e^{i delta_lm} S_lm (rho_lm^l + f_lm) h^N_lm,
//   T_lm = Gamma(l + 1 - 2 i k) / l! e^{pi k} e^{2 i k log(4 m Omega / sqrt(e))},
//   k = m H_real Omega,  h^N_lm = n_lm vPhi^(l+eps) Y_{l-eps}^{-m}(pi/2, phi).
//
// Written for FP64 issue rate: what the modes of a row share (log v, powers,
// S of either parity) is formed once (ModeRow), and T_lm has no logarithm or
// arctangent of its own.  With y = 2 k,
//   |Gamma(l + 1 - i y)|^2 e^{pi y} = prod_{j<=l} (j^2 + y^2) 2 pi y / (1 - e^{-2 pi y})
// (A&S 6.1.31, the closed form of the flux; y = m y_1, so one exponential serves
// every mode of a row, and one reciprocal square root its quotient's root), and arg Gamma(l + 1 - i y) =
// -y P_l(y^2 / (l + 1)^2) with a polynomial per l (fasttrig.h) for
// y <= 0.9 (l + 1), which every frequency of an inspiral meets (y < 2 m
// Omega, Omega < 0.45).  Larger y go through the complex log Gamma: an
// upward shift by the recurrence (A&S 6.1.15) and the Stirling series (A&S
// 6.1.40) at Re(z) >= 16; only exp() of it is used, so the branch of its
// logarithm does not matter.  The reference's SciPy-derived loggamma is not
// used.
//
// mode_eval_sums is the evaluation by the sums of log Gamma throughout, for tables of use_hm = 1.  They
// cancel from ~30 to order one and leave 4e-15 of rounding in the modulus (rms
// against 40 digits; 1.5e-15 the closed form).  On close rows (the fine pass, 0.05 M
// apart and less, and the end of the main pass) the third differences of the spline amplify
// rounding by 1e4 to 1e8, so that their c3 is rounding: 4e-15 of the modulus are up to 6e-8 of
// its norm.  k_modes leaves rows less than 0.2 M from a neighbour (4 in 10) to the sums, so that the tables
// do not move with the evaluation of the others; a change of one last bit in the
// sums (an arctangent by its series, logarithms shared by the modes) moves them too.
// With derotate = true the result is multiplied by e^{i m phi}: the
// e^{-i m phi} of the spherical harmonic is simply not applied, which is what
// the spline inputs of the synthesis need (eob/seobnrv4phm.py:2331).
#pragma once
#include "fac_coeffs.h"
#include "fasttrig.h"
#include "flux_eval.h"

namespace eob {

struct cdbl {
    double re, im;
};
EOB_HD cdbl cmul(cdbl a, cdbl b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }

// log Gamma(z) + log(prod shift) pieces: returns log|Gamma(z)| and arg Gamma(z) (mod 2 pi)
EOB_HD void cloggamma_shifted(double zr, double zi, double *lg_re, double *lg_im)
{
    // shift product P = prod (z + j) until Re(z) >= 16
    double pr = 1.0, pim = 0.0;
    while (zr < 16.0) {
        const double t = pr * zr - pim * zi;
        pim = pr * zi + pim * zr;
        pr = t;
        zr += 1.0;
    }
    // 1/w and 1/w^2
    const double den = 1.0 / (zr * zr + zi * zi);
    const double ir = zr * den, ii = -zi * den;
    const double i2r = ir * ir - ii * ii, i2i = 2.0 * ir * ii;
    // sum_k c_k w^{-(2k-1)}, c_k = B_2k / (2k (2k - 1)), k = 1..8, Horner in 1/w^2
    const double c[8] = {1.0 / 12.0, -1.0 / 360.0, 1.0 / 1260.0, -1.0 / 1680.0,
                         1.0 / 1188.0, -691.0 / 360360.0, 1.0 / 156.0, -3617.0 / 122400.0};
    double sr = c[7], si = 0.0;
    for (int k = 6; k >= 0; --k) {
        const double t = sr * i2r - si * i2i + c[k];
        si = sr * i2i + si * i2r;
        sr = t;
    }
    const double tr = sr * ir - si * ii;
    const double ti = sr * ii + si * ir;
    // (w - 1/2) log w - w + log(2 pi)/2
    const double lmod = 0.5 * log(zr * zr + zi * zi);
    const double larg = atan2(zi, zr);
    const double ar = zr - 0.5;
    double re = ar * lmod - zi * larg - zr + 0.91893853320467274178 + tr;
    double im = ar * larg + zi * lmod - zi + ti;
    // divide by P
    re -= 0.5 * log(pr * pr + pim * pim);
    im -= atan2(pim, pr);
    *lg_re = re;
    *lg_im = im;
}

// h_lm (or h_lm e^{i m phi} when derotate) with T_lm from the sums of log Gamma, exp() and the
// library's logarithms.  vh = (H_real v^3)^(1/3), y0 = (-1)^m Y_{l-eps}^m(pi/2, 0),
// lfact = log(l!), i = lm_index(l, m)
EOB_HD cdbl mode_eval_sums(const FacCoeffs &fc, int l, int m, double pre_re, double pre_im, double eta, double phi,
                           double pphi, double v, double vh, double Hreal, double vPhi, double y0, double lfact,
                           double h22_calib,
                           bool derotate)
{
    if (eta > 0.25 && eta < 0.25 + 1e-4) eta = 0.25;
    const int i = lm_index(l, m);
    const double v2 = v * v;
    const double Omega = v2 * v;
    const double vh3 = Hreal * Omega;
    const double eulerlog = kEulerGamma + log(2.0 * m * v);
    const int eps = (l + m) % 2;
    // |Y| part and Newtonian amplitude: n_lm vPhi^(l+eps) (-1)^m Y_{l-eps}^m(pi/2, 0)
    double vpow = 1.0;
    for (int q = 0; q < l + eps; ++q) vpow *= vPhi;
    const double S = (eps == 0) ? (Hreal * Hreal - 1.0) / (2.0 * eta) + 1.0 : v * pphi;
    // delta_lm
    // (the builder assigns vh^3, vh^6, vh^9 and v^5 only; the powers by one product each, as ever)
    double p = vh * vh * vh;
    double delta = fc.dvh[i][3] * p;
    p = p * vh * vh * vh;
    delta = fma(fc.dvh[i][6], p, delta);
    p = p * vh * vh * vh;
    delta = fma(fc.dvh[i][9], p, delta);
    p = v * v * v * v * v;
    delta = fma(fc.dv[i][5], p, delta);
    // rho_lm^l + f_lm
    double rho = 0.0;
#pragma unroll
    for (int k = 10; k >= 1; --k)
        rho = (rho + ((k == 6 || k == 8 || k == 10) ? fma(fc.rhol[i][k], eulerlog, fc.rho[i][k]) : fc.rho[i][k])) * v;
    rho += 1.0;
    if (l == 2 && m == 2) {
        const double v4 = v2 * v2;
        rho = fma(h22_calib, v4 * v4 * v4, rho);
    }
    double rpl = rho;
    for (int q = 1; q < l; ++q) rpl *= rho;
    double fr = 0.0;
    if (l <= 5) {  // f from v^1 and v^3 .. v^6
        fr = fc.fre[i][1] * v;
        p = v * v * v;
        fr = fma(fc.fre[i][3], p, fr);
#pragma unroll
        for (int k = 4; k <= 6; ++k) {
            p *= v;
            fr = fma(fc.fre[i][k], p, fr);
        }
    }
    const double fi = fc.fim_vh6[i] * vh3 * vh3;
    cdbl rf = {rpl + fr, fi};
    if (eta == 0.25 && (m % 2)) rf = {fr, fi};
    // T_lm
    const double k = m * Omega;
    const double hk = Hreal * k;
    double lgr, lgi;
    cloggamma_shifted(l + 1.0, -2.0 * hk, &lgr, &lgi);
    const double tmod = kPi * hk + lgr - lfact;
    double phase = 2.0 * hk * log(4.0 * k / 1.6487212707001281468) + lgi + delta;  // sqrt(e)
    if (!derotate) phase -= m * phi;
    double sp, cp;
    sincos(phase, &sp, &cp);
    const double amp = exp(tmod) * S * vpow * y0;
    const cdbl e = {amp * cp, amp * sp};
    return cmul(cmul(e, rf), cdbl{pre_re, pre_im});
}

// either zero, by its bits (a comparison of doubles takes an FP64 issue slot)
EOB_HD bool is_zero(double x)
{
#ifdef __CUDA_ARCH__
    return (__double_as_longlong(x) << 1) == 0;
#else
    return x == 0.0;
#endif
}

// What the modes of one trajectory point share.
struct ModeRow {
    double v, v2, lv;   // omega^(1/3), its square and its logarithm
    double vh3;         // H_real v^3
    double vh6, y1;     // its square and double
    double E1;          // 1 - e^{-2 pi y1}
    double vPhi, vPhi2, vPhi4;
    double Se, So;      // source terms of even and odd l + m
    double phi;
};

EOB_HD ModeRow mode_row(double v, double Hreal, double vPhi, double pphi, double inv2eta, double phi)
{
    ModeRow w;
    w.v = v;
    w.v2 = v * v;
    w.lv = eob_log(v);
    w.vh3 = Hreal * (w.v2 * v);
    w.vh6 = w.vh3 * w.vh3;
    w.y1 = 2.0 * w.vh3;
    w.E1 = -eob_expm1_neg((2.0 * kPi) * w.y1);
    w.vPhi = vPhi;
    w.vPhi2 = vPhi * vPhi;
    w.vPhi4 = w.vPhi2 * w.vPhi2;
    w.Se = fma(fma(Hreal, Hreal, -1.0), inv2eta, 1.0);
    w.So = v * pphi;
    w.phi = phi;
    return w;
}

// 1 - e^{-m x} from E1 = 1 - e^{-x}: 1 - (1 - a)(1 - b) = a + b - a b, no cancellation
EOB_HD double mode_expm(int m, double E1)
{
    if (m == 1) return E1;
    const double E2 = fma(E1, -E1, E1 + E1);
    if (m == 2) return E2;
    if (m == 3) return fma(E2, -E1, E2 + E1);
    const double E4 = fma(E2, -E2, E2 + E2);
    double e = E4;
    if (m == 8) e = fma(E4, -E4, E4 + E4);
    else {
        if (m & 2) e = fma(e, -E2, e + E2);
        if (m & 1) e = fma(e, -E1, e + E1);
    }
    return e;
}

// What depends on (l, m) alone.
struct ModeConst {
    double elog;   // gamma + log(2 m)
    double tail;   // log(4 m / sqrt(e))
    double y0;     // (-1)^m Y_{l-eps}^m(pi/2, 0)
    double m, il;  // m, 1 / (l + 1)
    double g[kLMax + 1];  // 2 pi prod_{j<=l} (1 + z / j^2), ascending in z
};

EOB_HD ModeConst mode_const(int l, int m)
{
    ModeConst c;
    c.elog = kEulerGamma + log(2.0 * m);
    c.tail = log(4.0 * m / 1.6487212707001281468);  // sqrt(e)
    c.y0 = ((m % 2) ? -1.0 : 1.0) * ylm_equator(l - (l + m) % 2, m);
    c.m = (double)m;
    c.il = 1.0 / (l + 1);
    for (int q = 0; q <= kLMax; ++q) c.g[q] = (q == 0) ? 1.0 : 0.0;
    double d = 2.0 * kPi;
    for (int j = 1; j <= l; ++j) {  // prod (j^2 + z), integers, then over (l!)^2
        for (int q = j; q >= 0; --q) c.g[q] = c.g[q] * (j * j) + (q > 0 ? c.g[q - 1] : 0.0);
        d /= (double)(j * j);
    }
    for (int q = 0; q <= l; ++q) c.g[q] *= d;
    return c;
}

// h_lm (or h_lm e^{i m phi} when derotate). i = lm_index(l, m).  HM: the table
// was built with use_hm = 1, which leaves the odd powers of v in rho_lm (and the
// logarithm beside v^7) to a few modes; otherwise a = tplspin brings them to
// most modes and the whole series is summed.
template <bool HM>
EOB_HD cdbl mode_term(const FacCoeffs &fc, int l, int m, const ModeConst &mc, const ModeRow &w, double pre_re,
                      double pre_im, double eta, double h22_calib, bool derotate)
{
    if (eta > 0.25 && eta < 0.25 + 1e-4) eta = 0.25;
    const int i = lm_index(l, m);
    const int eps = (l + m) % 2;
    const double v = w.v, v2 = w.v2, vh3 = w.vh3;
    // delta_lm: the builder assigns vh^3, vh^6, vh^9 and v^5 only
    double delta = vh3 * fma(vh3, fma(vh3, fc.dvh[i][9], fc.dvh[i][6]), fc.dvh[i][3]);
    delta = fma(fc.dv[i][5], v2 * v2 * v, delta);
    // rho_lm^l + f_lm (rho up to v^10, eulerlog parts at v^6, v^8, v^10 and, without HM, v^7; f for odd m <= 5, from
    // v^1 and v^3..v^6)
    const double el = mc.elog + w.lv;
    const double c10 = fma(fc.rhol[i][10], el, fc.rho[i][10]), c8 = fma(fc.rhol[i][8], el, fc.rho[i][8]),
                 c6 = fma(fc.rhol[i][6], el, fc.rho[i][6]);
    double rho;
    if (!HM || (l == m && (l & 1) == 0) || (l == 3 && m == 2) || (l == 4 && m == 2)) {
        // odd powers too
        const double *c = fc.rho[i];
        const double c7 = HM ? c[7] : fma(fc.rhol[i][7], el, c[7]);
        rho = fma(fma(c10, v, c[9]), v, c8);
        rho = fma(fma(rho, v, c7), v, c6);
        rho = fma(fma(rho, v, c[5]), v, c[4]);
        rho = fma(fma(rho, v, c[3]), v, c[2]);
        rho = fma(rho, v, c[1]) * v;
    } else {
        rho = fma(fma(fma(fma(c10, v2, c8), v2, c6), v2, fc.rho[i][4]), v2, fc.rho[i][2]) * v2;
    }
    rho += 1.0;
    if (l == 2 && m == 2) {
        const double v4 = v2 * v2;
        rho = fma(h22_calib, v4 * v4 * v4, rho);
    }
    const double rho2 = rho * rho;
    double rpl = (l & 1) ? rho * rho2 : rho2;  // l = 2, 3
    if (l >= 4) rpl *= rho2;
    if (l >= 6) rpl *= rho2;
    if (l >= 8) rpl *= rho2;
    double fi = 0.0;
    if ((m & 1) && l <= 5) {
        const double *f = fc.fre[i];
        const double fr = v * fma(v2, fma(v, fma(v, fma(v, f[6], f[5]), f[4]), f[3]), f[1]);
        fi = fc.fim_vh6[i] * w.vh6;
        rpl = (eta == 0.25) ? fr : rpl + fr;
    } else if (m & 1) {
        rpl = (eta == 0.25) ? 0.0 : rpl;
    }
    // |T_lm|: sqrt(a / E), and its phase without the logarithm's term
    const double y = mc.m * w.y1;
    double tmod, targ;
    const double q = y * mc.il, z = q * q;
    if (y >= 0.0 && z <= EOB_ARG_GAMMA_ZMAX) {
        targ = -y * (z <= EOB_ARG_GAMMA_ZLOW ? arg_gamma_over_y_low(l, z) : arg_gamma_over_y(l, z));
        const double y2 = y * y;
        double a = mc.g[l];
        for (int j = l - 1; j >= 0; --j) a = fma(a, y2, mc.g[j]);
        a *= y;
#ifdef __CUDA_ARCH__
        tmod = a * eob_rsqrt(a * mode_expm(m, w.E1));
#else
        tmod = sqrt(a / mode_expm(m, w.E1));
#endif
    } else {
        double lgr;
        cloggamma_shifted(l + 1.0, -y, &lgr, &targ);
        tmod = exp(fma(0.5 * kPi, y, lgr)) * sqrt(mc.g[l] * (1.0 / (2.0 * kPi)));  // g[l] = 2 pi / (l!)^2
    }
    double phase = fma(y, fma(3.0, w.lv, mc.tail), targ) + delta;
    if (!derotate) phase -= mc.m * w.phi;
    double sp, cp;
    eob_sincos(phase, &sp, &cp);
    double amp = tmod * mc.y0 * (eps ? w.So : w.Se);
    const int e = l + eps;
    if (e & 1) amp *= w.vPhi;
    if (e & 2) amp *= w.vPhi2;
    if (e & 4) amp *= w.vPhi4;
    if (e & 8) amp *= w.vPhi4 * w.vPhi4;
    // times the Newtonian prefix, real or imaginary for the reference's own, and rpl + i fi
    const bool real = is_zero(pre_im), imag = is_zero(pre_re);
    if (real || imag) amp *= real ? pre_re : pre_im;
    cdbl h;
    if (l == 3 && m == 3) {  // the one mode with an imaginary part of f
        h = cmul(cdbl{amp * cp, amp * sp}, cdbl{rpl, fi});
    } else {
        amp *= rpl;
        h = cdbl{amp * cp, amp * sp};
    }
    if (real) return h;
    if (imag) return cdbl{-h.im, h.re};
    return cmul(h, cdbl{pre_re, pre_im});
}

// the same from the reference's arguments (vPhiInput = 1 / (omega_c^2 r^3)), for a table of either use_hm
EOB_HD cdbl mode_eval(const FacCoeffs &fc, int l, int m, double pre_re, double pre_im, double eta, double r, double phi,
                      double pphi, double v, double Hreal, double vPhiInput, double h22_calib, bool derotate)
{
    const double e4 = (eta > 0.25 && eta < 0.25 + 1e-4) ? 0.25 : eta;
    const ModeRow w = mode_row(v, Hreal, r * cbrt(vPhiInput) * (v * v * v), pphi, 0.5 / e4, phi);
    return mode_term<false>(fc, l, m, mode_const(l, m), w, pre_re, pre_im, eta, h22_calib, derotate);
}

}  // namespace eob
