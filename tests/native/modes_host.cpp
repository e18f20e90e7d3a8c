// Host build of the multipole evaluation (eobgpu_gb300/csrc/physics/mode_eval.h)
// for CPU tests.
#include "../../eobgpu_gb300/csrc/physics/mode_eval.h"

extern "C" {

// par: m1, m2 (units of the total mass), eta, tplspin, chiS, chiA; row[n][6]: r, phi, pphi, v,
// Hreal, vPhi input; out[35][n] complex, (l, m) in the table's order, with the
// table's own equal-mass clamp of eta and unit prefix
void modes_eval(const double *par, int use_hm, const double *row, int n, double h22, double *out)
{
    eob::FacCoeffs fc;
    eob::fac_coeffs_build(&fc, use_hm, par[0], par[1], par[2], par[3], par[4], par[5]);
    for (int l = 2; l <= eob::kLMax; ++l)
        for (int m = 1; m <= l; ++m)
            for (int i = 0; i < n; ++i) {
                const double *q = row + 6 * i;
                const eob::cdbl h = eob::mode_eval(fc, l, m, 1.0, 0.0, par[2], q[0], q[1], q[2], q[3], q[4], q[5], h22,
                                                   false);
                double *o = out + 2 * ((long)eob::lm_index(l, m) * n + i);
                o[0] = h.re;
                o[1] = h.im;
            }
}

}  // extern "C"
