// Not-a-knot cubic splines of many series on the same knots, one thread block
// per group of binaries (the reference's tridiagonal slope system,
// src/interpolate.cu:10-267).
//
// The matrix depends on the knots alone, so a block factorises it once and
// every series of the binary then costs two linear recurrences.  Both the
// factorisation and the recurrences are scans:
//
//   rows      a_i m_{i-1} + b_i m_i + c_i m_{i+1} = d_i, normalised by b_i
//   diagonal  delta_i = 1 - u_i / delta_{i-1}, u_i = a_i c_{i-1} / (b_i b_{i-1}):
//             the ratio of the continuants p_i = p_{i-1} - u_i p_{i-2}, a scan
//             of 2 x 2 matrices
//   forward   e_i = (d_i - a_i e_{i-1}) / (b_i delta_i)       affine scan
//   backward  m_i = e_i - c_i m_{i+1} / (b_i delta_i)         affine scan
//
// Each thread owns r consecutive rows and carries their factors in registers;
// a chunk's affine map is composed over the block by shuffles (and over its
// warps through shared memory), then the chunk is run once more from its true
// inflow.  Global memory is touched row by row across the threads (coalesced):
// interval slopes go to shared memory on the way in, the solution on the way
// out.  FP64 issue bounds it (GB300 takes one FP64 instruction per 64 cycles
// and SM sub-partition): 16 FP64 instructions per row and series plus about 22
// per thread and series, against 112 when each series eliminated the matrix
// for itself with three right-hand sides and five divisions a row.
//
// NB binaries share a block of NT threads (thread = chunk * NB + binary);
// P = NT / NB chunks of at most RM rows make a tile.  Longer trajectories run
// tile after tile: the inverse pivots and the forward sums are then kept in
// planes that the outputs of the same rows overwrite last.  r depends on the
// binary's own length only, so its coefficients do not depend on the batch.
#pragma once
#include "physics/ham_eval.h"

namespace eob {

struct SplineSeries {
    const double *y;
    double *c1, *c2, *c3;  // outputs
    double *cd;            // scratch: forward sums; the slopes m where the caller keeps them
};

template <int NB, int NT, int RM>
struct SplineBlock {
    static_assert(RM % 2 == 1, "odd chunks: threads' rows fall in different shared-memory banks");
    static constexpr int P = NT / NB, NW = NT / 32, CW = 32 / NB;
    static constexpr int kSteps = (CW == 32) ? 5 : (CW == 16) ? 4 : (CW == 8) ? 3 : 2;
    static constexpr int kTile = P * RM;
    // leading dimension of a binary's rows: 4 mod 16, so that the NB
    // binaries of a half-warp use different banks too
    static constexpr int LD = ((kTile + 4 + 15) / 16) * 16 + 4;

    struct Smem {
        double h[NB * LD];   // interval lengths, row k of the tile at [k + 2]
        double rh[NB * LD];  // their reciprocals
        double s[NB * LD];   // slopes (y_{i+1} - y_i) / h_i
        double m[NB * LD];   // solution
        double wt[4][NW][NB];  // warp totals of the continuant matrices
        double fa[NW][NB], fb[NW][NB];  // forward scan: factor and sum of each warp
        double ba[NW][NB], bb[NW][NB];  // backward scan
        double carry[NB], diag[NB];
    };

    template <class Acc>
    static __device__ __forceinline__ double inverse(double h)
    {
        return Acc::kExact ? 1.0 / h : eob_rcp(h);
    }

    template <class Acc>
    static __device__ void run(const Acc &acc, Smem &sm, int s_begin, int s_end)
    {
        const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
        const int bl = tid % NB, c = tid / NB, cw = lane / NB;
        const int n = acc.rows(bl);
        const int T = (n + kTile - 1) / kTile;
        const int r = (n > 0) ? (((n + P * T - 1) / (P * T)) | 1) : 1;
        int Tmax = T;
        if constexpr (NB > 1) {
#pragma unroll
            for (int off = 1; off < NB; off <<= 1) Tmax = max(Tmax, __shfl_xor_sync(0xffffffffu, Tmax, off));
        }
        if (Tmax == 0) return;
        double *h = sm.h + bl * LD + 2, *rh = sm.rh + bl * LD + 2, *sl = sm.s + bl * LD + 2, *ms = sm.m + bl * LD;
        const double *x = acc.knots(bl);
        const size_t xst = acc.knot_stride(), st = acc.row_stride();
        double *ibp = acc.series(bl, s_end - 1).c1;  // inverse pivots between the sweeps (several tiles only)

        double al[RM], be[RM], A[RM], C[RM], e[RM];
        double fA[kSteps], bA[kSteps], fE = 1.0, bE = 1.0;  // scan factors of the two recurrences

        // interval lengths and reciprocals of the tile's rows (two rows of halo
        // before it); every load of a thread is issued before the first is used
        auto load_knots = [&](int base0) {
            double u[RM], v[RM];
#pragma unroll
            for (int q = 0; q < RM; ++q) {
                const int i = base0 + c + P * q;
                const bool in = q < r && i < n - 1;
                u[q] = in ? __ldg(x + (size_t)i * xst) : 0.0;
                v[q] = in ? __ldg(x + (size_t)(i + 1) * xst) : 1.0;
            }
#pragma unroll
            for (int q = 0; q < RM; ++q)
                if (q < r) {
                    const bool in = base0 + c + P * q < n - 1;
                    const double hv = v[q] - u[q];
                    h[c + P * q] = in ? hv : 0.0;
                    rh[c + P * q] = in ? inverse<Acc>(hv) : 0.0;
                }
            if (c < 2) {
                const int i = base0 + c - 2;
                const bool in = i >= 0 && i < n - 1;
                const double hv = in ? x[(size_t)(i + 1) * xst] - x[(size_t)i * xst] : 0.0;
                h[c - 2] = hv;
                rh[c - 2] = in ? inverse<Acc>(hv) : 0.0;
            }
            __syncthreads();
        };
        // a, b, c of row i from the intervals around it
        auto row_abc = [&](int i, double hm2, double hm1, double h0, double h1, double *a, double *b, double *cc) {
            const bool first = (i == 0), last = (i == n - 1);
            const double two = last ? hm2 + hm1 : (first ? h0 + h1 : hm1 + h0);
            *a = first ? 0.0 : (last ? two : h0);
            *b = first ? h1 : (last ? hm2 : 2.0 * two);
            *cc = first ? two : (last ? 0.0 : hm1);
        };
        // factors of the chunk's rows from the inverse pivot ib[j] (in e[j])
        auto weights = [&](int base0) {
#pragma unroll
            for (int j = 0; j < RM; ++j) {
                const int k = c * r + j, i = base0 + k;
                if (j < r && i < n) {
                    const double hm2 = h[k - 2], hm1 = h[k - 1], h0 = h[k], h1 = h[k + 1];
                    const double ib = e[j], ib3 = 3.0 * ib;
                    double a, b, cc;
                    row_abc(i, hm2, hm1, h0, h1, &a, &b, &cc);
                    A[j] = -a * ib;
                    C[j] = -cc * ib;
                    al[j] = h0 * ib3;
                    be[j] = hm1 * ib3;
                    if (i == 0) {
                        const double d = h0 + h1;
                        al[j] = (h0 + 2 * d) * h1 / d * ib;
                        be[j] = h0 * h0 / d * ib;
                    } else if (i == n - 1) {
                        const double d = hm2 + hm1;
                        al[j] = hm1 * hm1 / d * ib;
                        be[j] = (2 * d + hm1) * hm2 / d * ib;
                    }
                } else {
                    A[j] = C[j] = al[j] = be[j] = 0.0;
                }
            }
        };
        // composed factors of the two recurrences over the block
        auto scan_factors = [&]() {
            double pa = A[0], pc = C[0];
#pragma unroll
            for (int j = 1; j < RM; ++j)
                if (j < r) {
                    pa *= A[j];
                    pc *= C[j];
                }
#pragma unroll
            for (int k = 0; k < kSteps; ++k) {
                fA[k] = pa;
                bA[k] = pc;
                const double ua = __shfl_up_sync(0xffffffffu, pa, NB << k);
                const double uc = __shfl_down_sync(0xffffffffu, pc, NB << k);
                if (cw >= (1 << k)) pa *= ua;
                if (cw < CW - (1 << k)) pc *= uc;
            }
            fE = __shfl_up_sync(0xffffffffu, pa, NB);
            bE = __shfl_down_sync(0xffffffffu, pc, NB);
            if (cw == 0) fE = 1.0;
            if (cw == CW - 1) bE = 1.0;
            if (cw == CW - 1) sm.fa[w][bl] = pa;
            if (cw == 0) sm.ba[w][bl] = pc;
            __syncthreads();
        };
        // the inverse pivots of the tile (into e[]), from the one before it (0 for the first tile)
        auto factorise = [&](int base0, double idc) {
            double P1 = 1.0, P2 = 0.0, Q1 = 0.0, Q2 = 1.0, cprev = 0.0, c0 = 0.0, rb0 = 0.0;
            {
                const int k = c * r, i = base0 + k;
                if (i > 0 && i < n) {
                    double a, b;
                    row_abc(i - 1, 0.0, h[k - 2], h[k - 1], h[k], &a, &b, &c0);
                    rb0 = eob_rcp(b);
                    cprev = c0 * rb0;
                }
            }
#pragma unroll
            for (int j = 0; j < RM; ++j) {
                const int k = c * r + j, i = base0 + k;
                if (j < r && i < n) {
                    double a, b, cc;
                    row_abc(i, h[k - 2], h[k - 1], h[k], h[k + 1], &a, &b, &cc);
                    const double rb = eob_rcp(b), u = (a * rb) * cprev;
                    cprev = cc * rb;
                    const double t1 = fma(-u, Q1, P1), t2 = fma(-u, Q2, P2);
                    Q1 = P1;
                    Q2 = P2;
                    P1 = t1;
                    P2 = t2;
                }
            }
            // (p, q)_out = [P1 P2; Q1 Q2] (p, q)_in, composed over the chunks before
            auto before = [&](double p1, double p2, double q1, double q2) {  // this after (p1 p2; q1 q2)
                const double a1 = fma(P1, p1, P2 * q1), a2 = fma(P1, p2, P2 * q2);
                const double b1 = fma(Q1, p1, Q2 * q1), b2 = fma(Q1, p2, Q2 * q2);
                P1 = a1;
                P2 = a2;
                Q1 = b1;
                Q2 = b2;
            };
#pragma unroll
            for (int k = 0; k < kSteps; ++k) {
                const double p1 = __shfl_up_sync(0xffffffffu, P1, NB << k), p2 = __shfl_up_sync(0xffffffffu, P2, NB << k);
                const double q1 = __shfl_up_sync(0xffffffffu, Q1, NB << k), q2 = __shfl_up_sync(0xffffffffu, Q2, NB << k);
                if (cw >= (1 << k)) before(p1, p2, q1, q2);
            }
            if (cw == CW - 1) {
                sm.wt[0][w][bl] = P1;
                sm.wt[1][w][bl] = P2;
                sm.wt[2][w][bl] = Q1;
                sm.wt[3][w][bl] = Q2;
            }
            double p1 = __shfl_up_sync(0xffffffffu, P1, NB), p2 = __shfl_up_sync(0xffffffffu, P2, NB);
            double q1 = __shfl_up_sync(0xffffffffu, Q1, NB), q2 = __shfl_up_sync(0xffffffffu, Q2, NB);
            if (cw == 0) { p1 = q2 = 1.0; p2 = q1 = 0.0; }
            __syncthreads();
            double p = 1.0, q = idc;
            for (int v = 0; v < w; ++v) {
                const double t = fma(sm.wt[0][v][bl], p, sm.wt[1][v][bl] * q);
                q = fma(sm.wt[2][v][bl], p, sm.wt[3][v][bl] * q);
                p = t;
            }
            // 1 / (b delta) of the row before the chunk, then the elimination itself
            // (one rounding less per pivot than 1 / b times 1 / delta)
            double ib = fma(q1, p, q2 * q) / fma(p1, p, p2 * q) * rb0;
#pragma unroll
            for (int j = 0; j < RM; ++j) {
                const int k = c * r + j, i = base0 + k;
                if (j < r && i < n) {
                    double a, b, cc;
                    row_abc(i, h[k - 2], h[k - 1], h[k], h[k + 1], &a, &b, &cc);
                    const double d = fma(-(a * ib), c0, b);
                    ib = eob_rcp(d);
                    e[j] = ib;
                    c0 = cc;
                    rb0 = b;
                    if (i == n - 1) sm.diag[bl] = d;
                }
            }
            if (c == P - 1) sm.carry[bl] = ib * rb0;  // 1 / delta = b / (b delta)
            __syncthreads();
        };
        // slopes of series y on the tile's rows (and its halo): the quotients,
        // corrected by their remainders (a rounded reciprocal alone would add its
        // error to what cancels in the coefficients)
        auto quotient = [&](double d, int k) {
            const double v = d * rh[k];
            return fma(fma(-v, h[k], d), rh[k], v);
        };
        auto load_slopes = [&](int base0, const double *y) {
            double u[RM], v[RM];
#pragma unroll
            for (int q = 0; q < RM; ++q) {
                const int i = base0 + c + P * q;
                const bool in = q < r && i < n - 1;
                u[q] = in ? __ldg(y + (size_t)i * st) : 0.0;
                v[q] = in ? __ldg(y + (size_t)(i + 1) * st) : 0.0;
            }
#pragma unroll
            for (int q = 0; q < RM; ++q)
                if (q < r) sl[c + P * q] = quotient(v[q] - u[q], c + P * q);
            if (c < 2) {
                const int i = base0 + c - 2;
                const bool in = i >= 0 && i < n - 1;
                sl[c - 2] = in ? quotient(y[(size_t)(i + 1) * st] - y[(size_t)i * st], c - 2) : 0.0;
            }
            __syncthreads();
        };
        // forward sums of the chunk into e[], from the sum of the row before the tile
        auto forward = [&](int base0, double in) {
            double B = 0.0;
#pragma unroll
            for (int j = 0; j < RM; ++j)
                if (j < r) {
                    const int k = c * r + j, i = base0 + k;
                    const int sh = (i == 0) ? 1 : ((i == n - 1) ? -1 : 0);
                    e[j] = fma(be[j], sl[k + sh], al[j] * sl[k - 1 + sh]);
                    B = fma(A[j], B, e[j]);
                }
#pragma unroll
            for (int k = 0; k < kSteps; ++k) {
                const double u = __shfl_up_sync(0xffffffffu, B, NB << k);
                if (cw >= (1 << k)) B = fma(fA[k], u, B);
            }
            if (cw == CW - 1) sm.fb[w][bl] = B;
            const double x0 = __shfl_up_sync(0xffffffffu, B, NB);
            __syncthreads();
            double v = in;
            for (int q = 0; q < w; ++q) v = fma(sm.fa[q][bl], v, sm.fb[q][bl]);
            v = fma(fE, v, cw == 0 ? 0.0 : x0);
#pragma unroll
            for (int j = 0; j < RM; ++j)
                if (j < r) {
                    v = fma(A[j], v, e[j]);
                    e[j] = v;
                }
        };
        // the solution of the chunk into shared memory, from that of the row after the tile
        auto backward = [&](double in) {
            double B = 0.0;
#pragma unroll
            for (int j = RM - 1; j >= 0; --j)
                if (j < r) B = fma(C[j], B, e[j]);
#pragma unroll
            for (int k = 0; k < kSteps; ++k) {
                const double u = __shfl_down_sync(0xffffffffu, B, NB << k);
                if (cw < CW - (1 << k)) B = fma(bA[k], u, B);
            }
            if (cw == 0) sm.bb[w][bl] = B;
            const double x0 = __shfl_down_sync(0xffffffffu, B, NB);
            __syncthreads();
            double v = in;
            for (int q = NW - 1; q > w; --q) v = fma(sm.ba[q][bl], v, sm.bb[q][bl]);
            v = fma(bE, v, cw == CW - 1 ? 0.0 : x0);
#pragma unroll
            for (int j = RM - 1; j >= 0; --j)
                if (j < r) {
                    v = fma(C[j], v, e[j]);
                    ms[c * r + j] = v;
                }
            if (c == P - 1) ms[P * r] = in;
            __syncthreads();
        };
        // cubic coefficients of the tile's rows
        auto store = [&](int base0, int s, const SplineSeries &f) {
            for (int q = 0; q < r; ++q) {
                const int k = c + P * q, i = base0 + k;
                if (i >= n) break;
                const double m0 = ms[k];
                if (Acc::kKeepSlopes || Tmax > 1) f.cd[(size_t)i * st] = m0;
                if (i == n - 1) {
                    acc.put_last(bl, s, i, f, m0, sm.diag[bl], h[k - 2] + h[k - 1]);
                    continue;
                }
                const double sv = sl[k], rv = rh[k];
                const double t = (m0 + ms[k + 1] - 2 * sv) * rv;
                acc.put(bl, s, i, f, m0, (sv - m0) * rv - t, t * rv);
            }
            __syncthreads();
        };

        if (Tmax == 1) {
            load_knots(0);
            factorise(0, 0.0);
            weights(0);
            scan_factors();
            for (int s = s_begin; s < s_end; ++s) {
                const SplineSeries f = acc.series(bl, s);
                load_slopes(0, f.y);
                forward(0, 0.0);
                backward(0.0);
                store(0, s, f);
            }
            return;
        }
        // several tiles: forward over the tiles (inverse pivots and forward
        // sums to the planes), then backward
        auto own_rows = [&](int base0, double *plane, bool put) {
#pragma unroll
            for (int j = 0; j < RM; ++j) {
                const int i = base0 + c * r + j;
                if (j < r && i < n) {
                    if (put) plane[(size_t)i * st] = e[j];
                    else e[j] = plane[(size_t)i * st];
                } else if (!put) {
                    e[j] = 0.0;
                }
            }
        };
        double idc = 0.0;
        for (int t = 0; t < Tmax; ++t) {
            const int base0 = t * P * r;
            load_knots(base0);
            factorise(base0, idc);
            idc = sm.carry[bl];
            own_rows(base0, ibp, true);
            weights(base0);
            scan_factors();
            for (int s = s_begin; s < s_end; ++s) {
                const SplineSeries f = acc.series(bl, s);
                load_slopes(base0, f.y);
                forward(base0, (t > 0 && base0 <= n) ? f.cd[(size_t)(base0 - 1) * st] : 0.0);
                own_rows(base0, f.cd, true);
                __syncthreads();
            }
        }
        for (int t = Tmax - 1; t >= 0; --t) {
            const int base0 = t * P * r, next = base0 + P * r;
            load_knots(base0);
            own_rows(base0, ibp, false);
            weights(base0);
            scan_factors();
            for (int s = s_begin; s < s_end; ++s) {
                const SplineSeries f = acc.series(bl, s);
                load_slopes(base0, f.y);
                own_rows(base0, f.cd, false);
                backward(next < n ? f.cd[(size_t)next * st] : 0.0);
                store(base0, s, f);
            }
        }
    }
};

}  // namespace eob
