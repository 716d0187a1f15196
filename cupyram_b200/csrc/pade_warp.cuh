// pade_warp.cuh - pade_coefficients (pade.h) by one warp, with its arrays in
// shared memory.
//
// One thread alone took 1.1 ms for the sets of one ray (np 8): every step waits
// for its own arrays in local memory, and the two root searches run one after
// the other.  Here the lanes share the Taylor sums' products and the rows of
// the elimination, the numerator's and the denominator's roots are searched at
// once (a half-warp each), and a search's three Horner chains run in three
// lanes.  Every element sees the operations of pade.h in their order, so the
// coefficients are the same to the last bit.
#pragma once

#include "pade.h"

namespace cr {

struct PadeShared {
    cd m[kMaxN][kMaxN + 1];
    cd rhs[kMaxN], dg[kMaxN + 1], hs[kMaxN];
    double binom[kMaxN + 1][kMaxN + 1];
    double fct[kMaxN + 1];
    cd poly[2][kMaxNp + 2], d1[2][kMaxNp + 2], d2[2][kMaxNp + 2], roots[2][kMaxNp + 2];
};

// laguerre_root for both halves of the warp (half h: polynomial h of the same
// degree), in step.  Returns, per half, whether the search failed.
__device__ __forceinline__ bool laguerre_warp(PadeShared& S, int deg, cd* z, double err, int nter) {
    const int lane = threadIdx.x & 31, h = lane >> 4, s = lane & 15;
    const cd* poly = S.poly[h];
    for (int i = s; i < deg; i += 16) S.d1[h][i] = double(i + 1) * poly[i + 1];
    __syncwarp();
    for (int i = s; i + 1 < deg; i += 16) S.d2[h][i] = double(i + 1) * S.d1[h][i + 1];
    __syncwarp();
    // lane 0 of the half: the polynomial, lane 1: its derivative, lane 2: the second
    const cd* c = s == 1 ? S.d1[h] : s == 2 ? S.d2[h] : poly;
    const int top = s == 1 ? deg - 1 : s == 2 ? deg - 2 : deg;
    cd x = *z;
    double step = INFINITY;
    int it = 0, kick = 0;
    bool failed = false, on = true;
    while (true) {
        on = on && step > err && it < nter - 1;
        if (!__any_sync(0xffffffffu, on)) break;
        cd p = c[top - 1] + c[top] * x;
        for (int i = top - 2; i >= 0; --i) p = c[i] + x * p;
        const cd p0 = cd{__shfl_sync(0xffffffffu, p.re, 0, 16), __shfl_sync(0xffffffffu, p.im, 0, 16)};
        const cd p1 = cd{__shfl_sync(0xffffffffu, p.re, 1, 16), __shfl_sync(0xffffffffu, p.im, 1, 16)};
        const cd p2 = cd{__shfl_sync(0xffffffffu, p.re, 2, 16), __shfl_sync(0xffffffffu, p.im, 2, 16)};
        if (on && cabsd(p0) < 1e-20) on = false;
        if (on) {
            const cd f = p1 / p0;
            const cd g = f * f - p2 / p0;
            const cd hh = csqrt_p(double(deg - 1) * (double(deg) * g - f * f));
            const cd fp = f + hh, fm = f - hh;
            cd dx = (cabsd(fp) > cabsd(fm)) ? (-double(deg)) / fp : (-double(deg)) / fm;
            ++it;
            if (++kick == 9) {
                kick = 0;
                dx = cd{-dx.im, dx.re};  // multiply by i: leave a limit cycle
            }
            x = x + dx;
            step = cabsd(dx);
            if (it == 100) {
                failed = true;
                on = false;
            }
        }
    }
    *z = x;
    return failed;
}

// pade_coefficients with its 32 lanes; a[j] / b[j] (j < np) are valid in every
// lane's S.roots-derived output: pd of half 0 and half 1.  Returns the status
// (uniform).  Called by a whole warp.
__device__ inline int pade_warp(PadeShared& S, double freq, double c0, int np, int ns, double dr, int ip, cd* pd1,
                                cd* pd2) {
    const int lane = threadIdx.x & 31;
    if (np < 1 || np > kMaxNp || !(c0 > 0.0) || !(freq > 0.0)) return kPadeBadArgs;
    const int n = 2 * np;
    const double sig = 2.0 * M_PI * freq / c0 * dr;
    const double nu = (ip == 1) ? 0.0 : 1.0;
    const double alp = (ip == 1) ? 0.0 : -0.25;
    for (int i = 0; i <= n; ++i) {
        // the row of lane j from the row above (exact integers)
        if (lane <= n) S.binom[i][lane] = (lane == 0 || lane == i) ? 1.0
                                          : (i > 1 && lane < i) ? S.binom[i - 1][lane - 1] + S.binom[i - 1][lane]
                                                                : 0.0;
        __syncwarp();
    }
    if (lane == 0) {
        S.fct[0] = 1.0;
        for (int i = 1; i < n; ++i) S.fct[i] = double(i + 1) * S.fct[i - 1];
    }
    if (lane == 1) {
        cd h1 = cd{0.0, 0.5 * sig}, h2 = cd{alp, 0.0}, h3 = cd{-2.0 * nu, 0.0};
        S.hs[0] = h1 + h2 + h3;
        double e1 = -0.5, e2 = -1.0, e3 = -1.0;
        for (int i = 1; i < n; ++i) {
            h1 = cd{__dmul_rn(h1.re, e1), __dmul_rn(h1.im, e1)};
            h2 = cd{__dmul_rn(h2.re, e2), __dmul_rn(h2.im, e2)};
            const double q = -nu * e3;
            h3 = cd{__dmul_rn(q, h3.re), __dmul_rn(q, h3.im)};
            S.hs[i] = h1 + h2 + h3;
            e1 -= 1.0;
            e2 -= 1.0;
            e3 -= 1.0;
        }
    }
    __syncwarp();
    if (lane == 0) {
        S.dg[0] = cd{1.0, 0.0};
        S.dg[1] = S.hs[0];
    }
    __syncwarp();
    for (int i = 1; i < n; ++i) {
        cd t = cd{0.0, 0.0};
        if (lane < i) t = (S.binom[i][lane] * S.hs[lane]) * S.dg[i - lane];
        cd acc = S.hs[i];
        for (int j = 0; j < i; ++j)
            acc = acc + cd{__shfl_sync(0xffffffffu, t.re, j), __shfl_sync(0xffffffffu, t.im, j)};
        if (lane == 0) S.dg[i + 1] = acc;
        __syncwarp();
    }
    // the linear system, a row per lane
    if (lane < n) {
        const int i = lane;
        for (int j = 0; j <= n; ++j) S.m[i][j] = cd{0.0, 0.0};
        cd r = S.dg[i + 1];
        if (2 * i <= n - 1) S.m[i][2 * i] = cd{S.fct[i], 0.0};
        for (int j = 0; j <= i; ++j)
            if (2 * j + 1 <= n - 1) S.m[i][2 * j + 1] = (-S.binom[i + 1][j + 1] * S.fct[j]) * S.dg[i - j];
        const int c = n - 1 - i;  // stability constraint of this row
        if (c < ns && c < 2) {
            const double z = c == 0 ? -3.0 : -1.5;
            r = cd{-1.0, 0.0};
            double zp = 1.0;
            for (int j = 0; j < np; ++j) {
                zp *= z;
                S.m[i][2 * j] = cd{zp, 0.0};
                S.m[i][2 * j + 1] = cd{0.0, 0.0};
            }
        }
        S.rhs[i] = r;
    }
    __syncwarp();
    // elimination with partial pivoting: the first row of the largest modulus
    for (int i = 0; i < n; ++i) {
        if (i < n - 1) {
            const bool in = lane >= i && lane < n;
            double v = in ? cabsd(S.m[lane][i]) : -1.0;
            int at = lane;
            for (int d = 16; d >= 1; d >>= 1) {
                const double ov = __shfl_xor_sync(0xffffffffu, v, d);
                const int oa = __shfl_xor_sync(0xffffffffu, at, d);
                if (ov > v || (ov == v && oa < at)) {
                    v = ov;
                    at = oa;
                }
            }
            // a NaN modulus compares false, as in the serial search, and leaves row i in place
            const double own = cabsd(S.m[i][i]);
            const int piv = v > own ? at : i;
            if (piv != i) {
                if (lane == 0) {
                    const cd t = S.rhs[piv];
                    S.rhs[piv] = S.rhs[i];
                    S.rhs[i] = t;
                }
                for (int j = i + lane; j <= n; j += 32) {
                    const cd u = S.m[piv][j];
                    S.m[piv][j] = S.m[i][j];
                    S.m[i][j] = u;
                }
            }
            __syncwarp();
        }
        const cd inv = 1.0 / S.m[i][i];
        const cd ri = S.rhs[i] * inv;
        __syncwarp();
        if (lane == 0) S.rhs[i] = ri;
        if (i < n - 1) {
            for (int j = i + 1 + lane; j <= n; j += 32) S.m[i][j] = S.m[i][j] * inv;
            __syncwarp();
            const int rest = n - 1 - i;  // rows below, and columns i + 1 .. n - 1
            for (int q = lane; q < rest * rest; q += 32) {
                const int k = i + 1 + q / rest, j = i + 1 + q % rest;
                S.m[k][j] = S.m[k][j] - S.m[k][i] * S.m[i][j];
            }
            for (int k = i + 1 + lane; k < n; k += 32) S.rhs[k] = S.rhs[k] - S.m[k][i] * ri;
        }
        __syncwarp();
    }
    for (int i = n - 2; i >= 0; --i) {
        cd t = cd{0.0, 0.0};
        if (lane > i && lane < n) t = S.m[i][lane] * S.rhs[lane];
        cd acc = S.rhs[i];
        for (int j = i + 1; j < n; ++j)
            acc = acc - cd{__shfl_sync(0xffffffffu, t.re, j), __shfl_sync(0xffffffffu, t.im, j)};
        __syncwarp();
        if (lane == 0) S.rhs[i] = acc;
        __syncwarp();
    }
    // roots of both polynomials, a half-warp each
    const int h = lane >> 4, s = lane & 15;
    if (s == 0) S.poly[h][0] = cd{1.0, 0.0};
    for (int j = s; j < np; j += 16) S.poly[h][j + 1] = S.rhs[2 * j + h];
    __syncwarp();
    bool failed = false;
    for (int k = np - 1; k >= 2; --k) {
        cd x = cd{0.0, 0.0};
        failed |= laguerre_warp(S, k + 1, &x, 1e-12, 1000);
        failed |= laguerre_warp(S, k + 1, &x, 0.0, 5);
        if (__any_sync(0xffffffffu, failed)) return kPadeNoConverge;
        if (s == 0) {
            cd* poly = S.poly[h];
            S.roots[h][k] = x;
            // synthetic division by (X - x), coefficients shifted down one place
            for (int i = k; i >= 0; --i) poly[i] = poly[i] + x * poly[i + 1];
            for (int i = 0; i <= k; ++i) poly[i] = poly[i + 1];
        }
        __syncwarp();
    }
    if (s == 0) {
        const cd* poly = S.poly[h];
        if (np == 1) {
            S.roots[h][0] = -poly[0] / poly[1];
        } else {
            const cd disc = csqrt_p(poly[1] * poly[1] - 4.0 * (poly[0] * poly[2]));
            S.roots[h][1] = 0.5 * (-poly[1] + disc) / poly[2];
            S.roots[h][0] = 0.5 * (-poly[1] - disc) / poly[2];
        }
    }
    __syncwarp();
    if (lane < np) {
        pd1[lane] = -1.0 / S.roots[0][lane];
        pd2[lane] = -1.0 / S.roots[1][lane];
    }
    return kPadeOk;
}

}  // namespace cr
