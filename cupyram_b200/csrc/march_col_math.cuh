// march_col_math.cuh - complex and 2 x 2 matrix helpers, slices and output
// losses shared by the column-parallel march kernels (march_col.cu: factors in
// shared memory, march_reg.cu: factors in registers).
#pragma once

#include "march_common.cuh"

namespace crk {

template <typename V>
__device__ __forceinline__ V vmul(V a, V b) {
    V r;
    r.x = fma(a.x, b.x, -a.y * b.y);
    r.y = fma(a.x, b.y, a.y * b.x);
    return r;
}
template <typename V>
__device__ __forceinline__ V vfma(V a, V b, V c) {  // a * b + c
    V r;
    r.x = fma(a.x, b.x, fma(-a.y, b.y, c.x));
    r.y = fma(a.x, b.y, fma(a.y, b.x, c.y));
    return r;
}
template <typename V>
__device__ __forceinline__ V vzero() {
    V r;
    r.x = 0;
    r.y = 0;
    return r;
}
template <typename V>
__device__ __forceinline__ V vone() {
    V r;
    r.x = 1;
    r.y = 0;
    return r;
}

// Rows of CTA c of a cluster of C over nz rows (near-equal contiguous slices).
__device__ __forceinline__ void slice_of(int nz, int C, int c, int& R0, int& R1) {
    const int base = nz / C, extra = nz % C;
    R0 = 1 + c * base + (c < extra ? c : extra);
    R1 = R0 + base - 1 + (c < extra ? 1 : 0);
}

__host__ __device__ inline size_t r16(size_t b) { return (b + 15) & ~(size_t)15; }

// 2 x 2 complex matrix [[a, b], [c, d]].
struct M2 {
    double2 a, b, c, d;
};
__device__ __forceinline__ double2 cadd(double2 x, double2 y) { return c2(x.x + y.x, x.y + y.y); }
__device__ __forceinline__ M2 m2_mul(const M2& X, const M2& Y) {
    return {cadd(cmul(X.a, Y.a), cmul(X.b, Y.c)), cadd(cmul(X.a, Y.b), cmul(X.b, Y.d)),
            cadd(cmul(X.c, Y.a), cmul(X.d, Y.c)), cadd(cmul(X.c, Y.b), cmul(X.d, Y.d))};
}
// The maps act projectively (w = N / D), so a matrix may be rescaled at will:
// keep its largest component near 1.
__device__ __forceinline__ M2 m2_norm(M2 X) {
    const double m = fmax(fmax(fmax(fabs(X.a.x), fabs(X.a.y)), fmax(fabs(X.b.x), fabs(X.b.y))),
                          fmax(fmax(fabs(X.c.x), fabs(X.c.y)), fmax(fabs(X.d.x), fabs(X.d.y))));
    if (m > 0.0 && isfinite(m)) {
        const double s = 1.0 / m;
        X.a = c2(X.a.x * s, X.a.y * s);
        X.b = c2(X.b.x * s, X.b.y * s);
        X.c = c2(X.c.x * s, X.c.y * s);
        X.d = c2(X.d.x * s, X.d.y * s);
    }
    return X;
}
__device__ __forceinline__ M2 m2_eye() { return {c2(1.0, 0.0), c2(0.0, 0.0), c2(0.0, 0.0), c2(1.0, 0.0)}; }
__device__ __forceinline__ M2 m2_shfl(const M2& X, int from) {
    M2 r;
    r.a = c2(__shfl_sync(0xffffffffu, X.a.x, from), __shfl_sync(0xffffffffu, X.a.y, from));
    r.b = c2(__shfl_sync(0xffffffffu, X.b.x, from), __shfl_sync(0xffffffffu, X.b.y, from));
    r.c = c2(__shfl_sync(0xffffffffu, X.c.x, from), __shfl_sync(0xffffffffu, X.c.y, from));
    r.d = c2(__shfl_sync(0xffffffffu, X.d.x, from), __shfl_sync(0xffffffffu, X.d.y, from));
    return r;
}

// The Galerkin row m of the term (r1, r2, r3 of M + p D) from the f-window.
struct Rrow {
    double2 r1, r2, r3;
};

}  // namespace crk
