// march_reg.cu - column-parallel range march, complex128, factors in registers.
//
// One ray runs on a thread-block cluster of C CTAs.  The column's rows 1..nz
// are cut into C slices; a CTA runs one warp per term of the partial-fraction
// form (M + p_k D) x_k = M u, and a warp's 32 lanes cut the slice into
// segments of at most L rows (a template value).  Everything a step touches
// stays on the chip, and what it touches most stays in registers:
//
//   * registers of the lane that owns the rows: the elimination's coupling al
//     and the back-substitution factor -w of every row, and the workspace g;
//   * shared memory: the field, 1/den (read once a step), the terms'
//     solutions on their way to the sum, and the products of al and -w that
//     the scans below multiply by - they only change with the operator.
//
// A step's recurrences g_m = q b_m + al_m g_{m-1} (down) and x_m = g_m - w_m
// x_{m+1} (up) are first-order maps, and a lane's part in them is linear in
// what enters it: with e the value of g above its rows and v that of x below,
//
//     g_last  = h + A e           h, y: from its own rows alone
//     x_first = y + Z v + V e     A, Z, V: depend on the operator alone
//
// so a step carries only h and y, and knows every A, Z and V (and their
// products over lanes and slices) from the factorisation:
//
//     sweep    h downwards (every h_m kept), y upwards
//     scan     e of every lane (5 shuffle levels), then v, for a slice alone
//     exchange h and y of the slice to every CTA of the cluster
//     fold     gin, xin of the slice: weighted sums over all slices' h and y
//     sweep    true g from the lane's e, true x from its v
//     sum      u = c_inf u + sum_k c_k x_k, two terms added in registers
//              before the rest meet in shared memory
//
// Exchange.  A slice's h and y (32 bytes a term) are written straight into the
// shared memory of every CTA (st.async), completing on a barrier of the
// receiving warp; no CTA waits for a whole cluster.  Two mailboxes alternate:
// a CTA writes a mailbox again two steps later, after it received the values
// of the step between, which the reader sent after it had read this one.  A
// term's mailbox and phase follow from the number of steps that it took part in:
// the sets of a ray may differ in their number of terms, so a term may sit out
// steps anywhere in the march.
// Waits are bounded: one that gives up flags the ray (bit 1).
//
// b = M u is a1 (u_{m-1} + 4 u_m + u_{m+1}) with the factor a1 in the stored
// 1/den.
//
// Range logic, self-starter and outputs follow the batched march
// (cupyram/cupyram.py:273-380 run, :1001-1063 selfs, updat.py:38-140,
// outpt.py:11-57).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>

#include "march_col_math.cuh"
#include "march_reg.cuh"

namespace cg = cooperative_groups;

namespace crk {

namespace {

constexpr int kRegMaxTerms = CR_MAX_NP;
constexpr int kRegMaxCluster = 16;
constexpr size_t kRegSmemLimit = 227 * 1024;
constexpr unsigned kMailWaitLimit = 1u << 22;  // polls of a mailbox before giving up

// State of a CTA's range logic and outputs (written by one thread, between
// barriers).
struct RegCtl {
    double rs;
    double wa, wb;   // weights of the line's two rows
    long long line;  // index of the ray's line outputs, -1: another CTA writes them
    long long grid;  // index of the ray's grid outputs, -1: none
    int next;        // first step whose operator has to be looked at again
    int iz, ss, sb, bt, set;
    int lo, hi;      // rows to assemble again (lo > hi: none)
    int refactor;    // the operator changed
    int dead;        // a bounded wait gave up
    unsigned ua, ub; // offsets of the field of the line's two rows
    unsigned ndz, ndz_inv;  // grid row spacing and 2^32 / ndz rounded up (0 for 1)
    int nvz, nvr, ndr;
    // fixed for the march
    int rid, nz, R0, R1, n;  // the ray, its rows, the slice's rows R0 .. R1 (n)
    long long col;           // the ray's column
    double cfact, a1, a2;
    int seg;                 // rows of a segment of the factorisation
    int env, n_bt, n_rss, n_rsb;
    double dr, dz;
    const double *rb, *zb, *rp_ss, *rp_sb;
    double inv_dr, inv_per;  // 1 / dr; steps a cell of the bottom's segment takes (segment per_bt)
    int per_bt;
    int line_row;            // the line lies between this row and the next,
    double line_dir;         // this far down
    unsigned idle[CR_MAX_NP];  // steps so far that the term sat out
};
constexpr unsigned kCtlBytes = 320;
static_assert(sizeof(RegCtl) <= kCtlBytes, "RegCtl must fit its slot");

// Shared memory of a CTA (offsets in bytes; every CTA of a cluster uses the
// same): the CTA's own part, then one region per term, then the pairs' sums.
// Within the first two every offset is a constant, so that a warp addresses
// all its tables from one base.
template <int L, bool ALL>
struct RegOff {
    static constexpr unsigned P = 32u * (unsigned)L;
    static constexpr unsigned ck = 0;                      // residues of the active set
    static constexpr unsigned misc = ck + 16 * CR_MAX_NP;  // c_inf, u of row R0 - 1, u of row R1 + 1, zero
    static constexpr unsigned ctl = misc + 64;
    static constexpr unsigned edges = ctl + kCtlBytes;     // [32] offsets of the field above (low half) and below
    static constexpr unsigned U = edges + 128;             // field of the slice, slot [j][lane]
    static constexpr unsigned term0 = U + 16 * P;
    // of a term's region
    static constexpr unsigned Q = 0;                       // [P] a1 / den
    static constexpr unsigned SD = Q + 16 * P;             // [4][32] products of A over the 1, 2, 4, 8 lanes ending here
    static constexpr unsigned SU = SD + 4 * 512;           // [4][32] products of Z over the lanes beginning here
    static constexpr unsigned SX = SU + 4 * 512;           // [32] over 16 lanes: Z in lanes 0..15, A in lanes 16..31
    static constexpr unsigned V = SX + 512;                // [32]
    static constexpr unsigned EA = V + 512;                // [32] e of the lane per unit of gin
    static constexpr unsigned EZ = EA + 512;               // [32] v of the lane per unit of xin
    static constexpr unsigned EV = EZ + 512;               // [32] v of the lane per unit of gin
    static constexpr unsigned WA = EV + 512;               // [16] h of slice j in gin, [16] in xin
    static constexpr unsigned WB = WA + 512;               // [16] zero, [16] y of slice j in xin
    static constexpr unsigned mail = WB + 512;             // [2][16] {h, y} by sending CTA
    static constexpr unsigned fmat = mail + 1024;          // [4] factorisation map of the slice
    static constexpr unsigned tot = fmat + 64;             // [3] A, Z, V of the slice
    static constexpr unsigned xh = tot + 48;               // [2] c_k x of the halo rows R0 - 1 and R1 + 1
    static constexpr unsigned wghost = xh + 32;            // -w of row R0 - 1
    static constexpr unsigned bar = wghost + 16;           // [2] mbarriers of the mailboxes
    static constexpr unsigned term = bar + 16;             // size of a region
    // ALL: [term][P] x_k, else [pair][P] c_k x_k of two terms; over the same
    // bytes, during a factorisation, the Galerkin rows [3][P]
    __host__ __device__ static unsigned X(int terms) { return term0 + (unsigned)terms * term; }
    __host__ __device__ static unsigned F3(int terms) {
        const int rows = ALL ? terms : (terms + 1) / 2;
        return X(terms) + (unsigned)(rows > 3 ? rows : 3) * 16 * P;
    }
    // f3 of rows R0 - 1 .. R1 + 1, for grid outputs only
    __host__ __device__ static unsigned bytes(int terms, int nmax, int grids) {
        return F3(terms) + (grids ? 4 * (unsigned)(nmax + 2) : 0u);
    }
};

// ---- mailboxes ----
__device__ __forceinline__ unsigned remote_addr(unsigned local, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void mail_send(unsigned addr, unsigned bar, double2 v) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "l"(__double_as_longlong(v.x)), "l"(__double_as_longlong(v.y)), "r"(bar)
                 : "memory");
}
// The whole warp: announces `bytes` (lane 0) and waits for the phase.  Returns
// false when the wait gave up.
__device__ __forceinline__ bool mail_wait(unsigned bar, unsigned bytes, unsigned parity, int lane) {
    if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    for (unsigned it = 0; it < kMailWaitLimit; ++it) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity), "n"(100)
            : "memory");
        if (done) return true;
    }
    return false;
}

// 16-byte accesses by shared-memory address: the step's tables are addressed
// by 32-bit offsets from one register, which the generic pointers of the rest
// would double.
__device__ __forceinline__ double2 lds2(unsigned addr) {
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ unsigned lds1(unsigned addr) {
    unsigned v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void sts2(unsigned addr, double2 v) {
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}

__device__ __forceinline__ double2 shfl2(double2 v, int from) {
    return c2(__shfl_sync(0xffffffffu, v.x, from), __shfl_sync(0xffffffffu, v.y, from));
}
__device__ __forceinline__ double2 shfl2_up(double2 v, int d) {
    return c2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ double2 shfl2_down(double2 v, int d) {
    return c2(__shfl_down_sync(0xffffffffu, v.x, d), __shfl_down_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ double2 shfl2_xor(double2 v, int d) {
    return c2(__shfl_xor_sync(0xffffffffu, v.x, d), __shfl_xor_sync(0xffffffffu, v.y, d));
}

// What a thread keeps at hand; the rest of the CTA's state is in RegCtl.
struct RegCtx {
    unsigned char* sm;   // the CTA's shared memory
    unsigned char* tm;   // this warp's region
    unsigned sm32, tm32; // their shared-memory addresses
    RegCtl* ctl;
    int C, c;            // the cluster's CTAs, this one
    int term, lane;
    int npad;            // the lane's first npad positions hold no row
    int row0;            // row of position npad
    template <typename T>
    __device__ __forceinline__ T* at(unsigned off) const { return reinterpret_cast<T*>(sm + off); }
    __device__ __forceinline__ double2* own(unsigned off) const { return reinterpret_cast<double2*>(tm + off); }
};

// The first positions of a lane without rows: slices of n rows give lanes
// n / 32 rows, the last n % 32 lanes one more, right-aligned in L positions.
__device__ __forceinline__ void lane_rows(int n, int lane, int& start, int& cnt) {
    const int base = n >> 5, low = 32 - (n & 31);  // lanes below `low` hold base rows
    cnt = lane < low ? base : base + 1;
    start = lane < low ? lane * base : low * base + (lane - low) * (base + 1);
}
// Shared-memory slot of slice position p (0 .. n - 1).
__device__ __forceinline__ int slot_of(int n, int L, int p) {
    const int base = n >> 5, low = 32 - (n & 31);
    int lane, idx;
    if (p < low * base) {
        lane = p / base;
        idx = p - lane * base + (L - base);
    } else {
        const int q = p - low * base;
        lane = low + q / (base + 1);
        idx = q % (base + 1) + (L - base - 1);
    }
    return idx * 32 + lane;
}

// A lane has at most kMaxPad positions without a row (reg_rows).
constexpr int kMaxPad = 2;

// 1/den of the slice's rows for one term, into Q[position]; returns -w of row
// R0 - 1 in lane 0.  The recurrence w_m = r3 / (r2 - r1 w_{m-1}) is linear in
// homogeneous coordinates, (N, D)_m = [[0, r3], [-r1, r2]] (N, D): each lane
// multiplies its rows' matrices, the warp scans the products, the cluster
// folds in the slices above (one cluster barrier when C > 1), and each lane
// runs the recurrence from its true entry.  Segments (of ceil(nmax / 32) rows),
// order and scaling are those of march_col.cu: a segment's entry carries a
// rounding error that stays for as long as the operator does, so over a long
// march two kernels agree as closely as their entries do.
__device__ __noinline__ double2 reg_recurrence(const double2* D, int P, double2 p, double a1, double a2, int n,
                                               int rows, bool active, double2* fmat, double2* Q, int C, int c) {
    cg::cluster_group cl = cg::this_cluster();
    const int l = threadIdx.x & 31;
    const int p0 = min(n, l * rows), p1 = min(n, p0 + rows);
    M2 ex = m2_eye();
    if (active) {
        M2 seg = m2_eye();
        int since = 0;
#pragma unroll 1
        for (int q = p0; q < p1; ++q) {
            const double2 r1 = caxpd(a1, p, D[q]), r2 = caxpd(a2, p, D[P + q]), r3 = caxpd(a1, p, D[2 * P + q]);
            const double2 m1 = c2(-r1.x, -r1.y);
            seg = {cmul(r3, seg.c), cmul(r3, seg.d), cadd(cmul(m1, seg.a), cmul(r2, seg.c)),
                   cadd(cmul(m1, seg.b), cmul(r2, seg.d))};
            if (++since == 8) {
                seg = m2_norm(seg);
                since = 0;
            }
        }
        seg = m2_norm(seg);
#pragma unroll 1
        for (int d = 1; d < 32; d <<= 1) {
            const M2 prev = m2_shfl(seg, max(l - d, 0));
            if (l >= d) seg = m2_norm(m2_mul(seg, prev));
        }
        ex = m2_shfl(seg, max(l - 1, 0));
        if (l == 0) ex = m2_eye();
        if (l == 31) {
            fmat[0] = seg.a;
            fmat[1] = seg.b;
            fmat[2] = seg.c;
            fmat[3] = seg.d;
        }
    }
    double2 wp = c2(0.0, 0.0);
    if (C > 1) cl.sync();
    if (active) {
        double2 N = ex.b, E = ex.d;  // entry (N, E) = ex C (0, 1)
        if (c > 0) {
            // the slices above, in order (lane j holds CTA j's map)
            M2 Cm = m2_eye();
            if (l < c) {
                const double2* f = cl.map_shared_rank(fmat, l);
                Cm = {f[0], f[1], f[2], f[3]};
            }
#pragma unroll 1
            for (int d = 1; d < c; d <<= 1) {
                const M2 prev = m2_shfl(Cm, max(l - d, 0));
                if (l >= d) Cm = m2_norm(m2_mul(Cm, prev));
            }
            const double2 n0 = shfl2(Cm.b, c - 1), d0 = shfl2(Cm.d, c - 1);
            N = cadd(cmul(ex.a, n0), cmul(ex.b, d0));
            E = cadd(cmul(ex.c, n0), cmul(ex.d, d0));
        }
        wp = (N.x == 0.0 && N.y == 0.0) ? c2(0.0, 0.0) : cmul(N, crcp(E));
        double2 w = wp;
#pragma unroll 1
        for (int q = p0; q < p1; ++q) {
            const double2 r1 = caxpd(a1, p, D[q]), r2 = caxpd(a2, p, D[P + q]), r3 = caxpd(a1, p, D[2 * P + q]);
            const double2 qq = crcp(cfms(r2, r1, w));
            w = cmul(r3, qq);
            Q[q] = qq;
        }
        __syncwarp();
    }
    return c2(-wp.x, -wp.y);
}

// Affine scan over the lanes, h_l += M_l h_{l -/+ d}: the multipliers of level
// i are at tab + 512 i, those of the last level (at last) only hold in one half
// of the warp.  AHEAD: each level's multiplier is read a level before its use,
// the first (m) and the last (sx) by the caller.
template <bool UP, bool AHEAD>
__device__ __forceinline__ double2 lane_scan(double2 h, unsigned tab, unsigned last, double2 m, double2 sx, int l) {
#pragma unroll
    for (int lev = 0; lev < 4; ++lev) {
        double2 next = c2(0.0, 0.0);
        if (AHEAD && lev < 3) next = lds2(tab + (lev + 1) * 512u);
        if (!AHEAD) m = lds2(tab + lev * 512u);
        h = vfma(m, UP ? shfl2_down(h, 1 << lev) : shfl2_up(h, 1 << lev), h);
        m = next;
    }
    if (!AHEAD) sx = lds2(last);
    const double2 t = UP ? shfl2_down(h, 16) : shfl2_up(h, 16);
    const bool in = UP ? l < 16 : l >= 16;
    return vfma(in ? sx : c2(0.0, 0.0), t, h);
}

// Weights of the slices' h and y in this slice's gin and xin, from every
// slice's (A, Z, V): gin(c) = sum_{i<c} [A over i+1..c-1] h_i and
// xin(c) = sum_{j>c} [Z over c+1..j-1] (y_j + V_j gin(j)).
__device__ __noinline__ void reg_weights(double2* tot, double2* WA, double2* WB, int C, int c) {
    cg::cluster_group cl = cg::this_cluster();
    const int i = threadIdx.x & 31;
    const double2 one = c2(1.0, 0.0), zero = c2(0.0, 0.0);
    double2 A = one, Z = one, V = zero;
    if (i < C) {
        const double2* f = cl.map_shared_rank(tot, i);
        A = f[0];
        Z = f[1];
        V = f[2];
    }
    // lane i: the products of A over i .. c - 1 and of Z over c + 1 .. i, and then
    // without the first and the last
    double2 pa = i < c ? A : one, pz = i > c ? Z : one;
#pragma unroll 1
    for (int d = 1; d < C; d <<= 1) {
        const double2 qa = shfl2(pa, min(i + d, 31)), qz = shfl2(pz, max(i - d, 0));
        pa = i + d < 32 ? cmul(pa, qa) : pa;
        pz = i >= d ? cmul(pz, qz) : pz;
    }
    const double2 g = shfl2(pa, min(i + 1, 31)), y = shfl2(pz, max(i - 1, 0));
    // h of slice i reaches xin through V of every slice below both i and this one:
    // x_i = t_{i+1} + A_{i+1} x_{i+1}, t_j = [Z over c+1..j-1] V_j; scanned upwards
    // as maps x -> M x + T, each lane's own map that of lane i + 1
    double2 t = i > c && i < C ? cmul(y, V) : zero;
    double2 T = shfl2_down(t, 1), M = shfl2_down(A, 1);
    if (i + 1 >= C) {
        T = zero;
        M = one;
    }
#pragma unroll 1
    for (int d = 1; d < C; d <<= 1) {
        const double2 qm = shfl2(M, min(i + d, 31)), qt = shfl2(T, min(i + d, 31));
        if (i + d < 32) {
            T = vfma(M, qt, T);
            M = cmul(M, qm);
        }
    }
    if (i < 16) {
        WA[i] = i < c ? g : zero;
        WA[16 + i] = i < C ? T : zero;
        WB[i] = zero;
        WB[16 + i] = i > c && i < C ? y : zero;
    }
}

// Thomas factorisation of the active terms, the per-row factors left in the
// lanes' registers and all that a step multiplies by in shared memory.
// Called by every thread of every CTA of the cluster (two cluster barriers
// when C > 1).  The Galerkin rows are computed once per slice and shared by
// its terms.
template <int L, bool ALL>
__device__ __forceinline__ void reg_factor(const ColArgs& a, const RegCtx& x, cg::cluster_group& cl, int set,
                                           int n_active, double2 (&al)[L], double2 (&mw)[L]) {
    using O = RegOff<L, ALL>;
    constexpr int P = 32 * L;
    const int k = x.term, l = x.lane;
    const bool active = k < n_active;
    double2* D = x.at<double2>(O::X(blockDim.x >> 5));
    const RegCtl* ctl = x.ctl;
    const int n = ctl->n;
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
        const long long o = ctl->col + (long long)(ctl->R0 + q) * kTile;
        auto ld = [&](long long i) { return EnvRow{a.f1[i], a.f2[i], a.f3[i], a.ksq[i]}; };
        const Drow d = galerkin3(ld(o - kTile), ld(o), ld(o + kTile), ctl->cfact);
        D[q] = d.d1;
        D[P + q] = d.d2;
        D[2 * P + q] = d.d3;
    }
    __syncthreads();
    const double2 p = active ? a.pd2[((long long)ctl->rid * kSets + set) * CR_MAX_NP + k] : c2(0.0, 0.0);
    const double a1 = ctl->a1;
    const double2 mwp = reg_recurrence(D, P, p, a1, ctl->a2, n, ctl->seg, active, x.own(O::fmat), x.own(O::Q), x.C, x.c);
    if (active) {
        if (l == 0) *x.own(O::wghost) = mwp;
        double2* Q = x.own(O::Q);
        double2 pa = c2(1.0, 0.0), pw = c2(1.0, 0.0), qq[L];
        const int first = x.row0 - ctl->R0 - x.npad;  // position of the lane's j = 0
#pragma unroll
        for (int j = 0; j < L; ++j) {
            if (j >= kMaxPad || j >= x.npad) {
                const int q = first + j;
                qq[j] = Q[q];
                const double2 ci = cmul(caxpd(a1, p, D[q]), qq[j]), w = cmul(caxpd(a1, p, D[2 * P + q]), qq[j]);
                al[j] = c2(-ci.x, -ci.y);
                mw[j] = c2(-w.x, -w.y);
                pa = cmul(al[j], pa);
                pw = cmul(mw[j], pw);
            } else {  // no row: both maps pass their value through
                al[j] = c2(1.0, 0.0);
                mw[j] = c2(1.0, 0.0);
                qq[j] = c2(0.0, 0.0);
            }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < L; ++j) Q[j * 32 + l] = c2(a1 * qq[j].x, a1 * qq[j].y);
        // V: x_first per unit of e
        double2 v = c2(0.0, 0.0);
        {
            double2 g[L], e = c2(1.0, 0.0);
#pragma unroll
            for (int j = 0; j < L; ++j) {
                e = cmul(al[j], e);
                g[j] = e;
                if (j < kMaxPad && j < x.npad) g[j] = c2(0.0, 0.0);
            }
#pragma unroll
            for (int j = L - 1; j >= 0; --j) v = vfma(mw[j], v, g[j]);
        }
        x.own(O::V)[l] = v;
        // A and Z over 1, 2, .. lanes, and over all lanes above (EA) or below (EZ)
#pragma unroll
        for (int lev = 0; lev < 5; ++lev) {
            const int d = 1 << lev;
            if (lev < 4) {
                x.own(O::SD)[lev * 32 + l] = l >= d ? pa : c2(0.0, 0.0);
                x.own(O::SU)[lev * 32 + l] = l + d < 32 ? pw : c2(0.0, 0.0);
            } else {
                x.own(O::SX)[l] = l >= 16 ? pa : pw;
            }
            const double2 qa = shfl2(pa, max(l - d, 0)), qw = shfl2(pw, min(l + d, 31));
            if (l >= d) pa = cmul(pa, qa);
            if (l + d < 32) pw = cmul(pw, qw);
        }
        double2 ea = shfl2(pa, max(l - 1, 0)), ez = shfl2(pw, min(l + 1, 31));
        if (l == 0) ea = c2(1.0, 0.0);
        if (l == 31) ez = c2(1.0, 0.0);
        x.own(O::EA)[l] = ea;
        x.own(O::EZ)[l] = ez;
        // EV: v of the lane per unit of gin
        v = cmul(v, ea);
        __syncwarp();
        {
            const unsigned tl = x.tm32 + 16u * (unsigned)l;
            v = lane_scan<true, true>(v, tl + O::SU, 0u, lds2(tl + O::SU), lds2(tl + O::SX), l);
        }
        const double2 ev = shfl2_down(v, 1);
        x.own(O::EV)[l] = l == 31 ? c2(0.0, 0.0) : ev;
        double2* tot = x.own(O::tot);
        if (l == 31) tot[0] = pa;
        if (l == 0) {
            tot[1] = pw;
            tot[2] = v;
        }
    }
    if (x.C > 1) {
        cl.sync();
        if (active) reg_weights(x.own(O::tot), x.own(O::WA), x.own(O::WB), x.C, x.c);
    }
    __syncthreads();
}

// The rows of [lo, hi] that the CTA reads - its slice and one row each side -
// assembled by its own threads.  A row between two slices is written by both
// CTAs, with the same values, and each reads what it wrote: no CTA waits.
__device__ __noinline__ void reg_assemble(const ColArgs& a, const RegCtl* ctl, int lo, int hi) {
    const int first = max(lo, ctl->R0 - 1), last = min(hi, ctl->R1 + 1);
    if (first + (int)threadIdx.x <= last) {
        const RayDev ry = a.rays[ctl->rid];
        const EnvPtrs e = env_ptrs(a.envs[ctl->env], a.pool);
        for (int i = first + (int)threadIdx.x; i <= last; i += blockDim.x)
            assemble_rows(ry, e, ctl->ss, ctl->sb, ctl->iz, i, i, a.f1, a.f2, a.f3, a.ksq);
    }
    __syncthreads();
}

// The self-starter's delta in the slice and its halo (cupyram.py:1008-1022).
template <int L, bool ALL>
__device__ __noinline__ void reg_source(const ColArgs& a, RegCtx x) {
    using O = RegOff<L, ALL>;
    const RegCtl& s = *x.ctl;
    const RayDev ry = a.rays[s.rid];
    const EnvPtrs e = env_ptrs(a.envs[ry.env], a.pool);
    double2* U = x.at<double2>(O::U);
    double2* misc = x.at<double2>(O::misc);
    const double si = ry.zs / ry.dz;
    const int is = (int)floor(si);
    const double dis = si - is;
    const double amp = sqrt(2.0 * M_PI / ry.k0);
    const double step = ry.zmax / (double)(s.nz + 1);
    for (int q = 0; q < 2; ++q) {
        const int i = is + q;
        const double z = (i == s.nz + 1) ? ry.zmax : (double)i * step;
        const RowProps p = row_props(e, 0, 0, z, ry.lyrw_lambda, ry.attnf);
        const double alpw = sqrt((double)p.cw / ry.c0);
        const double wgt = (q == 0) ? (1.0 - dis) : dis;
        const double2 v = c2(wgt * amp / (ry.dz * alpw), 0.0);
        if (i < 1 || i > s.nz) continue;
        if (i >= s.R0 && i <= s.R1) U[slot_of(s.n, L, i - s.R0)] = v;
        else if (i == s.R0 - 1) misc[1] = v;
        else if (i == s.R1 + 1) misc[2] = v;
    }
}

// updat (updat.py:38-140) for step rn, by one thread: what changes, and the
// first step that has to be looked at again.  Steps in between cannot change
// the operator: the next profile, bottom segment or stability range lies
// further on, and the bottom's depth index (linear in range within a segment)
// stays in its cell; both bounds keep a step's margin for rounding.  One thread's
// seven divisions were 1.6 us of a step whose operator changes: the bounds multiply
// by reciprocals kept for the march and for the bottom's segment; the depth index
// itself is divided as the reference divides it.
__device__ __noinline__ void reg_updat(int rn, RegCtl* ctl) {
    const RegCtl& e = *ctl;
    const double dr = e.dr, r = (double)(rn + 1) * dr;
    bool reprofile = false;
    int iz = ctl->iz, ss = ctl->ss, sb = ctl->sb, bt = ctl->bt, set = ctl->set == 1 ? 2 : ctl->set;
    double stay = 1e9;  // steps that cannot change anything
    auto event = [&](double v) { stay = fmin(stay, floor(v * e.inv_dr) - 2.0 - (double)rn); };
    if (e.n_bt > 1) {
        while (bt < e.n_bt - 1 && r >= e.rb[bt + 1]) ++bt;
        const int b1 = min(bt + 1, e.n_bt - 1);
        const double r0 = e.rb[bt], r1 = e.rb[b1], z0 = e.zb[bt], z1 = e.zb[b1];
        const double zc = (b1 == bt) ? z0 : z0 + (r + 0.5 * dr - r0) * (z1 - z0) / (r1 - r0);
        iz = max(1, min(e.nz - 1, (int)floor(zc / e.dz)));
        if (b1 != bt) {
            event(r1);
            if (bt != e.per_bt) {
                ctl->per_bt = bt;
                ctl->inv_per = e.dz * (r1 - r0) / ((z1 - z0) * dr);  // infinite where the bottom is flat
            }
            const double f = zc / e.dz, inv_per = e.inv_per;
            if (z1 != z0) stay = fmin(stay, floor((inv_per > 0.0 ? floor(f) + 1.0 - f : floor(f) - f) * inv_per) - 1.0);
        }
    }
    if (e.n_rss > 1) {
        const int o2 = ss;
        while (ss < e.n_rss - 1 && r >= e.rp_ss[ss + 1]) ++ss;
        reprofile |= (ss != o2);
        if (ss < e.n_rss - 1) event(e.rp_ss[ss + 1]);
    }
    if (e.n_rsb > 1) {
        const int o2 = sb;
        while (sb < e.n_rsb - 1 && r >= e.rp_sb[sb + 1]) ++sb;
        reprofile |= (sb != o2);
        if (sb < e.n_rsb - 1) event(e.rp_sb[sb + 1]);
    }
    double rs = ctl->rs;
    if (r >= rs) {  // stability constraints off (cupyram.py:976-999)
        set = 3;
        rs = INFINITY;
    }
    if (rs < 1e300) event(rs);
    ctl->lo = reprofile ? 0 : min(ctl->iz, iz) + 1;
    ctl->hi = reprofile ? e.nz + 1 : max(ctl->iz, iz);  // iz unchanged: lo > hi
    ctl->refactor = reprofile || iz != ctl->iz || set != ctl->set;
    ctl->iz = iz;
    ctl->ss = ss;
    ctl->sb = sb;
    ctl->bt = bt;
    ctl->set = set;
    ctl->rs = rs;
    ctl->next = rn + (int)fmax(1.0, fmin(stay, 1e9));
}

// f3 of rows max(lo, R0 - 1) .. min(hi, R1 + 1) into shared memory, and the
// weights of the line's rows with it.
template <int L, bool ALL>
__device__ __noinline__ void reg_load_f3(const ColArgs& a, RegCtx x, int lo, int hi) {
    float* F3 = x.at<float>(RegOff<L, ALL>::F3(blockDim.x >> 5));
    RegCtl* ctl = x.ctl;
    const int first = max(lo, ctl->R0 - 1), last = a.compute_grids ? min(hi, ctl->R1 + 1) : -1;
    for (int i = first + (int)threadIdx.x; i <= last; i += blockDim.x)
        F3[i - (ctl->R0 - 1)] = a.f3[ctl->col + (long long)i * kTile];
    if (threadIdx.x == 0 && ctl->line >= 0) {
        const double dir = ctl->line_dir;
        const long long o = ctl->col + (long long)ctl->line_row * kTile;
        ctl->wa = (1.0 - dir) * (double)a.f3[o];
        ctl->wb = dir * (double)a.f3[o + kTile];
    }
}

// Offset of the field of a row in [R0 - 1, R1 + 1].
template <int L, bool ALL>
__device__ __forceinline__ unsigned u_offset(const RegCtl& s, int row) {
    using O = RegOff<L, ALL>;
    if (row < 1 || row > s.nz) return O::misc + 48;
    if (row == s.R0 - 1) return O::misc + 16;
    if (row == s.R1 + 1) return O::misc + 32;
    return O::U + 16u * (unsigned)slot_of(s.n, L, row - s.R0);
}

// The outputs' part of the CTA's state (one thread).
template <int L, bool ALL>
__device__ __noinline__ void reg_outputs(const ColArgs& a, RegCtl* ctl) {
    const RayDev& ry = a.rays[ctl->rid];
    const int ir = (int)floor(ry.zr / ry.dz), irow = max(ir, 1);
    const bool mine = irow >= ctl->R0 && irow <= ctl->R1;
    ctl->line = mine ? ry.line_off : -1;
    ctl->line_row = ir;
    ctl->line_dir = ry.zr / ry.dz - ir;
    ctl->ua = mine ? u_offset<L, ALL>(*ctl, ir) : 0;
    ctl->ub = mine ? u_offset<L, ALL>(*ctl, ir + 1) : 0;
    ctl->grid = a.compute_grids ? ry.grid_off : -1;
    ctl->ndz = (unsigned)ry.ndz;
    ctl->ndz_inv = ry.ndz > 1 ? (unsigned)((0x100000000ull + ry.ndz - 1) / (unsigned)ry.ndz) : 0u;
    ctl->nvz = ry.nvz;
}

// The sum over N terms (ALL) or pairs of terms of the rows j = k, k + terms, ..
// of this lane (and outputs among them).
template <int L, bool ALL, int N>
__device__ __forceinline__ void reg_sum(const ColArgs& a, const RegCtx& x, double2 ci, int k, int l, int terms,
                                        int out) {
    using O = RegOff<L, ALL>;
    constexpr unsigned P16 = 512u * L;
    const unsigned us = x.sm32 + O::U + 16u * (unsigned)l, xs0 = x.sm32 + O::X(terms) + 16u * (unsigned)l;
#pragma unroll 1
    for (int j = k; j < L; j += terms) {
        const unsigned ua = us + 512u * (unsigned)j, xa = xs0 + 512u * (unsigned)j;
        double2 xs[N];
#pragma unroll
        for (int q = 0; q < N; ++q) xs[q] = lds2(xa + (unsigned)q * P16);
        double2 acc = cmul(ci, lds2(ua));
        if (ALL) {  // two chains of c_k x_k
            double2 other = c2(0.0, 0.0);
#pragma unroll
            for (int q = 0; q < N; ++q) {
                const double2 ck = lds2(x.sm32 + O::ck + 16u * (unsigned)q);
                if (q & 1) other = vfma(ck, xs[q], other);
                else acc = vfma(ck, xs[q], acc);
            }
            acc = cadd(acc, other);
        } else {
#pragma unroll
            for (int q = 0; q < N; ++q) acc = cadd(acc, xs[q]);
        }
        // positions without a row stay zero
        if (j >= x.npad) sts2(ua, acc);
        if (a.compute_grids && out >= 0 && x.ctl->grid >= 0 && j >= x.npad) {
            const RegCtl* ctl = x.ctl;
            int start, cnt;
            lane_rows(ctl->n, l, start, cnt);
            const unsigned row = (unsigned)(ctl->R0 + start + j - x.npad);
            const unsigned q = ctl->ndz_inv ? __umulhi(row, ctl->ndz_inv) : row;  // row / ndz (row ndz < 2^32)
            if (q * ctl->ndz == row && (int)q <= ctl->nvz && q > 0) {
                const double f = x.at<float>(O::F3(terms))[(int)row - (ctl->R0 - 1)];
                a.cpg[ctl->grid + (long long)(q - 1) * ctl->nvr + out] = c2(acc.x * f, acc.y * f);
            }
        }
    }
}

// One range step of the active set; out >= 0: the step's field is output
// `out` (outpt.py:11-57; transmission loss follows at the end, reg_tl).
// step: index of the step, the self-starter's three included.
template <int L, bool ALL>
__device__ __forceinline__ void reg_step(const ColArgs& a, const RegCtx& x, int na, const double2 (&al)[L],
                                         const double2 (&mw)[L], int step, int out) {
    using O = RegOff<L, ALL>;
    constexpr unsigned P16 = 512u * L;  // bytes of a per-row table
    const int k = x.term, l = x.lane, terms = (int)(blockDim.x >> 5);
    const unsigned sm = x.sm32, tm = x.tm32, us = sm + O::U + 16u * (unsigned)l;
    RegCtl* ctl = x.ctl;
    const int half = (na + 1) >> 1;
    if (k < na) {
        const unsigned tl = tm + 16u * (unsigned)l;  // this lane's entries of the term's tables
        // Tables are read ahead of their use where registers are left for it; with 12
        // rows a lane the factors and the workspace take 144 of the 168.
        constexpr bool kAhead = L <= 10;
        const int npad = x.npad;
        double2 g[L];
        // h down the lane's rows, then y up
        double2 h = c2(0.0, 0.0), y = h, m, sx;
        {
            const unsigned edges = lds1(sm + O::edges + 4u * (unsigned)l);
            double2 up = lds2(sm + (edges & 0xffffu));
#pragma unroll
            for (int j = 0; j < L; ++j) g[j] = lds2(us + j * 512u);
            double2 after, q0, q1;
            if (kAhead) {
                after = lds2(sm + (edges >> 16));
                q0 = lds2(tl + O::Q);
                if (L > 1) q1 = lds2(tl + O::Q + 512u);
            }
#pragma unroll
            for (int j = 0; j < kMaxPad && j < L; ++j)
                if (j < npad) g[j] = up;
#pragma unroll
            for (int j = 0; j < L; ++j) {
                double2 q;
                if (kAhead) {
                    q = q0;
                    q0 = q1;
                    if (j + 2 < L) q1 = lds2(tl + O::Q + (j + 2) * 512u);
                } else {
                    q = lds2(tl + O::Q + j * 512u);
                    if (j + 1 == L) after = lds2(sm + (edges >> 16));
                }
                const double2 uc = g[j], un = j + 1 < L ? g[j + 1 < L ? j + 1 : 0] : after;
                const double2 b = c2(fma(4.0, uc.x, up.x + un.x), fma(4.0, uc.y, up.y + un.y));
                h = vfma(al[j], h, cmul(q, b));
                up = uc;
                g[j] = h;
            }
            if (kAhead) m = lds2(tl + O::SD);
#pragma unroll
            for (int j = L - 1; j >= 0; --j)
                y = vfma(mw[j], y, (j < kMaxPad && j < npad) ? c2(0.0, 0.0) : g[j]);
        }
        // e of every lane, the slice alone
        if (kAhead) sx = lds2(tl + O::SX);
        h = lane_scan<false, kAhead>(h, tl + O::SD, tl + O::SX, m, sx, l);
        double2 e = shfl2_up(h, 1);
        if (l == 0) e = c2(0.0, 0.0);
        // the mailbox of this step: the two alternate over the term's active steps
        const unsigned used = (unsigned)step - lds1(sm + O::ctl + (unsigned)offsetof(RegCtl, idle) + 4u * (unsigned)k);
        const unsigned box = used & 1u, par = (used >> 1) & 1u;
        const unsigned to = x.C > 1 ? remote_addr(tm + O::mail + 512u * box + 32u * (unsigned)x.c,
                                                  (unsigned)min(l, x.C - 1)) : 0u;
        const unsigned to_bar = to - 512u * box - 32u * (unsigned)x.c + (O::bar - O::mail) + 8u * box;
        if (x.C > 1) {
            const double2 t = shfl2(h, 31);
            if (l < x.C) mail_send(to, to_bar, t);
        }
        // v of every lane, the slice alone
        const double2 V = lds2(tl + O::V);
        if (kAhead) m = lds2(tl + O::SU);
        y = lane_scan<true, kAhead>(vfma(V, e, y), tl + O::SU, tl + O::SX, m, sx, l);
        double2 v = shfl2_down(y, 1);
        if (l == 31) v = c2(0.0, 0.0);
        if (x.C > 1) {
            const double2 t = shfl2(y, 0);
            if (l < x.C) mail_send(to + 16u, to_bar, t);
            double2 wa, wb, ea, ez, ev;
            if (kAhead) {
                wa = lds2(tl + O::WA);
                wb = lds2(tl + O::WB);
            }
            if (!ctl->dead && !mail_wait(tm + O::bar + 8u * box, 32u * (unsigned)x.C, par, l)) ctl->dead = 1;
            // lanes 0..15 fold gin, lanes 16..31 xin: lane j the values of CTA j % 16
            // (the weights of CTAs that are not there, and of y in gin, are zero)
            const unsigned mb = tm + O::mail + 512u * box + 32u * (unsigned)(l & 15);
            if (!kAhead) {
                wa = lds2(tl + O::WA);
                wb = lds2(tl + O::WB);
            }
            const double2 mh = lds2(mb), my = lds2(mb + 16u);
            if (kAhead) {
                ea = lds2(tl + O::EA);
                ez = lds2(tl + O::EZ);
                ev = lds2(tl + O::EV);
            }
            double2 f = vfma(wb, my, cmul(wa, mh));
#pragma unroll
            for (int d = 8; d >= 1; d >>= 1) f = cadd(f, shfl2_xor(f, d));
            const double2 other = shfl2_xor(f, 16);
            const double2 gin = l < 16 ? f : other, xin = l < 16 ? other : f;
            // for the halo rows, once the lane's x are known
            if (l == 0) sts2(tm + O::xh, gin);
            if (l == 0) sts2(tm + O::xh + 16u, xin);
            if (!kAhead) ea = lds2(tl + O::EA);
            e = vfma(ea, gin, e);
            if (!kAhead) ev = lds2(tl + O::EV);
            v = vfma(ev, gin, v);
            if (!kAhead) ez = lds2(tl + O::EZ);
            v = vfma(ez, xin, v);
        }
        // true g, then true x
#pragma unroll
        for (int j = 0; j < L; ++j) {
            e = cmul(al[j], e);
            g[j] = cadd(g[j], e);
        }
#pragma unroll
        for (int j = L - 1; j >= 0; --j) {
            v = vfma(mw[j], v, (j < kMaxPad && j < npad) ? c2(0.0, 0.0) : g[j]);
            g[j] = v;
        }
        const double2 ck = lds2(sm + O::ck + 16u * (unsigned)k);
        if (l == 0) {
            // x of row R1 + 1 is the entry from below; x of row R0 - 1 is
            // g_{R0-1} - w_{R0-1} x_{R0}, g_{R0-1} being the entry from above
            sts2(tm + O::xh, cmul(ck, vfma(lds2(tm + O::wghost), v, lds2(tm + O::xh))));
            sts2(tm + O::xh + 16u, cmul(ck, lds2(tm + O::xh + 16u)));
        }
        // the terms' share of the sum
        const bool up_warp = !ALL && k >= half;
        const unsigned xa = sm + O::X(terms) + 16u * (unsigned)l + (unsigned)(up_warp ? k - half : k) * P16;
        if (ALL) {
#pragma unroll
            for (int j = 0; j < L; ++j) sts2(xa + j * 512u, g[j]);
        } else if (up_warp || k + half < na) {
            // warps k and k + half are a pair: each leaves the other's half of the rows
            // and adds its own half to what the other left
            constexpr int H = L / 2;
            if (up_warp) {
#pragma unroll
                for (int j = 0; j < H; ++j) sts2(xa + j * 512u, cmul(ck, g[j]));
                asm volatile("bar.sync %0, 64;" ::"r"(1 + k - half) : "memory");
#pragma unroll
                for (int j = H; j < L; ++j) sts2(xa + j * 512u, vfma(ck, g[j], lds2(xa + j * 512u)));
            } else {
#pragma unroll
                for (int j = H; j < L; ++j) sts2(xa + j * 512u, cmul(ck, g[j]));
                asm volatile("bar.sync %0, 64;" ::"r"(1 + k) : "memory");
#pragma unroll
                for (int j = 0; j < H; ++j) sts2(xa + j * 512u, vfma(ck, g[j], lds2(xa + j * 512u)));
            }
        } else {
#pragma unroll
            for (int j = 0; j < L; ++j) sts2(xa + j * 512u, cmul(ck, g[j]));
        }
    }
    __syncthreads();
    // u = c_inf u + the terms' or pairs' sums
    const double2 ci = lds2(sm + O::misc);
    if constexpr (ALL) {
        switch (na) {
            case 1: reg_sum<L, ALL, 1>(a, x, ci, k, l, terms, out); break;
            case 2: reg_sum<L, ALL, 2>(a, x, ci, k, l, terms, out); break;
            case 3: reg_sum<L, ALL, 3>(a, x, ci, k, l, terms, out); break;
            case 4: reg_sum<L, ALL, 4>(a, x, ci, k, l, terms, out); break;
            case 5: reg_sum<L, ALL, 5>(a, x, ci, k, l, terms, out); break;
            case 6: reg_sum<L, ALL, 6>(a, x, ci, k, l, terms, out); break;
            case 7: reg_sum<L, ALL, 7>(a, x, ci, k, l, terms, out); break;
            case 8: reg_sum<L, ALL, 8>(a, x, ci, k, l, terms, out); break;
            case 9: reg_sum<L, ALL, 9>(a, x, ci, k, l, terms, out); break;
            default: reg_sum<L, ALL, 10>(a, x, ci, k, l, terms, out); break;
        }
    } else {
        switch (half) {
            case 1: reg_sum<L, ALL, 1>(a, x, ci, k, l, terms, out); break;
            case 2: reg_sum<L, ALL, 2>(a, x, ci, k, l, terms, out); break;
            case 3: reg_sum<L, ALL, 3>(a, x, ci, k, l, terms, out); break;
            case 4: reg_sum<L, ALL, 4>(a, x, ci, k, l, terms, out); break;
            default: reg_sum<L, ALL, 5>(a, x, ci, k, l, terms, out); break;
        }
    }
    if (k == terms - 1) {
        // halo rows outside the column (rows 0 and nz + 1) stay zero: lane 2 t + h
        // takes term t of the halo row above (h = 0) or below
        const unsigned t = (unsigned)l >> 1, hh = (unsigned)l & 1u;
        const double2 old = lds2(sm + O::misc + 16u + 16u * hh);
        double2 acc = lds2(sm + O::term0 + min((int)t, na - 1) * O::term + O::xh + 16u * hh);
        if ((int)t >= na) acc = c2(0.0, 0.0);
#pragma unroll
        for (int d = 16; d >= 2; d >>= 1) acc = cadd(acc, shfl2_xor(acc, d));
        if (l < 2) {
            const bool inside = l == 0 ? ctl->R0 > 1 : ctl->R1 < ctl->nz;
            acc = vfma(ci, old, acc);
            sts2(sm + O::misc + 16u + 16u * hh, inside ? acc : c2(0.0, 0.0));
            if (a.compute_grids && out >= 0 && l == 1 && !inside && ctl->grid >= 0) {  // grid row nz + 1: zero
                const unsigned row = (unsigned)ctl->nz + 1u, q = row / ctl->ndz;
                if (q * ctl->ndz == row && (int)q <= ctl->nvz)
                    a.cpg[ctl->grid + (long long)(q - 1) * ctl->nvr + out] = c2(0.0, 0.0);
            }
        }
    }
    __syncthreads();
    if (out >= 0 && threadIdx.x == 0 && ctl->line >= 0) {
        const double2 ua = lds2(sm + ctl->ua), ub = lds2(sm + ctl->ub);
        a.cpl[ctl->line + out] = c2(ctl->wa * ua.x + ctl->wb * ub.x, ctl->wa * ua.y + ctl->wb * ub.y);
    }
}

// Transmission loss of the emitted outputs from their complex pressure
// (outpt.py:11-57), shared by the cluster's threads; a non-finite line value
// flags the ray.
__device__ __noinline__ void reg_tl(const ColArgs& a, int rid, int C, int c, int n_out) {
    const RayDev& ry = a.rays[rid];
    const int tid = c * blockDim.x + threadIdx.x, nt = C * blockDim.x;
    int bad = 0;
    for (int t = tid; t < n_out; t += nt) {
        const double2 cp = a.cpl[ry.line_off + t];
        const double amp = hypot(cp.x, cp.y);
        bad |= !isfinite(amp);
        a.tll[ry.line_off + t] = tl_db(amp, (double)((t + 1) * ry.ndr) * ry.dr);
    }
    if (bad) atomicOr(a.flags + rid, 1);
    if (a.compute_grids && ry.grid_off >= 0) {
        const long long total = (long long)ry.nvz * n_out;
        for (long long q = tid; q < total; q += nt) {
            const int j = (int)(q / n_out), t = (int)(q % n_out);
            const long long o = ry.grid_off + (long long)j * ry.nvr + t;
            const double2 g = a.cpg[o];
            a.tlg[o] = tl_db(hypot(g.x, g.y), (double)((t + 1) * ry.ndr) * ry.dr);
        }
    }
}

// Registers of a thread: 8 L hold the factors, 4 L the workspace.  The longest
// segments are held to what two CTAs of six warps can share an SM with.
template <int L>
constexpr int reg_cap() { return L >= 8 ? 168 : 128; }

template <int L, bool ALL>
__global__ void __maxnreg__(reg_cap<L>()) march_reg_kernel(const __grid_constant__ ColArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using O = RegOff<L, ALL>;
    cg::cluster_group cl = cg::this_cluster();
    RegCtx x;
    x.sm = smem_raw;
    x.C = (int)cl.num_blocks();
    x.c = (int)cl.block_rank();
    x.term = threadIdx.x >> 5;
    x.lane = threadIdx.x & 31;
    x.tm = smem_raw + O::term0 + (unsigned)x.term * O::term;
    x.sm32 = smem_u32(x.sm);
    x.tm32 = smem_u32(x.tm);
    RegCtl* ctl = x.ctl = x.at<RegCtl>(O::ctl);
    double2* misc = x.at<double2>(O::misc);
    if (threadIdx.x == 0) {
        const int rid = a.col_ray[blockIdx.x / x.C];
        const RayDev& ry = a.rays[rid];
        const EnvPtrs e = env_ptrs(a.envs[ry.env], a.pool);
        if (x.c == 0) a.flags[rid] = 0;
        ctl->rid = rid;
        ctl->nz = ry.nz;
        slice_of(ry.nz, x.C, x.c, ctl->R0, ctl->R1);
        ctl->n = ctl->R1 - ctl->R0 + 1;
        ctl->col = ry.col;
        ctl->cfact = 0.5 / (ry.dz * ry.dz);
        ctl->a1 = ry.k0 * ry.k0 / 6.0;
        ctl->a2 = 2.0 * ry.k0 * ry.k0 / 3.0;
        ctl->seg = ((ry.nz + x.C - 1) / x.C + 31) / 32;
        ctl->nvr = ry.nvr;
        ctl->ndr = ry.ndr;
        ctl->iz = max(1, min(ry.nz - 1, (int)floor(e.zb[0] / ry.dz)));
        ctl->ss = ctl->sb = ctl->bt = 0;
        ctl->set = -1;
        ctl->next = 0;
        ctl->dead = 0;
        ctl->rs = ry.rs;
        ctl->env = ry.env;
        ctl->dr = ry.dr;
        ctl->dz = ry.dz;
        ctl->inv_dr = 1.0 / ry.dr;
        ctl->per_bt = -1;
        ctl->n_bt = e.n_bt;
        ctl->n_rss = e.n_rss;
        ctl->n_rsb = e.n_rsb;
        ctl->rb = e.rb;
        ctl->zb = e.zb;
        ctl->rp_ss = e.rp_ss;
        ctl->rp_sb = e.rp_sb;
        misc[1] = misc[2] = misc[3] = c2(0.0, 0.0);
        for (int k = 0; k < 2 * (int)(blockDim.x >> 5); ++k)
            mbar_init1(x.at<unsigned long long>(O::term0 + (unsigned)(k >> 1) * O::term + O::bar) + (k & 1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int p = threadIdx.x; p < 32 * L; p += blockDim.x) x.at<double2>(O::U)[p] = c2(0.0, 0.0);
    if (x.lane == 0) ctl->idle[x.term] = 0u;
    x.own(O::mail)[x.lane] = x.own(O::mail)[32 + x.lane] = c2(0.0, 0.0);
    __syncthreads();
    reg_assemble(a, ctl, 0, ctl->nz + 1);
    if (threadIdx.x == 0) {
        reg_source<L, ALL>(a, x);
        reg_outputs<L, ALL>(a, ctl);
    }
    cl.sync();  // every CTA's mailboxes are ready
    reg_load_f3<L, ALL>(a, x, 0, ctl->nz + 1);
    const int n = ctl->n;
    {
        int start, cnt;
        lane_rows(n, x.lane, start, cnt);
        x.npad = L - cnt;
        x.row0 = ctl->R0 + start;
    }
    // the field above and below each lane's rows: a neighbouring lane's row or the halo
    if (x.term == 0) {
        const int low = 32 - (n & 31), base = n >> 5, next = x.lane + 1;
        const bool top = x.lane == 0 || (base == 0 && x.lane <= low);
        const int npad_next = min(L - (next < low ? base : base + 1), L - 1);
        unsigned edges = top ? O::misc + 16 : O::U + 16u * (unsigned)((L - 1) * 32 + x.lane - 1);
        edges |= (x.lane == 31 ? O::misc + 32 : O::U + 16u * (unsigned)(npad_next * 32 + next)) << 16;
        x.at<unsigned>(O::edges)[x.lane] = edges;
    }

    // steps: two of 1/(1-X), one of the ip=2 operator (first output, at r = dr:
    // cupyram.py:703), then nr of the march
    double2 al[L], mw[L];
    const int steps = a.rays[ctl->rid].nr + 3;
    int na = 0, due = ctl->ndr, tlc = 0, stop;
#pragma unroll 1
    for (int s = 0; s < steps; s = stop) {
        int want = s == 0 ? 0 : 1;
        bool refactor = true;
        const int set = ctl->set;
        stop = s == 0 ? 2 : 3;
        if (s >= 3) {
            __syncthreads();
            if (threadIdx.x == 0) reg_updat(s - 3, ctl);
            __syncthreads();
            stop = min(steps, ctl->next + 3);
            want = ctl->set;
            refactor = ctl->refactor;
            if (ctl->lo <= ctl->hi) {
                reg_assemble(a, ctl, ctl->lo, ctl->hi);
                reg_load_f3<L, ALL>(a, x, ctl->lo, ctl->hi);
            }
        }
        if (refactor) {
            if (want != set) {
                na = a.pd_n[ctl->rid * kSets + want];
                const long long base = ((long long)ctl->rid * kSets + want) * CR_MAX_NP;
                if (threadIdx.x < kRegMaxTerms)
                    x.at<double2>(O::ck)[threadIdx.x] =
                        (int)threadIdx.x < na ? a.pfc[base + threadIdx.x] : c2(0.0, 0.0);
                if (threadIdx.x == 0) misc[0] = a.pfcinf[(long long)ctl->rid * kSets + want];
            }
            reg_factor<L, ALL>(a, x, cl, want, na, al, mw);
            if (threadIdx.x == 0) ctl->set = want;
        }
        // the steps that this operator serves
#pragma unroll 1
        for (int q = s; q < stop; ++q) {
            int out = -1;
            if (q >= 2 && --due == 0) {
                due = ctl->ndr;
                if (tlc < ctl->nvr) out = tlc;
                ++tlc;
            }
            reg_step<L, ALL>(a, x, na, al, mw, q, out);
        }
        if (x.term >= na && x.lane == 0) ctl->idle[x.term] += (unsigned)(stop - s);
    }
    if (threadIdx.x == 0 && ctl->dead) atomicOr(a.flags + ctl->rid, 2);
    __threadfence();
    cl.sync();  // every complex pressure is stored; no CTA still reads or writes another's shared memory
    reg_tl(a, ctl->rid, x.C, x.c, min(tlc, ctl->nvr));
}

constexpr int kRows[] = {1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12};

// Longest segment whose terms may each leave their solution to the sum (see
// reg_kernel): longer ones need the room.
constexpr int kAllRows = 9;

// The kernel of L rows a lane and its shared memory.
struct RegKernel {
    const void* f = nullptr;
    unsigned (*bytes)(int terms, int nmax, int grids) = nullptr;
    int regs = 0;
};
template <int L, bool ALL>
RegKernel reg_kernel_of() { return {(const void*)march_reg_kernel<L, ALL>, RegOff<L, ALL>::bytes, reg_cap<L>()}; }
template <int L>
RegKernel reg_kernel_at(bool all) {
    if constexpr (L <= kAllRows)
        if (all) return reg_kernel_of<L, true>();
    return reg_kernel_of<L, false>();
}
RegKernel reg_kernel(int L, bool all) {
    switch (L) {
        case 1: return reg_kernel_at<1>(all);
        case 2: return reg_kernel_at<2>(all);
        case 3: return reg_kernel_at<3>(all);
        case 4: return reg_kernel_at<4>(all);
        case 5: return reg_kernel_at<5>(all);
        case 6: return reg_kernel_at<6>(all);
        case 7: return reg_kernel_at<7>(all);
        case 8: return reg_kernel_at<8>(all);
        case 9: return reg_kernel_at<9>(all);
        case 10: return reg_kernel_at<10>(all);
        case 11: return reg_kernel_at<11>(all);
        case 12: return reg_kernel_at<12>(all);
    }
    return {};
}
// Every term leaves its x to the sum - no pairs that wait for one another - where
// that takes no CTA off an SM.
RegKernel reg_kernel(int L, int terms, int nmax, int grids) {
    const RegKernel pairs = reg_kernel(L, false), all = reg_kernel(L, true);
    if (!pairs.f || all.f == pairs.f) return pairs;
    const int by_regs = 65536 / (pairs.regs * 32 * terms);
    auto ctas = [&](const RegKernel& kn) {
        return std::min(by_regs, (int)(228 * 1024 / (kn.bytes(terms, nmax, grids) + 1024)));
    };
    return all.bytes(terms, nmax, grids) <= kRegSmemLimit && ctas(all) >= ctas(pairs) ? all : pairs;
}

cudaError_t reg_config(const RegKernel& kn, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int n_rays, int cluster,
                       int terms, int nz_max, int grids, cudaStream_t st) {
    const void* f = kn.f;
    const size_t smem = kn.bytes(terms, (nz_max + cluster - 1) / cluster, grids);
    if (smem > kRegSmemLimit) return cudaErrorInvalidValue;
    cudaError_t ce = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRegSmemLimit);
    if (ce == cudaSuccess && cluster > 8)
        ce = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (ce != cudaSuccess) return ce;
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3((unsigned)(n_rays * cluster), 1, 1);
    cfg.blockDim = dim3((unsigned)(32 * terms), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaSuccess;
}

bool reg_shape_ok(int cluster, int terms, int rows) {
    return terms >= 1 && terms <= kRegMaxTerms && cluster >= 1 && cluster <= kRegMaxCluster && reg_kernel(rows, false).f;
}

}  // namespace

int reg_rows(int nz, int cluster) {
    const int n = (nz + cluster - 1) / cluster, need = (n + 31) / 32;
    if (cluster > nz) return 0;
    for (int L : kRows)
        if (L >= need) return L;  // at most one more than needed: two positions of a lane may hold no row
    return 0;
}

cudaError_t launch_march_reg(const ColArgs& a, int n_rays, int cluster, int terms, int rows, int nz_max,
                             cudaStream_t st) {
    if (!reg_shape_ok(cluster, terms, rows)) return cudaErrorInvalidValue;
    const RegKernel kn = reg_kernel(rows, terms, (nz_max + cluster - 1) / cluster, a.compute_grids);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    cudaError_t ce = reg_config(kn, cfg, attr, n_rays, cluster, terms, nz_max, a.compute_grids, st);
    if (ce != cudaSuccess) return ce;
    void* args[] = {const_cast<ColArgs*>(&a)};
    ce = cudaLaunchKernelExC(&cfg, kn.f, args);
    return ce != cudaSuccess ? ce : cudaGetLastError();
}

int reg_max_active_clusters(int cluster, int terms, int rows, int nz_max, int grids) {
    if (!reg_shape_ok(cluster, terms, rows)) return 0;
    const RegKernel kn = reg_kernel(rows, terms, (nz_max + cluster - 1) / cluster, grids);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    if (reg_config(kn, cfg, attr, 1, cluster, terms, nz_max, grids, 0) != cudaSuccess) return 0;
    int n = 0;
    return cudaOccupancyMaxActiveClusters(&n, kn.f, &cfg) == cudaSuccess ? n : 0;
}

}  // namespace crk
