// mlp.cu - BF16 tensor-core kernels of the learned surrogate (training and
// inference of its MLP ensemble), FP32 accumulation.
//
// Every contraction of the MLP is one kernel, C = A B^T with both operands
// K-contiguous ("TN"):
//     forward        Y[B,N]  = X[B,K]  W[N,K]^T            (+ bias, ReLU)
//     input grad     dX[B,K] = dY[B,N] (W^T)[K,N]^T         (x ReLU mask)
//     weight grad    dW[N,K] = (dY^T)[N,B] (X^T)[K,B]^T
// with transposed BF16 copies of W, dY and X made by a tiled transpose.
//
// Shapes with N a multiple of 256 and K of 64 run on the 5th-generation tensor
// cores (tcgen05.mma, accumulators in tensor memory, operands and results moved
// by the tensor memory accelerator): gemm_tn_tile, gemm_tn_persistent for large
// outputs, ensemble_tile for an ensemble's output layers.  gemm_tn_tma takes
// outputs and masks whose rows do not start on 16-byte boundaries, gemm_tn_umma
// (operands by cp.async) stands behind CUPYRAM_B200_GEMM=cp.
//
// Other shapes run on gemm_tn: 128 x 32 tiles of A and B staged in shared memory
// with cp.async (two stages, XOR-swizzled 16-byte chunks so that ldmatrix reads
// are conflict-free), each of 8 warps running mma.sync m16n8k16 (bf16 x bf16 ->
// f32) on a 64 x 32 piece of the 128 x 128 block.  Shapes must be multiples of
// the tile (M, N of 128, K of 32); the host wrappers check that and the 16-byte
// alignment of every row.
//
// Plus the small kernels of a training step: column sums (bias gradients),
// the masked mean-squared-error gradient, Adam, and BF16 conversion.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>

#include "../../include/cupyram_b200_mlp.h"
#include "tensor_map.h"

namespace {

constexpr int BM = 128, BN = 128, BK = 32;
constexpr int kThreads = 256;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(smem_u32(p)));
}
__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Shared tile: 128 rows x 32 bf16 (four 16-byte chunks per row); chunk c of
// row r is stored at chunk c ^ ((r >> 1) & 3).
__device__ __forceinline__ int swz(int row, int chunk) { return row * BK + ((chunk ^ ((row >> 1) & 3)) << 3); }

struct EpiArgs {
    void* out;
    int ldo;
    const float* bias;
    const __nv_bfloat16* mask;
    int ldm;
};

template <int EPI>
__device__ __forceinline__ void store2(const EpiArgs& e, int row, int col, float v0, float v1) {
    if (EPI == CR_MLP_EPI_BIAS_RELU_BF16) {
        v0 = fmaxf(v0 + e.bias[col], 0.f);
        v1 = fmaxf(v1 + e.bias[col + 1], 0.f);
        *reinterpret_cast<__nv_bfloat162*>((__nv_bfloat16*)e.out + (size_t)row * e.ldo + col) =
            __floats2bfloat162_rn(v0, v1);
    } else if (EPI == CR_MLP_EPI_BIAS_F32) {
        *reinterpret_cast<float2*>((float*)e.out + (size_t)row * e.ldo + col) =
            make_float2(v0 + e.bias[col], v1 + e.bias[col + 1]);
    } else if (EPI == CR_MLP_EPI_F32) {
        *reinterpret_cast<float2*>((float*)e.out + (size_t)row * e.ldo + col) = make_float2(v0, v1);
    } else {  // CR_MLP_EPI_RELU_MASK_BF16: gradient through the ReLU whose output is `mask`
        const __nv_bfloat162 m = *reinterpret_cast<const __nv_bfloat162*>(e.mask + (size_t)row * e.ldm + col);
        v0 = __bfloat162float(m.x) > 0.f ? v0 : 0.f;
        v1 = __bfloat162float(m.y) > 0.f ? v1 : 0.f;
        *reinterpret_cast<__nv_bfloat162*>((__nv_bfloat16*)e.out + (size_t)row * e.ldo + col) =
            __floats2bfloat162_rn(v0, v1);
    }
}

template <int EPI>
__device__ __forceinline__ void store1(const EpiArgs& e, int row, int col, float v) {
    if (EPI == CR_MLP_EPI_BIAS_RELU_BF16) {
        ((__nv_bfloat16*)e.out)[(size_t)row * e.ldo + col] = __float2bfloat16_rn(fmaxf(v + e.bias[col], 0.f));
    } else if (EPI == CR_MLP_EPI_BIAS_F32) {
        ((float*)e.out)[(size_t)row * e.ldo + col] = v + e.bias[col];
    } else if (EPI == CR_MLP_EPI_F32) {
        ((float*)e.out)[(size_t)row * e.ldo + col] = v;
    } else {  // CR_MLP_EPI_RELU_MASK_BF16
        const float m = __bfloat162float(e.mask[(size_t)row * e.ldm + col]);
        ((__nv_bfloat16*)e.out)[(size_t)row * e.ldo + col] = __float2bfloat16_rn(m > 0.f ? v : 0.f);
    }
}

template <int EPI>
__global__ void __launch_bounds__(kThreads) gemm_tn(const __nv_bfloat16* __restrict__ A,
                                                     const __nv_bfloat16* __restrict__ B, int K, int lda, int ldb,
                                                     EpiArgs e) {
    __shared__ __align__(128) __nv_bfloat16 sA[2][BM * BK];
    __shared__ __align__(128) __nv_bfloat16 sB[2][BN * BK];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp & 1, wn = warp >> 1;  // 2 x 4 warps: 64 rows x 32 columns each
    const int bm = blockIdx.y * BM, bn = blockIdx.x * BN;
    const __nv_bfloat16* Ab = A + (size_t)bm * lda;
    const __nv_bfloat16* Bb = B + (size_t)bn * ldb;

    auto load = [&](int stage, int k0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int c = tid + i * kThreads;  // 512 chunks of 16 bytes per tile
            const int row = c >> 2, ch = c & 3;
            cp_async16(&sA[stage][swz(row, ch)], Ab + (size_t)row * lda + k0 + ch * 8);
            cp_async16(&sB[stage][swz(row, ch)], Bb + (size_t)row * ldb + k0 + ch * 8);
        }
        cp_commit();
    };

    float acc[4][4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;

    const int nk = K / BK;
    load(0, 0);
    for (int kt = 0; kt < nk; ++kt) {
        const int st = kt & 1;
        if (kt + 1 < nk) {
            load(st ^ 1, (kt + 1) * BK);
            cp_wait<1>();
        } else {
            cp_wait<0>();
        }
        __syncthreads();
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            uint32_t a[4][4], b[4][2];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) {
                const int row = wm * 64 + mi * 16 + (lane & 15);
                ldsm_x4(a[mi][0], a[mi][1], a[mi][2], a[mi][3], &sA[st][swz(row, ks * 2 + (lane >> 4))]);
            }
#pragma unroll
            for (int nj = 0; nj < 2; ++nj) {
                const int row = wn * 32 + nj * 16 + (lane & 7) + ((lane >> 4) << 3);
                ldsm_x4(b[2 * nj][0], b[2 * nj][1], b[2 * nj + 1][0], b[2 * nj + 1][1],
                        &sB[st][swz(row, ks * 2 + ((lane >> 3) & 1))]);
            }
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) mma_bf16(acc[mi][ni], a[mi], b[ni][0], b[ni][1]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
            const int row = bm + wm * 64 + mi * 16 + (lane >> 2);
            const int col = bn + wn * 32 + ni * 8 + (lane & 3) * 2;
            store2<EPI>(e, row, col, acc[mi][ni][0], acc[mi][ni][1]);
            store2<EPI>(e, row + 8, col, acc[mi][ni][2], acc[mi][ni][3]);
        }
}

// ---------------------------------------------------------------------------
// The same contraction on the 5th-generation tensor cores (tcgen05).
//
// A CTA of 4 warps owns a 128 x 256 block of C; its FP32 accumulator lives in
// tensor memory (128 lanes x 256 columns, so two CTAs share an SM's 512).  A
// tiles of 128 rows and B tiles of 256 rows x 64 bf16 (one 128-byte swizzle
// atom wide) are staged in shared memory by
// cp.async in the canonical K-major SWIZZLE_128B layout - row r at r x 128
// bytes, its 16-byte chunk c at chunk c ^ (r mod 8) - over two stages.  One
// thread issues the four m128 n256 k16 MMAs of a stage and commits them to
// the stage's mbarrier; the stage is refilled once that barrier flips.  The
// epilogue reads the accumulator with tcgen05.ld (warp w: lanes 32w..32w+31,
// i.e. rows 32w..32w+31 of the block), transposes 32 x 32 pieces through
// shared memory so that each store writes 32 consecutive columns of one row,
// and applies the same epilogues as the mma.sync kernel.  Every wait is bounded: a barrier that does not flip in
// time sets *err and the kernel finishes without the result.
// ---------------------------------------------------------------------------
constexpr int UBM = 128, UBN = 256, UBK = 64;
constexpr int kUThreads = 128;
constexpr int kUTileA = UBM * UBK * 2;      // bytes of one stage's A tile
constexpr int kUTileB = UBN * UBK * 2;      // bytes of one stage's B tile
constexpr int kUStage = kUTileA + kUTileB;  // multiple of 1024
constexpr unsigned kUWaitLimit = 1u << 26;

// Shared-memory matrix descriptor of a K-major SWIZZLE_128B tile (rows of
// 128 bytes, 8-row atoms 1024 bytes apart): start address and stride byte
// offset in 16-byte units, descriptor version 1, layout type 2 (128B swizzle).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)(1) << 16;              // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;      // stride byte offset: next 8-row atom
    d |= (uint64_t)1 << 46;                // version
    d |= (uint64_t)2 << 61;                // SWIZZLE_128B
    return d;
}
// Instruction descriptor: D f32, A and B bf16, both K-major, M 128, N 256.
constexpr uint32_t kUIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(UBN >> 3) << 17) | ((uint32_t)(UBM >> 4) << 24);

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
// true once the barrier's phase with this parity has completed; bounded
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
    for (unsigned it = 0; it < kUWaitLimit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

template <int EPI>
__global__ void __launch_bounds__(kUThreads) gemm_tn_umma(const __nv_bfloat16* __restrict__ A,
                                                         const __nv_bfloat16* __restrict__ B, int K, int lda, int ldb,
                                                         EpiArgs e, int* err) {
    extern __shared__ __align__(1024) unsigned char usmem[];
    // 1024-byte aligned stage tiles: A0 B0 A1 B1, then barriers and the TMEM address
    unsigned char* base = (unsigned char*)(((uintptr_t)usmem + 1023) & ~(uintptr_t)1023);
    auto tA = [&](int st) { return base + st * kUStage; };
    auto tB = [&](int st) { return base + st * kUStage + kUTileA; };
    uint64_t* bar = (uint64_t*)(base + 2 * kUStage);
    uint32_t* taddr_s = (uint32_t*)(bar + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int bm = blockIdx.y * UBM, bn = blockIdx.x * UBN;
    const __nv_bfloat16* Ab = A + (size_t)bm * lda;
    const __nv_bfloat16* Bb = B + (size_t)bn * ldb;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(taddr_s)),
                     "r"(UBN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *taddr_s;

    auto load = [&](int stage, int k0) {
        // rows of 8 chunks of 16 bytes: A 128 rows (8 chunks per thread), B 256 rows (16)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int c = tid + i * kUThreads;
            const int row = c >> 3, ch = c & 7;
            cp_async16(tA(stage) + row * 128 + ((ch ^ (row & 7)) << 4), Ab + (size_t)row * lda + k0 + ch * 8);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int c = tid + i * kUThreads;
            const int row = c >> 3, ch = c & 7;
            cp_async16(tB(stage) + row * 128 + ((ch ^ (row & 7)) << 4), Bb + (size_t)row * ldb + k0 + ch * 8);
        }
        cp_commit();
    };

    const int nk = K / UBK;
    bool ok = true;
    load(0, 0);
    for (int kt = 0; kt < nk; ++kt) {
        const int st = kt & 1;
        if (kt + 1 < nk) {
            // stage st^1 was last read by the MMAs of tile kt-1
            if (kt >= 1) ok &= mbar_wait(&bar[st ^ 1], ((kt - 1) >> 1) & 1);
            load(st ^ 1, (kt + 1) * UBK);
            cp_wait<1>();
        } else {
            cp_wait<0>();
        }
        // make this thread's shared-memory writes visible to the tensor cores
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t sa = smem_u32(tA(st)), sb = smem_u32(tB(st));
#pragma unroll
            for (int k = 0; k < UBK / 16; ++k) {
                // k16 slice: 32 bytes further along the swizzled rows
                const uint64_t da = umma_desc_sw128(sa + k * 32), db = umma_desc_sw128(sb + k * 32);
                const uint32_t acc = (kt > 0 || k > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                    :
                    : "r"(tmem), "l"(da), "l"(db), "r"(kUIdesc), "r"(acc)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&bar[st]))
                         : "memory");
        }
    }
    // all MMAs are done once the last commit's barrier flips
    ok &= mbar_wait(&bar[(nk - 1) & 1], ((nk - 1) >> 1) & 1);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!ok) {
        if (lane == 0) atomicExch(err, 1);
    } else {
        // 32 columns at a time: lane l reads row 32w + l from tensor memory,
        // the warp transposes the 32 x 32 piece through shared memory (the
        // stage tiles are idle now) and writes it one row per instruction,
        // 32 consecutive columns, so that every store fills whole sectors
        float* stg = reinterpret_cast<float*>(base) + warp * 32 * 33;
#pragma unroll 1
        for (int cc = 0; cc < UBN; cc += 32) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t v[16];
                const uint32_t ta = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(cc + 16 * h);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                    "[%16];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                      "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                      "=r"(v[15])
                    : "r"(ta));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 16; ++j) stg[lane * 33 + 16 * h + j] = __uint_as_float(v[j]);
            }
            __syncwarp();
#pragma unroll 4
            for (int r = 0; r < 32; ++r) store1<EPI>(e, bm + warp * 32 + r, bn + cc + lane, stg[r * 33 + lane]);
            __syncwarp();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(UBN));
}

constexpr size_t kUSmem = 2 * kUStage + 1024 + 64;

// ---------------------------------------------------------------------------
// The tcgen05 contraction with its operands brought in by the tensor memory
// accelerator (TMA) and its roles split over warps.
//
// Same block (128 x 256, FP32 accumulator in 256 TMEM columns), same
// SWIZZLE_128B K-major tiles and MMAs as gemm_tn_umma, but:
//   * lane 0 of warp 0 issues one cp.async.bulk.tensor per operand tile
//     (tensor maps over this GPU's memory, no multicast) that completes on
//     the stage's "full" mbarrier with the byte count it expects;
//   * lane 0 of warp 1 waits on "full", issues the four k16 MMAs of the
//     stage and commits them to the stage's "empty" mbarrier, which the
//     producer waits on before refilling the stage: no __syncthreads and no
//     thread-issued copies in the main loop;
//   * kTStages stages ring through shared memory;
//   * after the last commit every warp reads its 32 accumulator rows and
//     stores them as gemm_tn_umma does.
// Every wait is bounded; one that gives up sets *err and the kernel finishes
// without the result.
// ---------------------------------------------------------------------------
constexpr int kTStages = 2;  // 2 x 48 KB: two CTAs share an SM (and its 512 TMEM columns)
constexpr size_t kTSmem = (size_t)kTStages * kUStage + 1024 + 256;

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

template <int EPI>
__global__ void __launch_bounds__(kUThreads) gemm_tn_tma(const __grid_constant__ CUtensorMap mapA,
                                                        const __grid_constant__ CUtensorMap mapB, int K, EpiArgs e,
                                                        int* err) {
    extern __shared__ __align__(1024) unsigned char usmem[];
    unsigned char* base = (unsigned char*)(((uintptr_t)usmem + 1023) & ~(uintptr_t)1023);
    auto tA = [&](int st) { return base + st * kUStage; };
    auto tB = [&](int st) { return base + st * kUStage + kUTileA; };
    uint64_t* full = (uint64_t*)(base + kTStages * kUStage);
    uint64_t* empty = full + kTStages;
    uint64_t* done = empty + kTStages;
    uint32_t* taddr_s = (uint32_t*)(done + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int bm = blockIdx.y * UBM, bn = blockIdx.x * UBN;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(taddr_s)),
                     "r"(UBN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 32) {
        for (int s = 0; s < kTStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *taddr_s;
    const int nk = K / UBK;
    bool ok = true;

    int issued = 0;  // producer: tiles whose loads were issued
    if (warp == 0 && lane == 0) {
        // producer: stage st is refilled once the MMAs that read it have completed
        for (int kt = 0; kt < nk && ok; ++kt) {
            const int st = kt % kTStages;
            if (kt >= kTStages) ok &= mbar_wait(&empty[st], ((kt / kTStages) - 1) & 1);
            if (!ok) break;
            mbar_expect_tx(&full[st], (unsigned)kUStage);
            tma_load_2d(tA(st), &mapA, kt * UBK, bm, &full[st]);
            tma_load_2d(tB(st), &mapB, kt * UBK, bn, &full[st]);
            issued = kt + 1;
        }
    } else if (warp == 1 && lane == 0) {
        // MMA issuer
        for (int kt = 0; kt < nk && ok; ++kt) {
            const int st = kt % kTStages;
            ok &= mbar_wait(&full[st], (kt / kTStages) & 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t sa = smem_u32(tA(st)), sb = smem_u32(tB(st));
#pragma unroll
            for (int k = 0; k < UBK / 16; ++k) {
                const uint64_t da = umma_desc_sw128(sa + k * 32), db = umma_desc_sw128(sb + k * 32);
                const uint32_t acc = (kt > 0 || k > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                    :
                    : "r"(tmem), "l"(da), "l"(db), "r"(kUIdesc), "r"(acc)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&empty[st]))
                         : "memory");
        }
        // the accumulator is complete once every MMA issued so far is
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(done))
                     : "memory");
    }
    __syncwarp();
    // every thread: wait for the accumulator (bounded), then the epilogue
    ok &= mbar_wait(done, 0);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // a role thread that gave up is seen by the whole CTA
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    if (!ok && warp == 0 && lane == 0) {
        // no copy may still be writing this CTA's shared memory when it exits:
        // wait (bounded) for the last load issued into each stage
        for (int kt = issued - 1; kt >= 0 && kt >= issued - kTStages; --kt)
            mbar_wait(&full[kt % kTStages], (kt / kTStages) & 1);
    }
    if (!ok) {
        if (tid == 0) atomicExch(err, 1);
    } else {
        float* stg = reinterpret_cast<float*>(base) + warp * 32 * 33;  // the stage tiles are idle now
#pragma unroll 1
        for (int cc = 0; cc < UBN; cc += 32) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t v[16];
                const uint32_t ta = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(cc + 16 * h);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                    "[%16];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                      "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                      "=r"(v[15])
                    : "r"(ta));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 16; ++j) stg[lane * 33 + 16 * h + j] = __uint_as_float(v[j]);
            }
            __syncwarp();
#pragma unroll 4
            for (int r = 0; r < 32; ++r) store1<EPI>(e, bm + warp * 32 + r, bn + cc + lane, stg[r * 33 + lane]);
            __syncwarp();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(UBN));
}

// ---------------------------------------------------------------------------
// The default: gemm_tn_tma's loads and MMAs on blocks of 128 x BN, and an
// epilogue that leaves by the tensor memory accelerator too.
//
// The surrogate's contractions range from 512 x 512 to 8192 x 8192.  A block
// of 256 columns leaves a 512 x 512 product to 8 CTAs that each write 128 KB;
// blocks of 64 columns spread it over 32, with eight stages in flight (22 ->
// 9 us at K = 512).  The epilogue takes 32 (f32) or 64 (bf16) columns of a
// warp's 32 rows at a time from tensor memory, applies bias, ReLU or mask in
// registers, writes them to shared memory in the swizzle of the output's
// tensor map (conflict-free 16-byte stores, a row per lane) and stores the
// piece with one bulk copy while the next is prepared; the mask block came in
// by bulk copies during the main loop.  Element by element the sums over K are
// the MMAs' own, in the same order for every BN.
// ---------------------------------------------------------------------------
template <int EPI>
constexpr bool epi_bf16() { return EPI == CR_MLP_EPI_BIAS_RELU_BF16 || EPI == CR_MLP_EPI_RELU_MASK_BF16; }
template <int EPI, int BN, int ST>
struct TileGemm {
    static constexpr int kStage = kUTileA + BN * UBK * 2;
    static constexpr int kMask = EPI == CR_MLP_EPI_RELU_MASK_BF16 ? UBM * BN * 2 : 0;
    static constexpr size_t smem = (size_t)ST * kStage + kMask + BN * sizeof(float) + 1024 + 256;
    static_assert(ST * kStage >= 4 * 8192, "the output pieces reuse the stages");
};

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y, const void* src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(smem_u32(src))
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// 32 consecutive columns of this lane's row of the accumulator
__device__ __forceinline__ void tmem_ld32(uint32_t addr, float* v) {
    uint32_t u[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
        "%29,%30,%31}, [%32];"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
          "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]), "=r"(u[16]),
          "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]), "=r"(u[24]),
          "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(u[j]);
}

// Roles run by whole warps, with one elected lane at the instructions that one
// thread issues: a loop that only lane 0 entered kept addresses and descriptors in
// per-thread registers, and moving them over for every MMA and copy took longer than
// a narrow MMA itself (512 x 512 x 8192 with mask 44 -> 28 us, ensemble_tile 264 ->
// 207, 512 x 512 x 512 7.3 -> 6.4).
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0); }
__device__ __forceinline__ bool elect_lane() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
// The whole warp waits, and goes on or gives up together.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, unsigned parity) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity)) != 0;
}

// The MMAs of one stage (128 rows x 64 of A, the idesc's columns x 64 of B), by one thread.
__device__ __forceinline__ void mma_stage(uint32_t acc, uint32_t sa, uint32_t sb, uint32_t idesc, bool first) {
    const uint64_t da0 = umma_desc_sw128(sa), db0 = umma_desc_sw128(sb);
#pragma unroll
    for (int k = 0; k < UBK / 16; ++k) {
        const uint64_t da = da0 + 2 * k, db = db0 + 2 * k;  // 32 bytes on, in units of 16
        const uint32_t accum = (!first || k > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            :
            : "r"(acc), "l"(da), "l"(db), "r"(idesc), "r"(accum)
            : "memory");
    }
}
// The barrier completes once every MMA issued so far has.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// The tensor maps and bias of up to G contractions of one shape.
constexpr int kMaxGroup = 4;
template <int G>
struct TileMaps {
    CUtensorMap a[G], b[G], o[G], m[1];  // m: the mask, of single contractions
    const float* bias[G];
};
// 32 accumulator columns (of this lane's row) through bias (32 values in shared
// memory), ReLU or mask (the row's 64-byte half h of a swizzled block), into
// the lane's words of the output: 32 of f32, 16 of bf16.
template <int EPI>
__device__ __forceinline__ void epi_columns(uint32_t acc, const float* sbias, const unsigned char* mask_row, int row,
                                            int h, uint32_t* w) {
    float v[32];
    tmem_ld32(acc, v);
    if (EPI == CR_MLP_EPI_BIAS_RELU_BF16 || EPI == CR_MLP_EPI_BIAS_F32) {
        const float4* b4 = reinterpret_cast<const float4*>(sbias);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float4 b = b4[j];
            v[4 * j] += b.x;
            v[4 * j + 1] += b.y;
            v[4 * j + 2] += b.z;
            v[4 * j + 3] += b.w;
        }
    }
    if (EPI == CR_MLP_EPI_BIAS_RELU_BF16) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.f);
    }
    if (EPI == CR_MLP_EPI_RELU_MASK_BF16) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint4 m = *reinterpret_cast<const uint4*>(mask_row + (((4 * h + j) ^ (row & 7)) << 4));
            const uint32_t mm[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&mm[q]));
                v[8 * j + 2 * q] = f.x > 0.f ? v[8 * j + 2 * q] : 0.f;
                v[8 * j + 2 * q + 1] = f.y > 0.f ? v[8 * j + 2 * q + 1] : 0.f;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        if (!epi_bf16<EPI>()) {
            w[j] = __float_as_uint(v[j]);
        } else if ((j & 1) == 0) {
            const __nv_bfloat162 p = __floats2bfloat162_rn(v[j], v[j + 1]);
            w[j / 2] = *reinterpret_cast<const uint32_t*>(&p);
        }
    }
}
// A lane's 128 bytes into its row of a 32-row piece, in the output map's swizzle.
__device__ __forceinline__ void put_row(unsigned char* piece, int lane, const uint32_t (&w)[32]) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
        *reinterpret_cast<uint4*>(piece + lane * 128 + ((j ^ (lane & 7)) << 4)) =
            make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
}

// 32 bytes of a lane: a whole sector of its row.
__device__ __forceinline__ void store_sector(void* p, const uint32_t* w) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                 "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}

// Kernels launched by launch_next start beside the end of the one before: what a
// CTA sets up for itself - tensor memory, barriers - overlaps it (shared memory admits
// two CTAs of gemm_tn_tile on an SM, or one of any other tcgen05 kernel that waits here, so
// its 512 columns never run short).  Nothing of global
// memory is read or written before this returns, which is when that kernel has
// completed; the next launch may then start in the same way.  (Not for kernels whose
// inputs are const __restrict__: such loads may be moved above the wait.)  A training step of 512
// (17 launches) 185 -> 158 us, 4000 requests 322 -> 312.
__device__ __forceinline__ void launch_order() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <int EPI, int BN, int ST, int G>
__global__ void __launch_bounds__(kUThreads) gemm_tn_tile(const __grid_constant__ TileMaps<G> t, int K, int* err) {
    const int group = G > 1 ? blockIdx.z : 0;
    const CUtensorMap &mapA = t.a[group], &mapB = t.b[group], &mapO = t.o[group], &mapM = t.m[0];
    const float* bias = t.bias[group];
    using T = TileGemm<EPI, BN, ST>;
    constexpr bool kMasked = EPI == CR_MLP_EPI_RELU_MASK_BF16;
    constexpr bool kBias = EPI == CR_MLP_EPI_BIAS_RELU_BF16 || EPI == CR_MLP_EPI_BIAS_F32;
    constexpr uint32_t idesc =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(UBM >> 4) << 24);
    extern __shared__ __align__(1024) unsigned char usmem[];
    unsigned char* base = (unsigned char*)(((uintptr_t)usmem + 1023) & ~(uintptr_t)1023);
    auto tA = [&](int st) { return base + st * T::kStage; };
    auto tB = [&](int st) { return base + st * T::kStage + kUTileA; };
    unsigned char* masks = base + ST * T::kStage;  // [BN / 64] blocks of 128 rows x 64 columns
    float* sbias = (float*)(masks + T::kMask);  // the block's bias values
    uint64_t* full = (uint64_t*)(sbias + BN);
    uint64_t* empty = full + ST;
    uint64_t* done = empty + ST;
    uint64_t* mask_bar = done + 1;
    uint32_t* taddr_s = (uint32_t*)(mask_bar + 1);
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int bm = blockIdx.y * UBM, bn = blockIdx.x * BN;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(taddr_s)),
                     "r"(BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 32) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        mbar_init(mask_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    launch_order();
    if (kBias)
        for (int c = tid; c < BN; c += kUThreads) sbias[c] = bias[bn + c];
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *taddr_s;
    const int nk = K / UBK;
    bool ok = true;

    int issued = 0;  // producer: tiles whose loads were issued
    if (warp == 0) {
        for (int kt = 0; kt < nk && ok; ++kt) {
            const int st = kt % ST;
            if (kt >= ST) ok = warp_wait(&empty[st], ((kt / ST) - 1) & 1);
            if (!ok) break;
            if (elect_lane()) {
                mbar_expect_tx(&full[st], (unsigned)T::kStage);
                tma_load_2d(tA(st), &mapA, kt * UBK, bm, &full[st]);
                tma_load_2d(tB(st), &mapB, kt * UBK, bn, &full[st]);
                if (kMasked && kt == 0) {
                    mbar_expect_tx(mask_bar, (unsigned)T::kMask);
#pragma unroll 1
                    for (int c = 0; c < BN / 64; ++c)
                        tma_load_2d(masks + c * UBM * 128, &mapM, bn + 64 * c, bm, mask_bar);
                }
            }
            __syncwarp();
            issued = kt + 1;
        }
    } else if (warp == 1) {
        for (int kt = 0; kt < nk && ok; ++kt) {
            const int st = kt % ST;
            ok = warp_wait(&full[st], (kt / ST) & 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_lane()) {
                mma_stage(tmem, smem_u32(tA(st)), smem_u32(tB(st)), idesc, kt == 0);
                mma_commit(&empty[st]);
            }
            __syncwarp();
        }
        // the accumulator is complete once every MMA issued so far is
        if (elect_lane()) mma_commit(done);
    }
    __syncwarp();
    ok &= mbar_wait(done, 0);
    if (kMasked) ok &= mbar_wait(mask_bar, 0);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // a role thread that gave up is seen by the whole CTA
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    if (!ok && warp == 0 && lane == 0) {
        // no copy may still be writing this CTA's shared memory when it exits:
        // wait (bounded) for the last load issued into each stage
        for (int kt = issued - 1; kt >= 0 && kt >= issued - ST; --kt) mbar_wait(&full[kt % ST], (kt / ST) & 1);
        if (kMasked && issued > 0) mbar_wait(mask_bar, 0);
    }
    if (!ok) {
        if (tid == 0) atomicExch(err, 1);
    } else {
        constexpr int kCols = epi_bf16<EPI>() ? 64 : 32;  // columns of a piece: 128 bytes a row
        unsigned char* stg = base + warp * 8192;           // two pieces of 4 KB; the stages are idle now
        const uint32_t acc = tmem + ((uint32_t)(warp * 32) << 16);
        const int row = warp * 32 + lane;
#pragma unroll 1
        for (int c = 0; c < BN / kCols; ++c) {
            uint32_t w[32];  // the lane's 128 bytes
#pragma unroll
            for (int h = 0; h < kCols / 32; ++h)
                epi_columns<EPI>(acc + (uint32_t)(c * kCols + 32 * h), sbias + c * kCols + 32 * h,
                                 masks + c * UBM * 128 + row * 128, row, h, w + 16 * h);
            unsigned char* piece = stg + (c & 1) * 4096;
            if (c >= 2) {  // the copy that read this piece two turns ago is done with it
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                __syncwarp();
            }
            put_row(piece, lane, w);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) tma_store_2d(&mapO, bn + c * kCols, bm + warp * 32, piece);
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN));
}

// dst[c][r] = src[r][c] for a rows x cols BF16 matrix (32 x 32 tiles).
__global__ void transpose_bf16(const __nv_bfloat16* __restrict__ src, int lds, __nv_bfloat16* __restrict__ dst,
                               int ldd, int rows, int cols) {
    __shared__ __nv_bfloat16 t[32][33];
    const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int r = r0 + i, c = c0 + threadIdx.x;
        if (r < rows && c < cols) t[i][threadIdx.x] = src[(size_t)r * lds + c];
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int c = c0 + i, r = r0 + threadIdx.x;
        if (r < rows && c < cols) dst[(size_t)c * ldd + r] = t[threadIdx.x][i];
    }
}

// Several matrices of one launch (the layers of a network).
constexpr int kMaxMats = 32;
struct Mats {
    int n;
    int first[kMaxMats + 1];  // first block of each matrix
    const __nv_bfloat16* src[kMaxMats];
    void* dst[kMaxMats];
    int lds[kMaxMats], ldd[kMaxMats], rows[kMaxMats], cols[kMaxMats];
};
__device__ __forceinline__ int mat_of(const Mats& t, int block) {
    int i = 0;
    while (block >= t.first[i + 1]) ++i;
    return i;
}

// Place of (c, r) in row c of a transposed 64 x 64 tile: the 16-byte pieces of a row
// are permuted by the row's eighth, or the lanes of a warp, eight columns apart,
// would write one bank (with the column sums' eight loads in flight, a training step
// of 512: 158 -> 153 us).
__device__ __forceinline__ int tile_place(int c, int r) { return (((r >> 3) ^ (c >> 3)) & 7) * 8 + (r & 7); }

// A transposed tile; its rows are read and written 16 bytes at a time.
struct __align__(16) Tile64 {
    __nv_bfloat16 v[64][72];
};
static_assert(alignof(Tile64) >= 16 && sizeof(Tile64) % (64 * 16) == 0, "rows on 16-byte boundaries");

// dst[c][r] = src[r][c] in 64 x 64 tiles: 16-byte rows in and out (columns and
// rows multiples of 64, bases and strides 16-byte aligned).  All layers of a
// training step in one launch, instead of twelve of 3.5-11 us.
__global__ void __launch_bounds__(256) transpose_mats(const __grid_constant__ Mats t) {
    __shared__ Tile64 tile;
    const int i = mat_of(t, blockIdx.x), b = blockIdx.x - t.first[i], nc = t.cols[i] / 64;
    const int r0 = (b / nc) * 64, c0 = (b % nc) * 64;
    const __nv_bfloat16* src = t.src[i];
    launch_order();
    __nv_bfloat16* dst = (__nv_bfloat16*)t.dst[i];
    for (int q = threadIdx.x; q < 512; q += 256) {
        const int r = q >> 3, c = (q & 7) * 8;
        const uint4 v = *reinterpret_cast<const uint4*>(src + (size_t)(r0 + r) * t.lds[i] + c0 + c);
        const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&v);
#pragma unroll
        for (int j = 0; j < 8; ++j) tile.v[c + j][tile_place(c, r)] = e[j];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 512; q += 256) {
        const int c = q >> 3, r = (q & 7) * 8;
        *reinterpret_cast<uint4*>(dst + (size_t)(c0 + c) * t.ldd[i] + r0 + r) =
            *reinterpret_cast<const uint4*>(&tile.v[c][tile_place(c, r)]);
    }
}

// out[c] = sum_r src[r][c] (bias gradients): a block takes 64 columns, 32 of
// its rows of threads every 32nd row, folded in a fixed order.  One thread a
// column waited for 512 loads in turn (32-37 us a layer).
__global__ void __launch_bounds__(1024) col_sum_mats(const __grid_constant__ Mats t) {
    __shared__ float2 part[32][33];
    launch_order();
    const int i = mat_of(t, blockIdx.x), c = (blockIdx.x - t.first[i]) * 64 + 2 * threadIdx.x;
    const __nv_bfloat16* src = t.src[i];
    const bool pair = c + 1 < t.cols[i] && (((uintptr_t)src & 3) == 0) && t.lds[i] % 2 == 0;
    float2 s = make_float2(0.f, 0.f);
    const int rows = t.rows[i], ld = t.lds[i];
    if (pair) {
#pragma unroll 8
        for (int r = threadIdx.y; r < rows; r += 32) {
            const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(src + (size_t)r * ld + c));
            s.x += v.x;
            s.y += v.y;
        }
    } else {
        for (int r = threadIdx.y; r < rows; r += 32) {
            const __nv_bfloat16* q = src + (size_t)r * ld + c;
            if (c < t.cols[i]) s.x += __bfloat162float(q[0]);
            if (c + 1 < t.cols[i]) s.y += __bfloat162float(q[1]);
        }
    }
    part[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    for (int d = 16; d > 0; d >>= 1) {
        if ((int)threadIdx.y < d) {
            const float2 o = part[threadIdx.y + d][threadIdx.x];
            part[threadIdx.y][threadIdx.x].x += o.x;
            part[threadIdx.y][threadIdx.x].y += o.y;
        }
        __syncthreads();
    }
    if (threadIdx.y == 0) {
        float* out = (float*)t.dst[i];
        if (c < t.cols[i]) out[c] = part[0][threadIdx.x].x;
        if (c + 1 < t.cols[i]) out[c + 1] = part[0][threadIdx.x].y;
    }
}

// Masked mean squared error: grad = 2 (pred - y) / n_valid where valid,
// and the sum of squared errors accumulated into *sse.
__device__ __forceinline__ float mse_one(float pred, float y, bool valid, float inv_count, double& acc) {
    if (!valid) return 0.f;
    const float d = pred - y;
    acc += (double)d * d;
    return 2.f * d * inv_count;
}
// VEC: four entries a thread at a time (n a multiple of 4, aligned arrays).
template <bool VEC>
__global__ void mse_grad(const float* __restrict__ pred, const __nv_bfloat16* __restrict__ y,
                         const unsigned char* __restrict__ valid, long long n, float inv_count,
                         __nv_bfloat16* __restrict__ grad, double* __restrict__ sse) {
    __shared__ double red[256];
    double acc = 0.0;
    const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
    if (VEC) {
        for (long long i = first; i < n / 4; i += stride) {
            const float4 p = reinterpret_cast<const float4*>(pred)[i];
            const uint2 yb = reinterpret_cast<const uint2*>(y)[i];
            const uchar4 ok = reinterpret_cast<const uchar4*>(valid)[i];
            const float2 y0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&yb.x)),
                         y1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&yb.y));
            const float g0 = mse_one(p.x, y0.x, ok.x, inv_count, acc), g1 = mse_one(p.y, y0.y, ok.y, inv_count, acc),
                        g2 = mse_one(p.z, y1.x, ok.z, inv_count, acc), g3 = mse_one(p.w, y1.y, ok.w, inv_count, acc);
            const __nv_bfloat162 a = __floats2bfloat162_rn(g0, g1), b = __floats2bfloat162_rn(g2, g3);
            reinterpret_cast<uint2*>(grad)[i] =
                make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        }
    } else {
        for (long long i = first; i < n; i += stride)
            grad[i] = __float2bfloat16_rn(mse_one(pred[i], __bfloat162float(y[i]), valid[i], inv_count, acc));
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(sse, red[0]);
}

// Adam on FP32 master parameters; writes the BF16 copy used by the GEMMs.
struct AdamArgs {
    float lr, b1, b2, eps, c1, c2;
};
__device__ __forceinline__ float adam_one(float p, float g, float& m, float& v, const AdamArgs& a, float wd) {
    const float gi = g + wd * p;
    m = a.b1 * m + (1.f - a.b1) * gi;
    v = a.b2 * v + (1.f - a.b2) * gi * gi;
    return p - a.lr * (m * a.c1) / (sqrtf(v * a.c2) + a.eps);
}
__global__ void adam_step(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                          float* __restrict__ v, __nv_bfloat16* __restrict__ pb, long long n, AdamArgs a, float wd) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float mi = m[i], vi = v[i];
        const float pi = adam_one(p[i], g[i], mi, vi, a, wd);
        m[i] = mi;
        v[i] = vi;
        p[i] = pi;
        if (pb) pb[i] = __float2bfloat16_rn(pi);
    }
}

// The same over every layer's weights and biases in one launch, writing the
// weights' BF16 copy and its transpose too (64 x 64 tiles): bound by the 32
// bytes a parameter that it moves.  Eight Adam launches and four transposes
// read the weights twice.
struct AdamMats {
    int n;
    int first[kMaxMats + 1];  // first block: weights in 64 x 64 tiles, biases in runs of 4096
    float* p[kMaxMats];
    const float* g[kMaxMats];
    float *m[kMaxMats], *v[kMaxMats];
    __nv_bfloat16 *pb[kMaxMats], *pt[kMaxMats];  // NULL: a bias
    int rows[kMaxMats], cols[kMaxMats];
};
__global__ void __launch_bounds__(256) adam_mats(const __grid_constant__ AdamMats t, AdamArgs a, float wd) {
    launch_order();
    __shared__ Tile64 tile;
    int i = 0;
    while ((int)blockIdx.x >= t.first[i + 1]) ++i;
    const int b = blockIdx.x - t.first[i];
    if (!t.pb[i]) {
        const int n = t.rows[i];
        for (int q = b * 4096 + threadIdx.x; q < min(n, (b + 1) * 4096); q += 256) {
            float m = t.m[i][q], v = t.v[i][q];
            t.p[i][q] = adam_one(t.p[i][q], t.g[i][q], m, v, a, 0.f);
            t.m[i][q] = m;
            t.v[i][q] = v;
        }
        return;
    }
    const int nc = t.cols[i] / 64, r0 = (b / nc) * 64, c0 = (b % nc) * 64;
#pragma unroll 2
    for (int q = threadIdx.x; q < 1024; q += 256) {
        const int r = q >> 4, c = (q & 15) * 4;
        const size_t o = (size_t)(r0 + r) * t.cols[i] + c0 + c;
        float4 p = *reinterpret_cast<const float4*>(t.p[i] + o), m = *reinterpret_cast<const float4*>(t.m[i] + o),
               v = *reinterpret_cast<const float4*>(t.v[i] + o);
        const float4 g = *reinterpret_cast<const float4*>(t.g[i] + o);
        p.x = adam_one(p.x, g.x, m.x, v.x, a, wd);
        p.y = adam_one(p.y, g.y, m.y, v.y, a, wd);
        p.z = adam_one(p.z, g.z, m.z, v.z, a, wd);
        p.w = adam_one(p.w, g.w, m.w, v.w, a, wd);
        *reinterpret_cast<float4*>(t.p[i] + o) = p;
        *reinterpret_cast<float4*>(t.m[i] + o) = m;
        *reinterpret_cast<float4*>(t.v[i] + o) = v;
        __nv_bfloat162 w[2] = {__floats2bfloat162_rn(p.x, p.y), __floats2bfloat162_rn(p.z, p.w)};
        *reinterpret_cast<uint2*>(t.pb[i] + o) = *reinterpret_cast<const uint2*>(w);
        const int at = tile_place(c, r);
        tile.v[c][at] = w[0].x;
        tile.v[c + 1][at] = w[0].y;
        tile.v[c + 2][at] = w[1].x;
        tile.v[c + 3][at] = w[1].y;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 512; q += 256) {
        const int c = q >> 3, r = (q & 7) * 8;
        *reinterpret_cast<uint4*>(t.pt[i] + (size_t)(c0 + c) * t.rows[i] + r0 + r) =
            *reinterpret_cast<const uint4*>(&tile.v[c][tile_place(c, r)]);
    }
}

// Mean and standard deviation (over the members) of the ensemble's outputs,
// each scaled, shifted and clamped: one pass over the members' outputs
// instead of a stack, three elementwise passes and two reductions over it.
constexpr int kMaxMembers = 64;
struct Members {
    const float* out[kMaxMembers];
};
__device__ __forceinline__ float member_tl(float x, float scale, float mid, float lo, float hi) {
    float t = __fadd_rn(__fmul_rn(x, scale), mid);
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(t) : "f"(lo));  // a NaN stays
    asm("min.NaN.f32 %0, %0, %1;" : "+f"(t) : "f"(hi));
    return t;
}
template <int M>  // members held in registers; 0: any number, read twice
__global__ void __launch_bounds__(256) ensemble_stats(const __grid_constant__ Members p, int members, long long n4,
                                                      float scale, float mid, float lo, float hi,
                                                      float4* __restrict__ mean, float4* __restrict__ spread) {
    const float inv = 1.f / (float)members;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
        auto get = [&](int k) {
            float4 x = __ldcs(reinterpret_cast<const float4*>(p.out[k]) + i);
            x.x = member_tl(x.x, scale, mid, lo, hi);
            x.y = member_tl(x.y, scale, mid, lo, hi);
            x.z = member_tl(x.z, scale, mid, lo, hi);
            x.w = member_tl(x.w, scale, mid, lo, hi);
            return x;
        };
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f), q = s, x[M > 0 ? M : 1];
        auto add = [&](const float4& v) {
            s.x += v.x;
            s.y += v.y;
            s.z += v.z;
            s.w += v.w;
        };
        auto dev = [&](const float4& v) {
            q.x = fmaf(v.x - s.x, v.x - s.x, q.x);
            q.y = fmaf(v.y - s.y, v.y - s.y, q.y);
            q.z = fmaf(v.z - s.z, v.z - s.z, q.z);
            q.w = fmaf(v.w - s.w, v.w - s.w, q.w);
        };
        if (M > 0) {
#pragma unroll
            for (int k = 0; k < M; ++k) x[k] = get(k);
#pragma unroll
            for (int k = 0; k < M; ++k) add(x[k]);
        } else {
            for (int k = 0; k < members; ++k) add(get(k));
        }
        s = make_float4(s.x * inv, s.y * inv, s.z * inv, s.w * inv);
        if (M > 0) {
#pragma unroll
            for (int k = 0; k < M; ++k) dev(x[k]);
        } else {
            for (int k = 0; k < members; ++k) dev(get(k));
        }
        mean[i] = s;
        spread[i] = make_float4(sqrtf(q.x * inv), sqrtf(q.y * inv), sqrtf(q.z * inv), sqrtf(q.w * inv));
    }
}

__global__ void to_bf16(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = __float2bfloat16_rn(src[i]);
}

int grid_for(long long n) {
    long long b = (n + 255) / 256;
    return (int)(b < 4096 ? (b < 1 ? 1 : b) : 4096);
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// How cr_mlp_gemm_tc feeds its kernels: 1, the default, by the tensor memory
// accelerator (launch_tile_n chooses among gemm_tn_tile's blocks and
// gemm_tn_persistent; gemm_tn_tma for rows off 16-byte boundaries);
// CUPYRAM_B200_GEMM=persistent: gemm_tn_persistent at any size, =cp: gemm_tn_umma,
// fed by cp.async.
int gemm_feed() {
    const char* v = getenv("CUPYRAM_B200_GEMM");
    if (v && v[0] == 'c') return 0;
    if (v && v[0] == 'p') return 2;
    return 1;
}

// ---------------------------------------------------------------------------
// Persistent contraction with the epilogue overlapped, for outputs of at least
// two blocks an SM.
//
// One CTA per SM walks the output blocks (128 x 256) in a static round
// robin.  Six warps:
//   * warp 0: TMA producer over a kPStages-deep ring of stages (one elected lane
//     issues, as in gemm_tn_tile);
//   * warp 1: MMA issuer, accumulating block i in one of two TMEM
//     accumulators (columns 0..255 or 256..511, by i's parity), committing
//     each stage to its "empty" barrier and each finished block to its
//     accumulator's "full" barrier;
//   * warps 2..5: the epilogue, one TMEM lane quadrant each (quadrant =
//     warp mod 4): gemm_tn_tile's pieces and bulk stores of block i, while the
//     MMAs of block i + 1 run in the other accumulator.  Reading the last
//     columns releases the accumulator on its "empty" barrier.
// Every wait is bounded; a role that gives up stops, the CTA sets *err, and
// the output is incomplete.
//
// 8192 x 8192 x 512 into f32: 79 us (blocks of 256 columns by gemm_tn_tile, two
// CTAs of two stages on an SM: 91).  Without its stores it takes 50 us (38 the
// loads alone), with a K of 64 its 268 MB take 54 (a fill: 39); the two share the
// shared memory's bandwidth.  Eight epilogue warps (79 us), 32-byte stores straight
// from registers (88) and other walks over the blocks (80-81) gained nothing.
// ---------------------------------------------------------------------------
constexpr int kPStages = 4;
constexpr int kPThreads = 192;
constexpr size_t kPSmem = (size_t)kPStages * kUStage + 4 * 8192 + 4 * 64 * sizeof(float) + 1024 + 256;
static_assert(kPSmem <= 227 * 1024, "one CTA's shared memory");

template <int EPI>
__global__ void __launch_bounds__(kPThreads, 1)
    gemm_tn_persistent(const __grid_constant__ TileMaps<1> t, int M, int N, int K, int* err) {
    constexpr bool kBias = EPI == CR_MLP_EPI_BIAS_RELU_BF16 || EPI == CR_MLP_EPI_BIAS_F32;
    extern __shared__ __align__(1024) unsigned char usmem[];
    unsigned char* base = (unsigned char*)(((uintptr_t)usmem + 1023) & ~(uintptr_t)1023);
    auto tA = [&](int st) { return base + st * kUStage; };
    auto tB = [&](int st) { return base + st * kUStage + kUTileA; };
    unsigned char* stg_all = base + kPStages * kUStage;
    float* sbias_all = (float*)(stg_all + 4 * 8192);
    uint64_t* full = (uint64_t*)(sbias_all + 4 * 64);
    uint64_t* empty = full + kPStages;
    uint64_t* acc_full = empty + kPStages;   // [2]
    uint64_t* acc_empty = acc_full + 2;      // [2]
    uint32_t* taddr_s = (uint32_t*)(acc_empty + 2);
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int nk = K / UBK, nbm = M / UBM, nbn = N / UBN, nblocks = nbm * nbn;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(taddr_s)),
                     "r"(2 * UBN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 32) {
        for (int s = 0; s < kPStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 4);  // one arrival per epilogue warp
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    launch_order();
    const uint32_t tmem = *taddr_s;
    bool ok = true;
    int issued = 0;  // producer: k-tiles whose loads were issued (over all blocks)

    if (warp == 0) {
        int g = 0;
        for (int blk = blockIdx.x; blk < nblocks && ok; blk += gridDim.x) {
            const int bm = (blk % nbm) * UBM, bn = (blk / nbm) * UBN;
            for (int kt = 0; kt < nk && ok; ++kt, ++g) {
                const int st = g % kPStages;
                if (g >= kPStages) ok = warp_wait(&empty[st], ((g / kPStages) - 1) & 1);
                if (!ok) break;
                if (elect_lane()) {
                    mbar_expect_tx(&full[st], (unsigned)kUStage);
                    tma_load_2d(tA(st), &t.a[0], kt * UBK, bm, &full[st]);
                    tma_load_2d(tB(st), &t.b[0], kt * UBK, bn, &full[st]);
                }
                __syncwarp();
                issued = g + 1;
            }
        }
    } else if (warp == 1) {
        int g = 0, i = 0;
        for (int blk = blockIdx.x; blk < nblocks && ok; blk += gridDim.x, ++i) {
            const int a = i & 1;
            // the epilogue has drained this accumulator's previous block
            if (i >= 2) ok = warp_wait(&acc_empty[a], ((i / 2) - 1) & 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc_addr = tmem + (uint32_t)(a * UBN);
            for (int kt = 0; kt < nk && ok; ++kt, ++g) {
                const int st = g % kPStages;
                ok = warp_wait(&full[st], (g / kPStages) & 1);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_lane()) {
                    mma_stage(acc_addr, smem_u32(tA(st)), smem_u32(tB(st)), kUIdesc, kt == 0);
                    mma_commit(&empty[st]);
                }
                __syncwarp();
            }
            if (!ok) break;
            if (elect_lane()) mma_commit(&acc_full[a]);
            __syncwarp();
        }
    } else {
        // epilogue: TMEM lane quadrant q = warp mod 4 holds rows 32q..32q+31
        constexpr int kCols = epi_bf16<EPI>() ? 64 : 32;  // columns of a piece: 128 bytes a row
        const int q = warp & 3;
        unsigned char* stg = stg_all + (warp - 2) * 8192;  // two pieces of 4 KB
        float* sbias = sbias_all + (warp - 2) * 64;
        int i = 0, n = 0;  // blocks, pieces
        for (int blk = blockIdx.x; blk < nblocks && ok; blk += gridDim.x, ++i) {
            const int a = i & 1;
            const int bm = (blk % nbm) * UBM, bn = (blk / nbm) * UBN;
            ok &= mbar_wait(&acc_full[a], (i / 2) & 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * UBN);
#pragma unroll 1
            for (int c = 0; c < UBN / kCols; ++c, ++n) {
                if (kBias) {
                    __syncwarp();
                    for (int j = lane; j < kCols; j += 32) sbias[j] = t.bias[0][bn + c * kCols + j];
                    __syncwarp();
                }
                uint32_t w[32];  // the lane's 128 bytes
#pragma unroll
                for (int h = 0; h < kCols / 32; ++h)
                    epi_columns<EPI>(acc + (uint32_t)(c * kCols + 32 * h), sbias + 32 * h, nullptr, lane, h, w + 16 * h);
                if (c == UBN / kCols - 1) {
                    // this warp's reads of the accumulator are done: release it to the MMAs
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0)
                        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[a])) : "memory");
                }
                unsigned char* piece = stg + (n & 1) * 4096;
                if (n >= 2) {  // the copy that read this piece two turns ago is done with it
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    __syncwarp();
                }
                put_row(piece, lane, w);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) tma_store_2d(&t.o[0], bn + c * kCols, bm + q * 32, piece);
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    __syncwarp();
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    if (!ok && warp == 0 && lane == 0) {
        // no copy may still be writing this CTA's shared memory when it exits
        for (int g = issued - 1; g >= 0 && g >= issued - kPStages; --g)
            mbar_wait(&full[g % kPStages], (g / kPStages) & 1);
    }
    if (!ok && tid == 0) atomicExch(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * UBN));
}

// ---------------------------------------------------------------------------
// Output layers of an ensemble with the statistics in the epilogue.
//
// Each member's outputs were written (134 MB for 4096 requests), read again by
// ensemble_stats and thrown away: 4 x 54 us of contractions and 127 us of
// statistics for 4000 requests and four members.  Here a CTA accumulates the
// same 128 x 128 block of every member side by side in tensor memory (M x 128
// of the 512 columns; two members leave room for two blocks), and the epilogue
// turns them into mean and spread in registers: only the results leave, by whole
// 32-byte sectors of a lane's row (343 -> 207 us), and the hidden layers of all members share a launch each (160 -> 47 us
// over three layers: 256 CTAs a launch left the last of two waves half empty).
// Roles as in gemm_tn_persistent, with sixteen epilogue warps (a lane quadrant and
// 32 columns each), because four members leave no room for a second accumulator
// and the statistics are exposed: eight warps, with the results through shared
// memory and bulk copies, took 33 us more; blocks of 64 columns, two at a time, 4.
// Every value sees ensemble_stats' operations in
// its order.
// ---------------------------------------------------------------------------
struct EnsembleArgs {
    CUtensorMap a[kMaxGroup], b[kMaxGroup];
    const float* bias[kMaxGroup];
    float *mean, *spread;  // [rows][N], 32-byte aligned
    float scale, mid, lo, hi;
};
constexpr int kEBN = 128, kEStage = kUTileA + kEBN * UBK * 2, kEStages = 6;
constexpr int kEWarps = 16;  // of the epilogue
constexpr int kEThreads = 64 + 32 * kEWarps;
constexpr size_t kESmem = (size_t)kEStages * kEStage + kEWarps * kMaxGroup * 32 * sizeof(float) + 1024 + 256;

// 8 columns of this lane's row; they are there after tcgen05.wait::ld.
__device__ __forceinline__ void tmem_ld8(uint32_t addr, float* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "r"(addr));
}

template <int M>
__global__ void __launch_bounds__(kEThreads, 1)
    ensemble_tile(const __grid_constant__ EnsembleArgs t, int rows, int N, int K, int* err) {
    static_assert(M >= 2 && M <= kMaxGroup, "members side by side in tensor memory");
    constexpr int kBufs = M * kEBN * 2 <= 512 ? 2 : 1, kColumns = 512;
    constexpr uint32_t idesc =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kEBN >> 3) << 17) | ((uint32_t)(UBM >> 4) << 24);
    extern __shared__ __align__(1024) unsigned char usmem[];
    unsigned char* base = (unsigned char*)(((uintptr_t)usmem + 1023) & ~(uintptr_t)1023);
    auto tA = [&](int st) { return base + st * kEStage; };
    auto tB = [&](int st) { return base + st * kEStage + kUTileA; };
    float* sbias_all = (float*)(base + kEStages * kEStage);
    uint64_t* full = (uint64_t*)(sbias_all + kEWarps * kMaxGroup * 32);
    uint64_t* empty = full + kEStages;
    uint64_t* acc_full = empty + kEStages;      // [kBufs]
    uint64_t* acc_empty = acc_full + kBufs;     // [kBufs]
    uint32_t* taddr_s = (uint32_t*)(acc_empty + kBufs);
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int nk = K / UBK, nbm = rows / UBM, nblocks = nbm * (N / kEBN);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(taddr_s)),
                     "r"(kColumns));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 32) {
        for (int s = 0; s < kEStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < kBufs; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], kEWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    launch_order();
    const uint32_t tmem = *taddr_s;
    bool ok = true;
    int issued = 0;

    if (warp == 0) {
        int g = 0;
        for (int blk = blockIdx.x; blk < nblocks && ok; blk += gridDim.x) {
            const int bm = (blk % nbm) * UBM, bn = (blk / nbm) * kEBN;
            for (int k = 0; k < M && ok; ++k)
                for (int kt = 0; kt < nk && ok; ++kt, ++g) {
                    const int st = g % kEStages;
                    if (g >= kEStages) ok = warp_wait(&empty[st], ((g / kEStages) - 1) & 1);
                    if (!ok) break;
                    if (elect_lane()) {
                        mbar_expect_tx(&full[st], (unsigned)kEStage);
                        tma_load_2d(tA(st), &t.a[k], kt * UBK, bm, &full[st]);
                        tma_load_2d(tB(st), &t.b[k], kt * UBK, bn, &full[st]);
                    }
                    __syncwarp();
                    issued = g + 1;
                }
        }
    } else if (warp == 1) {
        int g = 0, i = 0;
        for (int blk = blockIdx.x; blk < nblocks && ok; blk += gridDim.x, ++i) {
            const int a = i % kBufs;
            if (i >= kBufs) ok = warp_wait(&acc_empty[a], ((i / kBufs) - 1) & 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int k = 0; k < M && ok; ++k)
                for (int kt = 0; kt < nk && ok; ++kt, ++g) {
                    const int st = g % kEStages;
                    ok = warp_wait(&full[st], (g / kEStages) & 1);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elect_lane()) {
                        mma_stage(tmem + (uint32_t)((a * M + k) * kEBN), smem_u32(tA(st)), smem_u32(tB(st)), idesc,
                                  kt == 0);
                        mma_commit(&empty[st]);
                    }
                    __syncwarp();
                }
            if (!ok) break;
            if (elect_lane()) mma_commit(&acc_full[a]);
            __syncwarp();
        }
    } else {
        const int q = warp & 3, c = 32 * ((warp - 2) >> 2);  // this warp's rows and columns of a block
        float* sbias = sbias_all + (warp - 2) * kMaxGroup * 32;
        const float inv = 1.f / (float)M;
        int i = 0;
        for (int blk = blockIdx.x; blk < nblocks && ok; blk += gridDim.x, ++i) {
            const int a = i % kBufs;
            const int bm = (blk % nbm) * UBM, bn = (blk / nbm) * kEBN + c;
            __syncwarp();
#pragma unroll
            for (int k = 0; k < M; ++k) sbias[k * 32 + lane] = t.bias[k][bn + lane];
            __syncwarp();
            ok &= mbar_wait(&acc_full[a], (i / kBufs) & 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const size_t out = (size_t)(bm + q * 32 + lane) * N + bn;
#pragma unroll 1
            for (int h = 0; h < 32; h += 8) {
                float x[M][8];
#pragma unroll
                for (int k = 0; k < M; ++k)
                    tmem_ld8(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)((a * M + k) * kEBN + c + h), x[k]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                uint32_t mean[8], spread[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float s, d = 0.f;
#pragma unroll
                    for (int k = 0; k < M; ++k) {
                        // the loads land at the wait: no use of x may move above it
                        asm volatile("" : "+f"(x[k][j]));
                        x[k][j] = member_tl(x[k][j] + sbias[k * 32 + h + j], t.scale, t.mid, t.lo, t.hi);
                        s = k ? s + x[k][j] : x[k][j];
                    }
                    s *= inv;
#pragma unroll
                    for (int k = 0; k < M; ++k) d = fmaf(x[k][j] - s, x[k][j] - s, d);
                    mean[j] = __float_as_uint(s);
                    spread[j] = __float_as_uint(sqrtf(d * inv));
                }
                if (h == 24) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0)
                        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[a])) : "memory");
                }
                store_sector(t.mean + out + h, mean);
                store_sector(t.spread + out + h, spread);
            }
        }
    }
    __syncwarp();
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    if (!ok && warp == 0 && lane == 0) {
        for (int g = issued - 1; g >= 0 && g >= issued - kEStages; --g)
            mbar_wait(&full[g % kEStages], (g / kEStages) & 1);
    }
    if (!ok && tid == 0) atomicExch(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kColumns));
}

using crk::encode_tiled;
using crk::EncodeTiledFn;

// Tensor map of a rows x K bf16 operand (row stride ld elements) in boxes of
// `box_rows` rows x 64 elements, 128-byte swizzle: the layout the MMAs read.
bool operand_map(CUtensorMap* map, const void* ptr, int rows, int K, int ld, int box_rows) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)UBK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor map of a rows x cols output (f32 or bf16) or mask in boxes of 128
// bytes x box_rows rows, 128-byte swizzle.
bool tile_map(CUtensorMap* map, const void* ptr, bool bf16, int rows, int cols, int ld, int box_rows) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const int eb = bf16 ? 2 : 4;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * eb};
    const cuuint32_t box[2] = {(cuuint32_t)(128 / eb), (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
               const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct TileOperands {
    const void *A, *B;
    int M, N, K, lda, ldb;
};

// A launch that may start before the stream's last kernel has ended (launch_order).
template <typename... P, typename... A>
cudaError_t launch_next(void (*f)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, f, args...);
}

// G equal contractions (o and e of each) by gemm_tn_tile.
template <int EPI, int BN, int ST, int G>
cudaError_t launch_tile(const TileOperands* o, const EpiArgs* e, int* err, cudaStream_t st) {
    using T = TileGemm<EPI, BN, ST>;
    TileMaps<G> t;
    for (int g = 0; g < G; ++g) {
        if (!operand_map(&t.a[g], o[g].A, o[g].M, o[g].K, o[g].lda, UBM) ||
            !operand_map(&t.b[g], o[g].B, o[g].N, o[g].K, o[g].ldb, BN) ||
            !tile_map(&t.o[g], e[g].out, epi_bf16<EPI>(), o[g].M, o[g].N, e[g].ldo, 32))
            return cudaErrorUnknown;
        t.bias[g] = e[g].bias;
    }
    t.m[0] = t.o[0];
    if (T::kMask && !tile_map(&t.m[0], e[0].mask, true, o[0].M, o[0].N, e[0].ldm, UBM)) return cudaErrorUnknown;
    auto* f = gemm_tn_tile<EPI, BN, ST, G>;
    const cudaError_t ce = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::smem);
    if (ce != cudaSuccess) return ce;
    return launch_next(f, dim3(o[0].N / BN, o[0].M / UBM, G), kUThreads, T::smem, st, t, o[0].K, err);
}

int sm_count() {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

template <int EPI>
cudaError_t launch_persistent(const TileOperands& o, const EpiArgs& e, int* err, cudaStream_t st) {
    TileMaps<1> t;
    if (!operand_map(&t.a[0], o.A, o.M, o.K, o.lda, UBM) || !operand_map(&t.b[0], o.B, o.N, o.K, o.ldb, UBN) ||
        !tile_map(&t.o[0], e.out, epi_bf16<EPI>(), o.M, o.N, e.ldo, 32))
        return cudaErrorUnknown;
    t.m[0] = t.o[0];
    t.bias[0] = e.bias;
    auto* f = gemm_tn_persistent<EPI>;
    const cudaError_t ce = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPSmem);
    if (ce != cudaSuccess) return ce;
    const int blocks = (o.M / UBM) * (o.N / UBN), sms = sm_count();
    return launch_next(f, dim3(std::min(blocks, sms)), kPThreads, kPSmem, st, t, o.M, o.N, o.K, err);
}

bool aligned32(const void* p) { return ((uintptr_t)p & 31) == 0; }

// The persistent kernel once every SM has two of its blocks (256 columns; 78 us
// at 8192 x 8192 x 512, 91 by blocks of gemm_tn_tile), else the widest block that
// still gives every SM work.  walk: the persistent
// kernel at any size (a mask takes its shared memory: never there).
template <int EPI>
cudaError_t launch_tile_n(const TileOperands& o, const EpiArgs& e, bool walk, int* err, cudaStream_t st) {
    const long long rows = o.M / UBM, sms = sm_count();
    if constexpr (EPI != CR_MLP_EPI_RELU_MASK_BF16) {
        if (walk || rows * (o.N / 256) >= 2 * sms) return launch_persistent<EPI>(o, e, err, st);
    }
    if (rows * (o.N / 128) >= sms) return launch_tile<EPI, 128, 3, 1>(&o, &e, err, st);
    return launch_tile<EPI, 64, 7, 1>(&o, &e, err, st);
}

// G equal hidden layers (bias, ReLU, bf16) in one launch.
template <int G>
cudaError_t launch_hidden(const TileOperands* o, const EpiArgs* e, int* err, cudaStream_t st) {
    const long long rows = (long long)(o[0].M / UBM) * G;
    if (rows * (o[0].N / 128) >= sm_count()) return launch_tile<CR_MLP_EPI_BIAS_RELU_BF16, 128, 3, G>(o, e, err, st);
    return launch_tile<CR_MLP_EPI_BIAS_RELU_BF16, 64, 7, G>(o, e, err, st);
}

template <int M>
cudaError_t launch_ensemble(const EnsembleArgs& t, int rows, int N, int K, int* err, cudaStream_t st) {
    const cudaError_t ce =
        cudaFuncSetAttribute(ensemble_tile<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kESmem);
    if (ce != cudaSuccess) return ce;
    return launch_next(ensemble_tile<M>, dim3(std::min((rows / UBM) * (N / kEBN), sm_count())), kEThreads, kESmem, st, t,
                       rows, N, K, err);
}

}  // namespace

extern "C" {

int cr_mlp_gemm(int epi, const void* A, const void* B, int M, int N, int K, int lda, int ldb, void* out, int ldo,
                const float* bias, const void* mask, int ldm, void* stream) {
    if (M <= 0 || N <= 0 || K <= 0 || M % BM || N % BN || K % BK) return CR_MLP_EBADSHAPE;
    if (lda < K || ldb < K || lda % 8 || ldb % 8 || ldo < N || ldo % 2 || !aligned16(A) || !aligned16(B) || !out)
        return CR_MLP_EBADSHAPE;
    if ((epi == CR_MLP_EPI_BIAS_RELU_BF16 || epi == CR_MLP_EPI_BIAS_F32) && !bias) return CR_MLP_EBADSHAPE;
    if (epi == CR_MLP_EPI_RELU_MASK_BF16 && (!mask || ldm < N || ldm % 2)) return CR_MLP_EBADSHAPE;
    EpiArgs e{out, ldo, bias, (const __nv_bfloat16*)mask, ldm};
    const dim3 grid(N / BN, M / BM);
    cudaStream_t st = (cudaStream_t)stream;
    auto a = (const __nv_bfloat16*)A;
    auto b = (const __nv_bfloat16*)B;
    switch (epi) {
        case CR_MLP_EPI_BIAS_RELU_BF16: gemm_tn<CR_MLP_EPI_BIAS_RELU_BF16><<<grid, kThreads, 0, st>>>(a, b, K, lda, ldb, e); break;
        case CR_MLP_EPI_BIAS_F32: gemm_tn<CR_MLP_EPI_BIAS_F32><<<grid, kThreads, 0, st>>>(a, b, K, lda, ldb, e); break;
        case CR_MLP_EPI_F32: gemm_tn<CR_MLP_EPI_F32><<<grid, kThreads, 0, st>>>(a, b, K, lda, ldb, e); break;
        case CR_MLP_EPI_RELU_MASK_BF16: gemm_tn<CR_MLP_EPI_RELU_MASK_BF16><<<grid, kThreads, 0, st>>>(a, b, K, lda, ldb, e); break;
        default: return CR_MLP_EBADSHAPE;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : CR_MLP_ECUDA;
}

int cr_mlp_gemm_tc(int epi, const void* A, const void* B, int M, int N, int K, int lda, int ldb, void* out, int ldo,
                   const float* bias, const void* mask, int ldm, int* err, void* stream) {
    if (M <= 0 || N <= 0 || K <= 0 || M % UBM || N % UBN || K % UBK) return CR_MLP_EBADSHAPE;
    if (lda < K || ldb < K || lda % 8 || ldb % 8 || ldo < N || ldo % 2 || !aligned16(A) || !aligned16(B) || !out ||
        !err)
        return CR_MLP_EBADSHAPE;
    if ((epi == CR_MLP_EPI_BIAS_RELU_BF16 || epi == CR_MLP_EPI_BIAS_F32) && !bias) return CR_MLP_EBADSHAPE;
    if (epi == CR_MLP_EPI_RELU_MASK_BF16 && (!mask || ldm < N || ldm % 2)) return CR_MLP_EBADSHAPE;
    EpiArgs e{out, ldo, bias, (const __nv_bfloat16*)mask, ldm};
    const dim3 grid(N / UBN, M / UBM);
    cudaStream_t st = (cudaStream_t)stream;
    auto a = (const __nv_bfloat16*)A;
    auto b = (const __nv_bfloat16*)B;
    cudaError_t ce = cudaSuccess;
    const int feed = gemm_feed();
    // outputs (and a mask) whose rows start on 16-byte boundaries leave by bulk copies
    const bool half = epi == CR_MLP_EPI_BIAS_RELU_BF16 || epi == CR_MLP_EPI_RELU_MASK_BF16;
    const bool out16 = aligned16(out) && ldo % (half ? 8 : 4) == 0;
    if (feed >= 1 && out16 && (epi != CR_MLP_EPI_RELU_MASK_BF16 || (aligned16(mask) && ldm % 8 == 0))) {
        const TileOperands o{A, B, M, N, K, lda, ldb};
        const bool walk = feed == 2;
        switch (epi) {
            case CR_MLP_EPI_BIAS_RELU_BF16: ce = launch_tile_n<CR_MLP_EPI_BIAS_RELU_BF16>(o, e, walk, err, st); break;
            case CR_MLP_EPI_BIAS_F32: ce = launch_tile_n<CR_MLP_EPI_BIAS_F32>(o, e, walk, err, st); break;
            case CR_MLP_EPI_F32: ce = launch_tile_n<CR_MLP_EPI_F32>(o, e, walk, err, st); break;
            case CR_MLP_EPI_RELU_MASK_BF16: ce = launch_tile_n<CR_MLP_EPI_RELU_MASK_BF16>(o, e, walk, err, st); break;
            default: return CR_MLP_EBADSHAPE;
        }
        return ce == cudaSuccess ? 0 : CR_MLP_ECUDA;
    }
    if (feed >= 1) {
        // operands by the tensor memory accelerator (tensor maps over this GPU's memory)
        CUtensorMap ma, mb;
        if (!operand_map(&ma, A, M, K, lda, UBM) || !operand_map(&mb, B, N, K, ldb, UBN)) return CR_MLP_ECUDA;
        switch (epi) {
#define CR_TMA_CASE(E)                                                                                       \
    case E:                                                                                                  \
        ce = cudaFuncSetAttribute(gemm_tn_tma<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTSmem);   \
        if (ce == cudaSuccess) gemm_tn_tma<E><<<grid, kUThreads, kTSmem, st>>>(ma, mb, K, e, err);            \
        break;
            CR_TMA_CASE(CR_MLP_EPI_BIAS_RELU_BF16)
            CR_TMA_CASE(CR_MLP_EPI_BIAS_F32)
            CR_TMA_CASE(CR_MLP_EPI_F32)
            CR_TMA_CASE(CR_MLP_EPI_RELU_MASK_BF16)
#undef CR_TMA_CASE
            default: return CR_MLP_EBADSHAPE;
        }
        if (ce != cudaSuccess) return CR_MLP_ECUDA;
        return cudaGetLastError() == cudaSuccess ? 0 : CR_MLP_ECUDA;
    }
    switch (epi) {
#define CR_UMMA_CASE(E)                                                                                    \
    case E:                                                                                                \
        ce = cudaFuncSetAttribute(gemm_tn_umma<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kUSmem); \
        if (ce == cudaSuccess) gemm_tn_umma<E><<<grid, kUThreads, kUSmem, st>>>(a, b, K, lda, ldb, e, err);      \
        break;
        CR_UMMA_CASE(CR_MLP_EPI_BIAS_RELU_BF16)
        CR_UMMA_CASE(CR_MLP_EPI_BIAS_F32)
        CR_UMMA_CASE(CR_MLP_EPI_F32)
        CR_UMMA_CASE(CR_MLP_EPI_RELU_MASK_BF16)
#undef CR_UMMA_CASE
        default: return CR_MLP_EBADSHAPE;
    }
    if (ce != cudaSuccess) return CR_MLP_ECUDA;
    return cudaGetLastError() == cudaSuccess ? 0 : CR_MLP_ECUDA;
}

int cr_mlp_transpose(const void* src, int lds, void* dst, int ldd, int rows, int cols, void* stream) {
    if (rows <= 0 || cols <= 0 || lds < cols || ldd < rows) return CR_MLP_EBADSHAPE;
    const dim3 grid((cols + 31) / 32, (rows + 31) / 32), block(32, 8);
    transpose_bf16<<<grid, block, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)src, lds, (__nv_bfloat16*)dst, ldd,
                                                              rows, cols);
    return cudaGetLastError() == cudaSuccess ? 0 : CR_MLP_ECUDA;
}

int cr_mlp_col_sum(const void* src, int ld, int rows, int cols, float* out, void* stream) {
    if (rows <= 0 || cols <= 0 || ld < cols) return CR_MLP_EBADSHAPE;
    Mats t{};
    t.n = 1;
    t.first[1] = (cols + 63) / 64;
    t.src[0] = (const __nv_bfloat16*)src;
    t.dst[0] = out;
    t.lds[0] = ld;
    t.rows[0] = rows;
    t.cols[0] = cols;
    col_sum_mats<<<t.first[1], dim3(32, 32), 0, (cudaStream_t)stream>>>(t);
    return cudaGetLastError() == cudaSuccess ? 0 : CR_MLP_ECUDA;
}

int cr_mlp_mse_grad(const float* pred, const void* target, const unsigned char* valid, long long n, float inv_count,
                    void* grad, double* sse, void* stream) {
    if (n <= 0) return CR_MLP_EBADSHAPE;
    const bool vec = n % 4 == 0 && aligned16(pred) && ((uintptr_t)target & 7) == 0 && ((uintptr_t)grad & 7) == 0 &&
                     ((uintptr_t)valid & 3) == 0;
    cudaStream_t st = (cudaStream_t)stream;
    auto y = (const __nv_bfloat16*)target;
    auto gr = (__nv_bfloat16*)grad;
    // four blocks an SM: each block's sum of squares is one atomic
    const long long want = ((vec ? n / 4 : n) + 255) / 256;
    const int grid = (int)(want < 592 ? want : 592);
    if (vec) mse_grad<true><<<grid, 256, 0, st>>>(pred, y, valid, n, inv_count, gr, sse);
    else mse_grad<false><<<grid, 256, 0, st>>>(pred, y, valid, n, inv_count, gr, sse);
    return cudaGetLastError() == cudaSuccess ? 0 : CR_MLP_ECUDA;
}

static AdamArgs adam_args(float lr, float beta1, float beta2, float eps, int step) {
    return AdamArgs{lr, beta1, beta2, eps, 1.f / (1.f - powf(beta1, (float)step)),
                    1.f / (1.f - powf(beta2, (float)step))};
}

int cr_mlp_adam(float* p, const float* g, float* m, float* v, void* p_bf16, long long n, float lr, float beta1,
                float beta2, float eps, int step, float weight_decay, void* stream) {
    if (n <= 0 || step < 1) return CR_MLP_EBADSHAPE;
    adam_step<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(p, g, m, v, (__nv_bfloat16*)p_bf16, n,
                                                             adam_args(lr, beta1, beta2, eps, step), weight_decay);
    return cudaGetLastError() == cudaSuccess ? 0 : CR_MLP_ECUDA;
}

namespace {
int mlp_gemm_any(int epi, int tc, const void* A, const void* B, int M, int N, int K, int lda, int ldb, void* out,
                 const float* bias, const void* mask, int ldm, int* err, void* stream) {
    if (tc && N % UBN == 0 && K % UBK == 0)
        return cr_mlp_gemm_tc(epi, A, B, M, N, K, lda, ldb, out, N, bias, mask, ldm, err, stream);
    return cr_mlp_gemm(epi, A, B, M, N, K, lda, ldb, out, N, bias, mask, ldm, stream);
}
bool mlp_dims_ok(const cr_mlp_net* net, int batch) {
    if (!net || net->layers < 1 || batch <= 0 || batch % 128) return false;
    for (int l = 0; l <= net->layers; ++l)
        if (net->dims[l] <= 0 || net->dims[l] % 128) return false;
    return true;
}
}  // namespace

int cr_mlp_forward(const cr_mlp_net* net, int batch, const void* x, int ldx, float* out, int tc, int* err,
                   void* stream) {
    if (!mlp_dims_ok(net, batch) || !x || !out) return CR_MLP_EBADSHAPE;
    const void* in = x;
    int ld = ldx;
    for (int l = 0; l < net->layers; ++l) {
        const bool last = l == net->layers - 1;
        void* to = last ? (void*)out : net->act[l + 1];
        const int rc = mlp_gemm_any(last ? CR_MLP_EPI_BIAS_F32 : CR_MLP_EPI_BIAS_RELU_BF16, tc, in, net->w16[l], batch,
                                    net->dims[l + 1], net->dims[l], ld, net->dims[l], to, net->b[l], nullptr, 0, err,
                                    stream);
        if (rc) return rc;
        in = to;
        ld = net->dims[l + 1];
    }
    return CR_MLP_OK;
}

int cr_mlp_backward(const cr_mlp_net* net, int batch, const void* x, int ldx, int tc, int* err, void* stream) {
    if (!mlp_dims_ok(net, batch) || !x || ldx % 8 || !aligned16(x)) return CR_MLP_EBADSHAPE;
    cudaStream_t st = (cudaStream_t)stream;
    const int L = net->layers;
    for (int l = 0; l < L; ++l)  // transpose_mats moves 16 bytes at a time
        if (!aligned16(net->grad[l]) || !aligned16(net->grad_t[l]) || !aligned16(net->act_t[l]) ||
            (l > 0 && !aligned16(net->act[l])))
            return CR_MLP_EBADSHAPE;
    // gradients down to the first layer's output, through the ReLU whose output was act[l]
    for (int l = L - 1; l > 0; --l) {
        const int rc = mlp_gemm_any(CR_MLP_EPI_RELU_MASK_BF16, tc, net->grad[l], net->wt16[l], batch, net->dims[l],
                                    net->dims[l + 1], net->dims[l + 1], net->dims[l + 1], net->grad[l - 1], nullptr,
                                    net->act[l], net->dims[l], err, stream);
        if (rc) return rc;
    }
    // dW = grad^T act: both transposed to batch-contiguous rows, and the bias
    // gradients, kMaxMats / 2 layers to a launch
    for (int l0 = 0; l0 < L; l0 += kMaxMats / 2) {
        Mats t{}, c{};
        for (int l = l0; l < L && l < l0 + kMaxMats / 2; ++l) {
            const int d_out = net->dims[l + 1], d_in = net->dims[l];
            auto put = [&](const void* src, int ld, void* dst, int cols) {
                const int i = t.n++;
                t.src[i] = (const __nv_bfloat16*)src;
                t.dst[i] = dst;
                t.lds[i] = ld;
                t.ldd[i] = batch;
                t.rows[i] = batch;
                t.cols[i] = cols;
                t.first[i + 1] = t.first[i] + (batch / 64) * (cols / 64);
            };
            put(net->grad[l], d_out, net->grad_t[l], d_out);
            put(l == 0 ? x : net->act[l], l == 0 ? ldx : d_in, net->act_t[l], d_in);
            const int i = c.n++;
            c.src[i] = (const __nv_bfloat16*)net->grad[l];
            c.dst[i] = net->gb[l];
            c.lds[i] = c.cols[i] = d_out;
            c.rows[i] = batch;
            c.first[i + 1] = c.first[i] + d_out / 64;
        }
        if (launch_next(transpose_mats, dim3(t.first[t.n]), dim3(256), 0, st, t) != cudaSuccess ||
            launch_next(col_sum_mats, dim3(c.first[c.n]), dim3(32, 32), 0, st, c) != cudaSuccess)
            return CR_MLP_ECUDA;
    }
    for (int l = L - 1; l >= 0; --l) {
        const int rc = mlp_gemm_any(CR_MLP_EPI_F32, tc, net->grad_t[l], net->act_t[l], net->dims[l + 1], net->dims[l],
                                    batch, batch, batch, net->gw[l], nullptr, nullptr, 0, err, stream);
        if (rc) return rc;
    }
    return CR_MLP_OK;
}

int cr_mlp_step(const cr_mlp_net* net, float lr, float beta1, float beta2, float eps, int step, float weight_decay,
                void* stream) {
    if (!mlp_dims_ok(net, 128) || step < 1) return CR_MLP_EBADSHAPE;
    for (int l0 = 0; l0 < net->layers; l0 += kMaxMats / 2) {
        AdamMats t{};
        for (int l = l0; l < net->layers && l < l0 + kMaxMats / 2; ++l) {
            const int d_out = net->dims[l + 1], d_in = net->dims[l];
            // the fused kernel moves 16 bytes at a time; matrices that start elsewhere go
            // through the single-matrix calls
            if (!aligned16(net->w[l]) || !aligned16(net->gw[l]) || !aligned16(net->mw[l]) || !aligned16(net->vw[l]) ||
                !aligned16(net->w16[l]) || !aligned16(net->wt16[l])) {
                int rc = cr_mlp_adam(net->w[l], net->gw[l], net->mw[l], net->vw[l], net->w16[l], (long long)d_out * d_in,
                                     lr, beta1, beta2, eps, step, weight_decay, stream);
                if (!rc) rc = cr_mlp_transpose(net->w16[l], d_in, net->wt16[l], d_out, d_out, d_in, stream);
                if (!rc)
                    rc = cr_mlp_adam(net->b[l], net->gb[l], net->mb[l], net->vb[l], nullptr, d_out, lr, beta1, beta2, eps,
                                     step, 0.f, stream);
                if (rc) return rc;
                continue;
            }
            const int w = t.n, b = w + 1;
            t.n += 2;
            t.p[w] = net->w[l];
            t.g[w] = net->gw[l];
            t.m[w] = net->mw[l];
            t.v[w] = net->vw[l];
            t.pb[w] = (__nv_bfloat16*)net->w16[l];
            t.pt[w] = (__nv_bfloat16*)net->wt16[l];
            t.rows[w] = d_out;
            t.cols[w] = d_in;
            t.first[w + 1] = t.first[w] + (d_out / 64) * (d_in / 64);
            t.p[b] = net->b[l];
            t.g[b] = net->gb[l];
            t.m[b] = net->mb[l];
            t.v[b] = net->vb[l];
            t.rows[b] = d_out;
            t.cols[b] = 1;
            t.first[b + 1] = t.first[b] + (d_out + 4095) / 4096;
        }
        if (t.n == 0) continue;
        if (launch_next(adam_mats, dim3(t.first[t.n]), dim3(256), 0, (cudaStream_t)stream, t,
                        adam_args(lr, beta1, beta2, eps, step), weight_decay) != cudaSuccess)
            return CR_MLP_ECUDA;
    }
    return CR_MLP_OK;
}

namespace {
// The members' networks have one shape, and every contraction is one that the
// default tcgen05 path takes with bulk-copy epilogues.
bool ensemble_fits(const cr_mlp_net* const* nets, int members, int batch, const void* x, int ldx, int tc,
                   const float* mean, const float* spread) {
    if (!tc || members < 2 || members > kMaxGroup || gemm_feed() != 1 || ldx < nets[0]->dims[0] || ldx % 8 ||
        !aligned16(x) || !aligned32(mean) || !aligned32(spread))
        return false;
    const int L = nets[0]->layers;
    for (int k = 0; k < members; ++k) {
        if (nets[k]->layers != L || !mlp_dims_ok(nets[k], batch)) return false;
        for (int l = 0; l <= L; ++l)
            if (nets[k]->dims[l] != nets[0]->dims[l]) return false;
        for (int l = 0; l < L; ++l)
            if (nets[k]->dims[l + 1] % UBN || nets[k]->dims[l] % UBK || !nets[k]->b[l] ||
                !aligned16(nets[k]->w16[l]) || (l > 0 && !aligned16(nets[k]->act[l])))
                return false;
    }
    return true;
}
}  // namespace

int cr_mlp_ensemble_predict(const cr_mlp_net* const* nets, int members, int batch, const void* x, int ldx,
                            float* const* outs, int tc, float scale, float mid, float lo, float hi, float* mean,
                            float* spread, int* err, void* stream) {
    if (!nets || members < 1 || members > kMaxMembers || !x || !outs || !mean || !spread) return CR_MLP_EBADSHAPE;
    for (int k = 0; k < members; ++k)
        if (!nets[k] || !mlp_dims_ok(nets[k], batch) ||
            nets[k]->dims[nets[k]->layers] != nets[0]->dims[nets[0]->layers])
            return CR_MLP_EBADSHAPE;  // the statistics are over outputs of one width
    cudaStream_t st = (cudaStream_t)stream;
    if (!err || !ensemble_fits(nets, members, batch, x, ldx, tc, mean, spread)) {
        for (int k = 0; k < members; ++k) {
            const int rc = cr_mlp_forward(nets[k], batch, x, ldx, outs[k], tc, err, stream);
            if (rc) return rc;
        }
        const long long n = (long long)batch * nets[0]->dims[nets[0]->layers];
        return cr_mlp_ensemble_stats(outs, members, n, scale, mid, lo, hi, mean, spread, stream);
    }
    const int L = nets[0]->layers;
    const int* d = nets[0]->dims;
    cudaError_t ce = cudaSuccess;
    for (int l = 0; l < L - 1 && ce == cudaSuccess; ++l) {
        TileOperands o[kMaxGroup];
        EpiArgs e[kMaxGroup];
        for (int k = 0; k < members; ++k) {
            o[k] = {l ? nets[k]->act[l] : x, nets[k]->w16[l], batch, d[l + 1], d[l], l ? d[l] : ldx, d[l]};
            e[k] = {nets[k]->act[l + 1], d[l + 1], nets[k]->b[l], nullptr, 0};
        }
        ce = members == 2 ? launch_hidden<2>(o, e, err, st)
                          : (members == 3 ? launch_hidden<3>(o, e, err, st) : launch_hidden<4>(o, e, err, st));
    }
    if (ce != cudaSuccess) return CR_MLP_ECUDA;
    EnsembleArgs t;
    const int K = d[L - 1], N = d[L];
    for (int k = 0; k < members; ++k) {
        if (!operand_map(&t.a[k], L > 1 ? nets[k]->act[L - 1] : x, batch, K, L > 1 ? K : ldx, UBM) ||
            !operand_map(&t.b[k], nets[k]->w16[L - 1], N, K, K, kEBN))
            return CR_MLP_ECUDA;
        t.bias[k] = nets[k]->b[L - 1];
    }
    t.mean = mean;
    t.spread = spread;
    t.scale = scale;
    t.mid = mid;
    t.lo = lo;
    t.hi = hi;
    ce = members == 2 ? launch_ensemble<2>(t, batch, N, K, err, st)
                      : (members == 3 ? launch_ensemble<3>(t, batch, N, K, err, st)
                                      : launch_ensemble<4>(t, batch, N, K, err, st));
    return ce == cudaSuccess ? CR_MLP_OK : CR_MLP_ECUDA;
}

int cr_mlp_ensemble_stats(const float* const* preds, int members, long long n, float scale, float mid, float lo,
                          float hi, float* mean, float* spread, void* stream) {
    if (!preds || members < 1 || members > kMaxMembers || n <= 0 || n % 4 || !aligned16(mean) || !aligned16(spread))
        return CR_MLP_EBADSHAPE;
    Members p{};
    for (int k = 0; k < members; ++k) {
        if (!preds[k] || !aligned16(preds[k])) return CR_MLP_EBADSHAPE;
        p.out[k] = preds[k];
    }
    cudaStream_t st = (cudaStream_t)stream;
    const long long n4 = n / 4, want = (n4 + 255) / 256;
    const int grid = (int)(want < 148 * 16 ? want : 148 * 16);
    auto m4 = (float4*)mean;
    auto s4 = (float4*)spread;
    switch (members) {
        case 2: ensemble_stats<2><<<grid, 256, 0, st>>>(p, members, n4, scale, mid, lo, hi, m4, s4); break;
        case 3: ensemble_stats<3><<<grid, 256, 0, st>>>(p, members, n4, scale, mid, lo, hi, m4, s4); break;
        case 4: ensemble_stats<4><<<grid, 256, 0, st>>>(p, members, n4, scale, mid, lo, hi, m4, s4); break;
        default: ensemble_stats<0><<<grid, 256, 0, st>>>(p, members, n4, scale, mid, lo, hi, m4, s4); break;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : CR_MLP_ECUDA;
}

int cr_mlp_to_bf16(const float* src, void* dst, long long n, void* stream) {
    if (n <= 0) return CR_MLP_EBADSHAPE;
    to_bf16<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(src, (__nv_bfloat16*)dst, n);
    return cudaGetLastError() == cudaSuccess ? 0 : CR_MLP_ECUDA;
}

}  // extern "C"
