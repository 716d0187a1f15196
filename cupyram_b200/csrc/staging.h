// staging.h - host-device copies of pageable memory through pinned rings (host
// code; needs nothing of CUDA but the runtime's copy and event calls).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>

namespace crk {

// Pinned staging of host-to-device copies.  A pageable cudaMemcpy is staged
// by the driver through its own pinned buffers, one host copy at a time; here
// each device has a ring of two pinned chunks, allocated once: while one
// chunk's DMA runs, host threads fill the other, so the host copy and the
// transfer overlap and the copy itself runs on several cores.
constexpr int kStageDevices = 64;
constexpr size_t kStageChunk = 16u << 20;  // bytes per chunk
constexpr size_t kStageMin = 4u << 20;     // smaller copies go direct
constexpr int kStageThreads = 4;
struct StageRing {
    unsigned char* buf[2] = {nullptr, nullptr};
    cudaEvent_t done[2] = {nullptr, nullptr};
    cudaEvent_t out[32] = {};  // staged_d2h: one per piece
};
inline StageRing g_stage[kStageDevices];
inline std::mutex g_stage_mu[kStageDevices];

inline void copy_parallel(unsigned char* dst, const unsigned char* src, size_t n) {
    if (n < (1u << 20)) {
        memcpy(dst, src, n);
        return;
    }
    std::thread th[kStageThreads - 1];
    const size_t part = (n / kStageThreads + 63) & ~size_t(63);
    for (int t = 1; t < kStageThreads; ++t) {
        const size_t lo = std::min(n, part * t), hi = std::min(n, part * (t + 1));
        th[t - 1] = std::thread([=] { memcpy(dst + lo, src + lo, hi - lo); });
    }
    memcpy(dst, src, std::min(n, part));
    for (auto& x : th) x.join();
}

// Host-to-device copy of `bytes` through the device's pinned ring, ordered on
// `st`.  Returns when the last chunk's copy has been queued (the caller
// synchronises the stream); the ring is held until then.
inline cudaError_t staged_h2d(int dev, void* dst, const void* src, size_t bytes, cudaStream_t st) {
    if (dev < 0 || dev >= kStageDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_stage_mu[dev]);
    StageRing& R = g_stage[dev];
    cudaError_t ce = cudaSuccess;
    for (int k = 0; k < 2 && ce == cudaSuccess; ++k) {
        if (!R.buf[k]) ce = cudaHostAlloc((void**)&R.buf[k], kStageChunk, cudaHostAllocPortable);
        if (ce == cudaSuccess && !R.done[k]) ce = cudaEventCreateWithFlags(&R.done[k], cudaEventDisableTiming);
    }
    const unsigned char* s = (const unsigned char*)src;
    unsigned char* d = (unsigned char*)dst;
    int k = 0;
    for (size_t off = 0; off < bytes && ce == cudaSuccess; off += kStageChunk, k ^= 1) {
        const size_t n = std::min(kStageChunk, bytes - off);
        ce = cudaEventSynchronize(R.done[k]);  // the chunk's previous DMA has finished
        if (ce != cudaSuccess) break;
        copy_parallel(R.buf[k], s + off, n);
        ce = cudaMemcpyAsync(d + off, R.buf[k], n, cudaMemcpyHostToDevice, st);
        if (ce == cudaSuccess) ce = cudaEventRecord(R.done[k], st);
    }
    // the ring is reused by the next call only after these copies: wait for them
    for (int j = 0; j < 2 && ce == cudaSuccess; ++j) ce = cudaEventSynchronize(R.done[j]);
    return ce;
}

// Device-to-host copy of `bytes` into pageable memory through the same ring, in
// pieces of 1 MB: their DMAs are queued at once and host threads copy each piece
// out as it arrives.  The driver's own staging copies on one thread, which for a
// freshly allocated result spends its time on page faults (12 MB: 3.9 ms, here
// 1.9 ms).  Returns with the copy complete.
constexpr size_t kOutPiece = 1u << 20;
constexpr size_t kOutMin = 2u << 20;  // smaller copies go direct
constexpr int kOutThreads = 6;
constexpr int kOutPieces = (int)(2 * kStageChunk / kOutPiece);
static_assert(kOutPieces <= 32, "an event per piece");
inline cudaError_t staged_d2h(int dev, void* dst, const void* src, size_t bytes, cudaStream_t st) {
    if (dev < 0 || dev >= kStageDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_stage_mu[dev]);
    StageRing& R = g_stage[dev];
    cudaError_t ce = cudaSuccess;
    for (int k = 0; k < 2 && ce == cudaSuccess; ++k) {
        if (!R.buf[k]) ce = cudaHostAlloc((void**)&R.buf[k], kStageChunk, cudaHostAllocPortable);
        if (ce == cudaSuccess && !R.done[k]) ce = cudaEventCreateWithFlags(&R.done[k], cudaEventDisableTiming);
    }
    for (int k = 0; k < kOutPieces && ce == cudaSuccess; ++k)
        if (!R.out[k]) ce = cudaEventCreateWithFlags(&R.out[k], cudaEventDisableTiming);
    for (int k = 0; k < 2 && ce == cudaSuccess; ++k) ce = cudaEventSynchronize(R.done[k]);
    auto piece = [&](int k) { return R.buf[k / (kOutPieces / 2)] + (size_t)(k % (kOutPieces / 2)) * kOutPiece; };
    for (size_t off = 0; off < bytes && ce == cudaSuccess; off += 2 * kStageChunk) {
        const size_t span = std::min(2 * kStageChunk, bytes - off);
        const int n = (int)((span + kOutPiece - 1) / kOutPiece);
        auto size = [&](int k) { return std::min(kOutPiece, span - (size_t)k * kOutPiece); };
        int queued = 0;
        for (; queued < n && ce == cudaSuccess; ++queued) {
            ce = cudaMemcpyAsync(piece(queued), (const unsigned char*)src + off + (size_t)queued * kOutPiece,
                                 size(queued), cudaMemcpyDeviceToHost, st);
            if (ce == cudaSuccess) ce = cudaEventRecord(R.out[queued], st);
        }
        std::atomic<int> turn{0}, failed{(int)cudaSuccess};
        auto work = [&] {
            for (int k = turn++; k < n; k = turn++) {
                const cudaError_t e = cudaEventSynchronize(R.out[k]);
                if (e != cudaSuccess) {
                    failed = (int)e;
                    return;
                }
                memcpy((unsigned char*)dst + off + (size_t)k * kOutPiece, piece(k), size(k));
            }
        };
        if (ce == cudaSuccess) {
            std::thread th[kOutThreads - 1];
            // a new thread's device is device 0, whichever the caller's is
            auto on_device = [&] {
                const cudaError_t e = cudaSetDevice(dev);
                if (e == cudaSuccess) work();
                else failed = (int)e;
            };
            try {
                for (int t = 0; t + 1 < std::min(n, kOutThreads); ++t) th[t] = std::thread(on_device);
            } catch (const std::exception&) {
                // no more threads to be had: those that run and this one do the work
            }
            work();
            for (auto& x : th)
                if (x.joinable()) x.join();
            ce = (cudaError_t)failed.load();
        }
        if (ce != cudaSuccess) cudaStreamSynchronize(st);  // no DMA still writes the ring
    }
    return ce;
}

}  // namespace crk
