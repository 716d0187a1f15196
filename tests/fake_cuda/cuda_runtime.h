// A stand-in for the CUDA runtime, enough to run the host code of
// csrc/staging.h and csrc/lanes.h without a device.  Streams are queues of
// work that runs when an event or the stream is waited for; every call is
// checked to be made with the stream's device current, as a call with another
// device current would create a context there.
#pragma once
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <mutex>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidDevice = 101, cudaErrorNotReady = 600 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice, cudaMemcpyDeviceToHost };
constexpr unsigned cudaHostAllocPortable = 1, cudaEventDisableTiming = 2, cudaStreamNonBlocking = 1;

namespace fake {
inline thread_local int device = 0;
inline int wrong_device = 0, streams_made = 0, streams_alive = 0;
inline std::recursive_mutex mu;
struct Stream {
    int device;
    std::deque<std::function<void()>> work;
};
struct Event {
    int device;
    Stream* stream = nullptr;
};
inline void check(int dev) {
    if (dev != device) ++wrong_device;
}
inline void run(Stream* s, size_t n) {
    for (; n > 0 && !s->work.empty(); --n) {
        s->work.front()();
        s->work.pop_front();
    }
}
}  // namespace fake
typedef fake::Stream* cudaStream_t;
typedef fake::Event* cudaEvent_t;

#define FAKE_LOCK std::lock_guard<std::recursive_mutex> fake_lock(fake::mu)
inline cudaError_t cudaSetDevice(int d) {
    fake::device = d;
    return cudaSuccess;
}
inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = malloc(n);
    return cudaSuccess;
}
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    FAKE_LOCK;
    ++fake::streams_made;
    ++fake::streams_alive;
    *s = new fake::Stream{fake::device, {}};
    return cudaSuccess;
}
inline cudaError_t cudaStreamDestroy(cudaStream_t s) {
    FAKE_LOCK;
    --fake::streams_alive;
    delete s;
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = new fake::Event{fake::device};
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete e;
    return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s) {
    FAKE_LOCK;
    fake::check(s->device);
    s->work.push_back([=] { memcpy(dst, src, n); });
    return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    FAKE_LOCK;
    fake::check(s->device);
    e->stream = s;
    // the event completes when the work in front of it has run
    s->work.push_back([e] { e->stream = nullptr; });
    return cudaSuccess;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    FAKE_LOCK;
    fake::check(e->device);
    while (e->stream && !e->stream->work.empty()) fake::run(e->stream, 1);
    return cudaSuccess;
}
inline cudaError_t cudaStreamQuery(cudaStream_t s) {
    FAKE_LOCK;
    fake::check(s->device);
    return s->work.empty() ? cudaSuccess : cudaErrorNotReady;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    FAKE_LOCK;
    fake::check(s->device);
    fake::run(s, s->work.size());
    return cudaSuccess;
}
