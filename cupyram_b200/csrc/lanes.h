// lanes.h - streams of the engines' launches, kept for the next engine (host
// code; needs nothing of CUDA but the runtime's stream and event calls).
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <vector>

namespace crk {

// A stream with an event.
struct StreamLane {
    cudaStream_t stream = nullptr;
    cudaEvent_t done = nullptr;
};

// Creating and destroying a lane costs about 70 us, and an uneven batch takes
// dozens.  At most kKept idle ones per device are kept; clear destroys them.
class LanePool {
public:
    static constexpr int kDevices = 64;
    static constexpr size_t kKept = 128;

    // A lane of the current device, dev.
    cudaError_t take(int dev, StreamLane* out) {
        if (dev >= 0 && dev < kDevices) {
            std::lock_guard<std::mutex> lock(mu_);
            if (!idle_[dev].empty()) {
                *out = idle_[dev].back();
                idle_[dev].pop_back();
                return cudaSuccess;
            }
        }
        StreamLane l;
        cudaError_t ce = cudaStreamCreateWithFlags(&l.stream, cudaStreamNonBlocking);
        if (ce == cudaSuccess) ce = cudaEventCreateWithFlags(&l.done, cudaEventDisableTiming);
        if (ce != cudaSuccess && l.stream) cudaStreamDestroy(l.stream);
        else *out = l;
        return ce;
    }

    // Waits for what still runs on the lane.
    void give(int dev, StreamLane l) {
        if (!l.stream) return;
        bool idle = cudaStreamQuery(l.stream) == cudaSuccess;
        if (!idle) {
            cudaGetLastError();  // the query's "not ready"
            idle = cudaStreamSynchronize(l.stream) == cudaSuccess;
        }
        if (idle && dev >= 0 && dev < kDevices) {
            std::lock_guard<std::mutex> lock(mu_);
            if (idle_[dev].size() < kKept) {
                idle_[dev].push_back(l);
                return;
            }
        }
        destroy(l);
    }

    void clear() {
        std::lock_guard<std::mutex> lock(mu_);
        for (auto& lanes : idle_) {
            for (const StreamLane& l : lanes) destroy(l);
            lanes.clear();
        }
    }

private:
    static void destroy(const StreamLane& l) {
        cudaEventDestroy(l.done);
        cudaStreamDestroy(l.stream);
    }
    std::mutex mu_;
    std::vector<StreamLane> idle_[kDevices];
};

}  // namespace crk
