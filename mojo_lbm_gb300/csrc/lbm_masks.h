// Who may use masks that are not those of the flags alone (host side of lbm_run and lbm_batch_run).
//
// Calls on one handle may overlap on several streams with boundary values of their own, and a call
// captured into a caller's graph is replayed at times and on streams that the handle does not see.  So
// masks that another call may read while this one builds come from the flags alone.  Masks of a run's bc
// (without_resting_walls) belong to the first stream that steps the handle outside a capture, whose calls
// are ordered by that stream.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace lbm {

// From this many steps on a run builds its masks without the walls at rest: the unconditional rebuild
// (62 us on 256^3 cells, 4 us on 256^2) costs less than the bc reads it saves (15 to 23 us and 0.4 us a
// step).
constexpr int64_t kRestingMinSteps = 32;

inline bool is_captured(cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &st) != cudaSuccess) cudaGetLastError();  // (legacy stream during a capture)
    return st != cudaStreamCaptureStatusNone;
}

// The stream whose calls, outside captures, own such masks: the first one to ask.  (By its id: the
// per-thread default streams share a handle value, and a destroyed stream's is given out again.)
struct MaskOwner {
    bool owned = false;
    unsigned long long id = 0;
    bool is(cudaStream_t s) {
        unsigned long long sid = 0;
        if (cudaStreamGetId(s, &sid) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        if (!owned) {
            owned = true;
            id = sid;
        }
        return sid == id;
    }
};

// Memory that a handle can do without: taken at its first use, kept until the handle is destroyed.
struct SpareBuffer {
    void* p = nullptr;
    bool failed = false;
    bool get(size_t bytes) {
        if (p || failed) return p != nullptr;
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // (another stream may be captured meanwhile)
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (cudaMalloc(&p, bytes) != cudaSuccess) {
            cudaGetLastError();  // cleared: the handle works without
            p = nullptr;
            failed = true;
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
        return p != nullptr;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
    }
};

}  // namespace lbm
