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
#include <cstdint>

namespace lbm {

// From this many steps on a run builds its masks without the walls at rest, in every run anew, for the bc
// reads that its steps save.  Cavities, whose walls rest but for the lid: runs with such masks / with those of
// the flags, us, and the ratio's mean and range over 30 configurations in 3D, 60 in 2D and 20 batches:
//   8 steps     96^3 float32 217.6 / 229.7, 40^3 45.9 / 43.8, 1024^2 101.4 / 95.2; 1.00 (0.88 to 1.12), 1.03 (0.93 to
//               1.08), 0.99 (0.96 to 1.02)
//   16 steps    407.4 / 440.8, 77.2 / 75.7, 188.8 / 181.3; 0.96 (0.85 to 1.05), 1.00 (0.89 to 1.05), 0.97 (0.93 to 1.00)
//   32 steps    787.7 / 869.4, 141.1 / 143.2, 370.1 / 364.0; 0.93 (0.84 to 1.04), 0.98 (0.87 to 1.06), 0.95 (0.91 to 0.98)
//   128 steps   2996 / 3374, 436.4 / 483.0, 1377 / 1377; 0.88 (0.82 to 0.96), 0.98 (0.86 to 1.07), 0.93 (0.88 to 0.98)
// 32 is where every kind gains on average, tiled 2D grids, which have few walls, included (0.997).  (256^3
// float32 371 / 378 us a step, Float16C fast 236 / 252.)
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
