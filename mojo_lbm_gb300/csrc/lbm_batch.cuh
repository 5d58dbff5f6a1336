// Batched step: many domains of different size, one launch.
//
// Each domain is a complete single-domain problem (its own grid, tiled layout, f / bc / flags
// buffers and tau), described by a StepArgs.  The work units are the 256-cell tiles of all domains,
// numbered consecutively domain after domain; a CTA steps a few consecutive ones.  It looks its domain
// up in a table (one word per unit), brings the domain's StepArgs into shared memory, reads the first
// unit's masks and only then waits for the previous kernel (programmatic dependent launch), so that
// this overlaps it; each unit runs the body of the single-domain kernel (pair_cells on large double-buffer
// batches other than KBC and D3Q27, else tile_cell), and a batched step equals the single-domain steps
// bit for bit.  Two descriptor arrays hold the even and odd step of every domain (buffers swapped,
// esoteric parity), so the kernel only picks one.
// 128 cylinder channels (14.9 M D2Q9 float32 cells, links included; floor 158 us): 226 us a step with one
// persistent CTA per slot walking 76 units a cell per thread, 213 us with the short walks, 190 us with
// cell pairs.  Bound by issue and by the warps next to walls (a narrow channel has them everywhere).
#pragma once

#include "lbm_aux.cuh"
#include "lbm_pair.cuh"

namespace lbm {

struct BatchArgs {
    const StepArgs* dom;          // ndom descriptors for this step's parity
    const uint32_t* unit_begin;   // ndom + 1 offsets of the domains' first tile units
    const uint32_t* unit_domain;  // the domain of each unit
    const uint2* masks;           // cell masks, 256 per unit: those of the flags, or of this run
    uint32_t ndom, total_units;
    uint32_t per_cta;             // consecutive units of one CTA
    int32_t ready;                // the kernel before this one is part of the same run (its descriptors and
                                  // masks are complete)
};

__device__ __forceinline__ uint32_t find_domain(const uint32_t* begin, uint32_t ndom, uint32_t u) {
    uint32_t lo = 0, hi = ndom;  // begin[lo] <= u < begin[hi]
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(begin + mid) <= u) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Resident CTAs per SM of the batched kernel; LINKS: with the interpolated bounce-back fused in
// (each descriptor's link table; tile_min_blocks of the single-domain kernel).
template <class L, int COLL, bool LINKS>
constexpr int batch_min_blocks() {
    if constexpr (LINKS) return tile_min_blocks<L, COLL, true>();
    else return (L::Q == 9) ? 5 : ((COLL == LBM_KBC || L::Q == 27) ? 3 : 4);
}

// A CTA's walk over its units: the descriptor of the current unit's domain in shared memory (reloaded
// where the range crosses into the next domain) and the unit's tile in that domain.
struct BatchWalk {
    uint32_t u, end, first, next;  // unit, end of the range, units of the current domain: [first, next)
    __device__ __forceinline__ BatchWalk(const BatchArgs& b) {
        u = blockIdx.x * b.per_cta;
        end = min(u + b.per_cta, b.total_units);
        first = next = 0u;
    }
    __device__ __forceinline__ uint32_t tile(const BatchArgs& b, StepArgs* sa) {
        if (u >= next) {  // block-uniform
            const uint32_t d = __ldg(b.unit_domain + u);
            if (next != 0u) __syncthreads();  // every thread is done with the previous descriptor
            static_assert(sizeof(StepArgs) % 4 == 0, "copied in words");
            const uint32_t* src = reinterpret_cast<const uint32_t*>(b.dom + d);
            uint32_t* dst = reinterpret_cast<uint32_t*>(sa);
            for (uint32_t i = threadIdx.x; i < sizeof(StepArgs) / 4; i += blockDim.x) {
                uint32_t v;  // (volatile: kept behind the wait)
                asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(src + i) : "memory");
                dst[i] = v;
            }
            first = __ldg(b.unit_begin + d);
            next = __ldg(b.unit_begin + d + 1);
            __syncthreads();
        }
        return u - first;
    }
};

template <class L, int METHOD, bool F16C, int COLL, int LES, bool LINKS = false>
__global__ void __launch_bounds__(256, (batch_min_blocks<L, COLL, LINKS>())) step_kernel_batch(const BatchArgs b) {
    __shared__ StepArgs sa;
    if (!b.ready) asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t tid = threadIdx.x;
    bool waited = !b.ready;
    for (BatchWalk w(b); w.u < w.end; ++w.u) {
        const uint32_t tile = w.tile(b, &sa);
        const bool general = tile_general(load_byte(sa.tile_near + tile), tid);
        uint2 m = make_uint2(0u, 0u);
        if (general) m = load_masks(b.masks + ((size_t)w.u * kTileCells + tid));
        if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
        waited = true;
        tile_forms<L, METHOD, F16C, COLL, LES, false, LINKS, false>(sa, tile, tid, general, m, nullptr, nullptr, nullptr);
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The same with two cells per thread (double buffer).
template <class L, bool F16C, int COLL, int LES>
__global__ void __launch_bounds__(kPairThreads, (pair_min_blocks<L, LBM_DOUBLE_BUFFER, F16C, COLL, LES, false>()))
    step_kernel_batch_pair(const BatchArgs b) {
    __shared__ StepArgs sa;
    if (!b.ready) asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t t = threadIdx.x;
    bool waited = !b.ready;
    for (BatchWalk w(b); w.u < w.end; ++w.u) {
        const uint32_t tile = w.tile(b, &sa);
        PairMasks pm;
        pm.load<false>(load_byte(sa.tile_near + tile), b.masks + (size_t)w.u * kTileCells, 0u, t);
        if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
        waited = true;
        pair_step<L, LBM_DOUBLE_BUFFER, F16C, COLL, LES, false, false>(sa, tile, t, pm);
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// warp_near bit of warp box i (unit i / 8, warp i % 8) from the box summaries of its domain
// (one thread per box; 0 past the last box).
__device__ __forceinline__ uint32_t batch_near_box(const BatchArgs& b, uint32_t i, const uint8_t* box_sum) {
    const uint32_t u = i / kTileWarps;
    if (u >= b.total_units) return 0u;
    const uint32_t d = find_domain(b.unit_begin, b.ndom, u);
    const uint32_t first = b.unit_begin[d];
    return warp_near(box_sum + (size_t)first * kTileWarps, b.dom[d].lay, u - first, i % kTileWarps);
}

// Brings the summary of warp box `box` of the batch (unit box / 8) up to date (update_box_summary;
// flags_seen and box_sum hold 32 cells and one byte per box of the batch).  One thread per box.
__device__ __forceinline__ void batch_box_summary(const BatchArgs& b, uint32_t box, uint8_t* box_sum,
                                                  uint8_t* flags_seen, uint32_t* changed, uint32_t gen, int force) {
    const uint32_t u = box / kTileWarps;
    if (u >= b.total_units) return;
    const uint32_t d = find_domain(b.unit_begin, b.ndom, u);
    const uint32_t first = b.unit_begin[d];
    const StepArgs& a = b.dom[d];
    const uint32_t lb = box - first * kTileWarps;  // box index within the domain
    update_box_summary(a.flags, lb, flags_seen + (size_t)first * kTileCells, box_sum + (size_t)first * kTileWarps, a.lay,
                       changed, gen, force);
}

struct BatchLinkArgs {
    const StepArgs* dom;   // descriptors of the step that just ran: f_out is the lattice to fix
    const int32_t* domain;
    const int32_t* ids;
    const int32_t* dirs;
    const float* dists;
    float* force;
    int64_t n;
    float q_clamp;
    int32_t bouzidi, compute_force, ddf;
};

// linkwise_bounceback_kernel (src/lbm/geometry/interpolated_BB.mojo:46-141) over the links of all
// domains: each link carries its domain, and works on that domain's freshly written lattice.
template <class L, bool F16C>
__global__ void link_kernel_batch(const BatchLinkArgs b) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= b.n) return;
    const StepArgs& a = b.dom[b.domain[t]];
    LinkArgs la;
    la.lay = a.lay;
    la.f = a.f_out;
    la.force = b.force;
    la.ids = b.ids;
    la.dirs = b.dirs;
    la.dists = b.dists;
    la.n = b.n;
    la.q_clamp = b.q_clamp;
    la.bouzidi = b.bouzidi;
    la.compute_force = b.compute_force;
    la.ddf = b.ddf;
    link_one<L, F16C>(la, t);
}

using BatchLaunch = cudaError_t (*)(const BatchArgs&, cudaStream_t);

inline uint32_t batch_grid(const BatchArgs& b) { return (b.total_units + b.per_cta - 1u) / b.per_cta; }

template <class L, int METHOD, bool F16C, int COLL, int LES>
cudaError_t launch_step_batch(const BatchArgs& b, cudaStream_t s) {
    if (b.total_units == 0) return cudaSuccess;
    return launch_pdl(step_kernel_batch<L, METHOD, F16C, COLL, LES, false>, batch_grid(b), kTileCells, s, b);
}
// The batched step with the links fused in (lbm_batch_set_link_mode, double buffer).
template <class L, int METHOD, bool F16C, int COLL, int LES>
cudaError_t launch_step_batch_links(const BatchArgs& b, cudaStream_t s) {
    if (b.total_units == 0) return cudaSuccess;
    return launch_pdl(step_kernel_batch<L, METHOD, F16C, COLL, LES, true>, batch_grid(b), kTileCells, s, b);
}
// Two cells per thread (double buffer).
template <class L, int METHOD, bool F16C, int COLL, int LES>
cudaError_t launch_step_batch_pair(const BatchArgs& b, cudaStream_t s) {
    static_assert(METHOD == LBM_DOUBLE_BUFFER, "double buffer");
    if (b.total_units == 0) return cudaSuccess;
    return launch_pdl(step_kernel_batch_pair<L, F16C, COLL, LES>, batch_grid(b), kPairThreads, s, b);
}

}  // namespace lbm
