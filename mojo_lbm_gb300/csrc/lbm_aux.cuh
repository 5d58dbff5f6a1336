// Auxiliary kernels around the step: float64 conservation reductions, link-wise interpolated
// bounce-back, momentum-exchange drag (initial state and macroscopic outputs: lbm_fields.cuh).
#pragma once

#include "lbm_fields.cuh"

namespace lbm {

template <class L>
__device__ __forceinline__ Cell decode_cell(const LayoutDesc& lay, uint32_t n, Nbr& nb) {
    Cell c;
    c.n = n;
    c.tile = lay.d_T.div(n);
    c.loc = n - c.tile * lay.T;
    const uint32_t lyz = lay.d_tx.div(c.loc);
    c.lx = c.loc - lyz * (uint32_t)lay.tx;
    c.lz = lay.d_ty.div(lyz);
    c.ly = lyz - c.lz * (uint32_t)lay.ty;
    const uint32_t byz = lay.d_ntx.div(c.tile);
    c.bx = c.tile - byz * (uint32_t)lay.ntx;
    c.bz = lay.d_nty.div(byz);
    c.by = byz - c.bz * (uint32_t)lay.nty;
    c.x = (int32_t)(c.bx * lay.tx + c.lx);
    c.y = (int32_t)(c.by * lay.ty + c.ly);
    c.z = (int32_t)(c.bz * lay.tz + c.lz);
    c.r = ((uint32_t)c.x * (uint32_t)lay.ny + (uint32_t)c.y) * (uint32_t)lay.nz + (uint32_t)c.z;
    cell_nbr<L>(lay, c, nb);
    return c;
}

// Post-collision populations a cell owns after the last completed step, before streaming:
// its own slots (double buffer) or the slots esoteric_pull_store_f_vec wrote them to
// (src/lbm/kernels/ops/load_and_store.mojo:89-159).
template <class L, bool F16C, bool ESO>
__device__ __forceinline__ void gather_post(const typename Pop<F16C>::T* f, const LayoutDesc& lay, const Cell& c,
                                            const Nbr& nb, bool after_odd, float (&out)[L::Q]) {
    using P = Pop<F16C>;
    constexpr int Q = L::Q;
    const uint32_t T = lay.T;
    const uint64_t TQ = (uint64_t)T * Q;
    const uint64_t own = c.loc + TQ * c.tile;
    if constexpr (!ESO) {
        static_for<0, Q>([&](auto qc) { out[qc.value] = P::ld(f + own + (uint64_t)T * qc.value); });
    } else {
        out[0] = P::ld(f + own);
        static_for<1, Q - 1, 2>([&](auto qc) {
            constexpr int pos = qc.value, neg = pos + 1;
            constexpr int sx = L::c(pos, 0), sy = L::c(pos, 1), sz = L::c(pos, 2);
            const uint64_t nbase = nb.template loc<sx, sy, sz>() + TQ * nb.template til<sx, sy, sz>();
            out[pos] = P::ld(f + nbase + (uint64_t)T * (after_odd ? pos : neg));
            out[neg] = P::ld(f + own + (uint64_t)T * (after_odd ? neg : pos));
        });
    }
}

// ---- float64 reductions ---------------------------------------------------------------------
// Deterministic two-pass sums: a fixed grid of kReduceBlocks blocks writes one partial per block
// into scratch, and one block adds the partials in a fixed order.
constexpr int kReduceBlocks = 1024;
constexpr int kReduceThreads = 256;
constexpr int kReduceWidth = 4;

template <int W>
__device__ __forceinline__ void block_sum_store(double (&v)[W], double* dst) {
    __shared__ double sm[kReduceThreads / 32][W];
    static_for<0, W>([&](auto kc) {
        double x = v[kc.value];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        v[kc.value] = x;
    });
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) static_for<0, W>([&](auto kc) { sm[warp][kc.value] = v[kc.value]; });
    __syncthreads();
    if (threadIdx.x < 32) {
        static_for<0, W>([&](auto kc) {
            double x = (lane < (int)(blockDim.x >> 5)) ? sm[lane][kc.value] : 0.0;
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            if (lane == 0) dst[kc.value] = x;
        });
    }
}

// Mass and momentum of one cell's populations without float64 arithmetic in the common case: this GPU
// runs float64 at about 1/64 of its float32 rate, and the 19 conversions and 49 additions a D3Q19 cell
// needs in float64 took 2.35 ms on 256^3 cells (the populations are read in 0.19 ms); this form
// takes 0.265 ms.
// Each population is split exactly against two fixed grids (adding and subtracting 1.5 * 2^k rounds to
// a multiple of 2^(k - 23)): f = h + m + l with h a multiple of 2^-21, m of 2^-41 and |l| <= 2^-42.  While
// sum |f| < 2 a cell's sums of h are exact in float32, and so are those of m: |m| <= 2^-22, 27 of which
// are 27 * 2^19 units of 2^-41, below 2^24 (with units of 2^-42 the sums of 17 or more could round).  Both
// pass as integers into 32-bit accumulators, which hold them exactly for kMassFlush cells (27 * 2^25 <
// 2^31); only the sums of l round, in float32 and at 2^-56 or below (64 cells of 27 sum to less than
// 2^-31), where float64 holds a sum of order 1 to 2^-53.  A cell with sum |f| of
// 2 or more, NaN, or so small that float64's relative precision would beat those absolute errors
// (0 < sum |f| < 2^-10) is added in float64.
constexpr int kMassFlush = 64;

struct MassSum {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};  // mass, momentum
    int32_t hi[4] = {0, 0, 0, 0}, mid[4] = {0, 0, 0, 0};
    float lo[4] = {0.f, 0.f, 0.f, 0.f};
    int32_t shifted = 0, pending = 0;      // DDF-shifted cells (1 each), cells since the last flush

    template <int D>
    __device__ __forceinline__ void flush() {
        static_for<0, D + 1>([&](auto kc) {
            constexpr int k = kc.value;
            acc[k] += (double)hi[k] * 0x1p-21 + ((double)mid[k] * 0x1p-41 + (double)lo[k]);
            hi[k] = mid[k] = 0;
            lo[k] = 0.f;
        });
        acc[0] += (double)shifted;
        shifted = pending = 0;
    }

    template <class L>
    __device__ __forceinline__ void add(const float (&f)[L::Q], bool ddf) {
        constexpr int Q = L::Q, D = L::D;
        float size = 0.f;
        static_for<0, Q>([&](auto qc) { size += fabsf(f[qc.value]); });
        if (!(size < 2.f) || (size < 0x1p-10f && size > 0.f)) {
            double rho = ddf ? 1.0 : 0.0, m[3] = {0.0, 0.0, 0.0};
            static_for<0, Q>([&](auto qc) {
                constexpr int q = qc.value;
                rho += (double)f[q];
                static_for<0, D>([&](auto dc) {
                    constexpr int d = dc.value;
                    if constexpr (L::c(q, d) > 0) m[d] += (double)f[q];
                    else if constexpr (L::c(q, d) < 0) m[d] -= (double)f[q];
                });
            });
            acc[0] += rho;
            static_for<0, D>([&](auto dc) { acc[1 + dc.value] += m[dc.value]; });
            return;
        }
        float H[4] = {0.f, 0.f, 0.f, 0.f}, M[4] = {0.f, 0.f, 0.f, 0.f}, R[4] = {0.f, 0.f, 0.f, 0.f};
        static_for<0, Q>([&](auto qc) {
            constexpr int q = qc.value;
            constexpr float k1 = 6.f, k2 = 1.5f * 0x1p-18f;  // multiples of 2^-21 and of 2^-41
            const float h = (f[q] + k1) - k1, r = f[q] - h;
            const float m = (r + k2) - k2, l = r - m;
            H[0] += h;
            M[0] += m;
            R[0] += l;
            static_for<0, D>([&](auto dc) {
                constexpr int d = dc.value;
                if constexpr (L::c(q, d) > 0) { H[1 + d] += h; M[1 + d] += m; R[1 + d] += l; }
                else if constexpr (L::c(q, d) < 0) { H[1 + d] -= h; M[1 + d] -= m; R[1 + d] -= l; }
            });
        });
        static_for<0, D + 1>([&](auto kc) {
            constexpr int k = kc.value;
            hi[k] += __float2int_rn(H[k] * 0x1p21f);
            mid[k] += __float2int_rn(M[k] * 0x1p41f);
            lo[k] += R[k];
        });
        shifted += ddf ? 1 : 0;
        if (++pending == kMassFlush) flush<D>();
    }
};

struct MassArgs {
    LayoutDesc lay;
    const void* f;
    const uint8_t* flags;
    double* partial;  // kReduceBlocks * 4
    int32_t ddf, even;
};

// Mass and momentum of the post-collision populations of every cell the step updates
// (not SOLID, not EXCLUDE); `even` carries after_odd_step.
template <class L, bool F16C, bool ESO>
__global__ void __launch_bounds__(kReduceThreads) mass_partial_kernel(const MassArgs a) {
    using S = typename Pop<F16C>::T;
    MassSum sum;
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < a.lay.ncells; n += gridDim.x * blockDim.x) {
        const uint8_t flag = a.flags[n];
        if ((flag & 0x0F) == LBM_FLAG_SOLID || (flag & LBM_FLAG_EXCLUDE)) continue;
        Nbr nb;
        const Cell c = decode_cell<L>(a.lay, n, nb);
        float f[L::Q];
        gather_post<L, F16C, ESO>((const S*)a.f, a.lay, c, nb, a.even != 0, f);
        sum.add<L>(f, a.ddf != 0);
    }
    sum.flush<L::D>();
    block_sum_store<4>(sum.acc, a.partial + (size_t)blockIdx.x * 4);
}

// Adds `nparts` partials of width W in a fixed order; one block.
template <int W>
__global__ void __launch_bounds__(kReduceThreads) final_sum_kernel(const double* partial, int nparts, double* out) {
    double acc[W];
    static_for<0, W>([&](auto kc) { acc[kc.value] = 0.0; });
    for (int i = threadIdx.x; i < nparts; i += blockDim.x)
        static_for<0, W>([&](auto kc) { acc[kc.value] += partial[(size_t)i * W + kc.value]; });
    block_sum_store<W>(acc, out);
}

// Column sums of an n x D float array (link fastest), partials of width 4.
static __global__ void __launch_bounds__(kReduceThreads) colsum_partial_kernel(const float* v, int64_t n, int D,
                                                                        double* partial) {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        acc[0] += (double)v[i];
        acc[1] += (double)v[i + n];
        if (D == 3) acc[2] += (double)v[i + 2 * n];
    }
    block_sum_store<4>(acc, partial + (size_t)blockIdx.x * 4);
}

// ---- interpolated bounce-back --------------------------------------------------------------
struct LinkArgs {
    LayoutDesc lay;
    void* f;
    float* force;
    const int32_t* ids;
    const int32_t* dirs;
    const float* dists;
    int64_t n;
    float q_clamp;
    int32_t bouzidi, compute_force, ddf;
};

// linkwise_bounceback_kernel (src/lbm/geometry/interpolated_BB.mojo:46-141); fluid ids are
// decoded as idx_to_ijk does (:24-43).  Float16C is decoded with use_float16c and the force adds
// the weight under DDF shift (output/drag.mojo:88-93).
template <class L, bool F16C>
__device__ __forceinline__ void link_one(const LinkArgs& a, const int64_t t) {
    using P = Pop<F16C>;
    using S = typename P::T;
    constexpr int Q = L::Q, D = L::D;
    const uint32_t li = (uint32_t)a.ids[t];
    if (li >= a.lay.ncells) return;
    Nbr nb;
    const Cell c = decode_cell<L>(a.lay, li, nb);
    const int i = a.dirs[t];
    if (i < 0 || i >= Q) return;
    const int oi = (i == 0) ? 0 : ((i & 1) ? i + 1 : i - 1);
    const uint32_t T = a.lay.T;
    const uint64_t TQ = (uint64_t)T * Q;
    const uint64_t own = c.loc + TQ * c.tile;
    S* f = (S*)a.f;
    float q = a.dists[t];
    q = q < a.q_clamp ? a.q_clamp : q;
    const float f_into = P::ld_rw(f + own + (uint64_t)T * i);
    float f_bb = f_into;
    if (a.bouzidi) {
        if (q > 0.5f) {
            const float f_out = P::ld_rw(f + own + (uint64_t)T * oi);
            f_bb = 0.5f / q * f_into + (2.f * q - 1.f) / (2.f * q) * f_out;
        } else {
            // x_f - c_i, one of the lattice's neighbour shifts
            uint64_t xff = 0;
            static_for<0, Q>([&](auto qc) {
                constexpr int qq = qc.value;
                constexpr int sx = -L::c(qq, 0), sy = -L::c(qq, 1), sz = -L::c(qq, 2);
                if (qq == i) xff = nb.template loc<sx, sy, sz>() + TQ * nb.template til<sx, sy, sz>();
            });
            const float f_xff = P::ld_rw(f + xff + (uint64_t)T * oi);
            f_bb = 2.f * q * f_into + (1.f - 2.f * q) * f_xff;
        }
        P::st(f + own + (uint64_t)T * i, f_bb);
    }
    if (a.compute_force) {
        float w = 0.f;
        static_for<0, Q>([&](auto qc) { if (qc.value == i) w = wf<L>(qc.value); });
        const float fa = a.ddf ? f_into + w : f_into, fb = a.ddf ? f_bb + w : f_bb;
        static_for<0, D>([&](auto dc) {
            int cd = 0;
            static_for<0, Q>([&](auto qc) { if (qc.value == i) cd = L::c(qc.value, dc.value); });
            a.force[t + a.n * dc.value] = (float)cd * (fa + fb);
        });
    }
}

template <class L, bool F16C>
__global__ void link_kernel(const LinkArgs a) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.n) return;
    link_one<L, F16C>(a, t);
}

struct DragArgs {
    LayoutDesc lay;
    const void* f;
    const uint8_t* flags;
    const int32_t* ids;
    float* force;
    int64_t n;
    int32_t ddf;
};

// calculate_drag_around_object (src/lbm/output/drag.mojo:16-105): push-neighbour flags, raw
// SOLID compare, F = sum 2 f_q c_q (+ weight under DDF shift).
template <class L, bool F16C>
__global__ void drag_kernel(const DragArgs a) {
    using P = Pop<F16C>;
    using S = typename P::T;
    constexpr int Q = L::Q, D = L::D;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.n) return;
    const uint32_t li = (uint32_t)a.ids[t];
    if (li >= a.lay.ncells) return;
    Nbr nb;
    const Cell c = decode_cell<L>(a.lay, li, nb);
    const uint32_t T = a.lay.T;
    const uint64_t own = c.loc + (uint64_t)T * Q * c.tile;
    const S* f = (const S*)a.f;
    float acc[3] = {0.f, 0.f, 0.f};
    static_for<0, Q>([&](auto qc) {
        constexpr int q = qc.value;
        constexpr int sx = L::c(q, 0), sy = L::c(q, 1), sz = L::c(q, 2);
        const uint8_t pf = a.flags[nb.template loc<sx, sy, sz>() + T * nb.template til<sx, sy, sz>()];
        if (pf == LBM_FLAG_SOLID) {
            float fl = P::ld(f + own + (uint64_t)T * q);
            if (a.ddf) fl += wf<L>(q);
            static_for<0, D>([&](auto dc) {
                constexpr int d = dc.value;
                if constexpr (L::c(q, d) > 0) acc[d] += 2.f * fl;
                else if constexpr (L::c(q, d) < 0) acc[d] -= 2.f * fl;
            });
        }
    });
    static_for<0, D>([&](auto dc) { a.force[t + a.n * dc.value] = acc[dc.value]; });
}

}  // namespace lbm
