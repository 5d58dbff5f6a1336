// Kernels between the lattice and the row-major fields (rho, u, Q): initial state and macroscopic
// outputs.
//
// The lattice's tiles run x fastest (src/lbm/layoutstruct.mojo:37-92), the fields z fastest in 3D
// and y fastest in 2D (examples/LDC.mojo:47-48), so a warp that reads 32 consecutive cells of a
// tile would touch 32 sectors of every field.  These kernels work on bricks of 1024 (small grids: 256)
// cells instead: 32 lanes of each warp along x (and y) times 32 (8) planes along the fields' fast axis.  The lattice
// is read plane by plane in its own order, the fields move through shared memory (one padded row of
// fast-axis cells per lane, free of bank conflicts) and leave, or arrive, as whole
// 128-byte lines.  The floor is HBM, Q populations and the fields once each (228 us for rho and u of
// 256^3 D3Q19 float32 cells); what bounds them is the load latency and about 500 instructions a cell.
// Measured there, one thread per cell in tile order before, bricks now: rho and u 1160 -> 391 us, the
// Q-criterion 2112 -> 627 us (452 and 1120 us with the layout decoded per flag byte, 64-bit offsets
// and the gradient weights per derivative).  Few cells, thin grids and tiles of short rows do better with
// one thread per cell and have kernels of that form (by_cell).
#pragma once

#include "lbm_step.cuh"

namespace lbm {

// Decoded cell position, shared by the auxiliary kernels.
struct Cell {
    uint32_t n, loc, tile, lx, ly, lz, bx, by, bz;
    int32_t x, y, z;
    uint32_t r;  // row-major output index (x*ny + y)*nz + z
};

// Neighbour tables of a decoded cell.
template <class L>
__device__ __forceinline__ void cell_nbr(const LayoutDesc& lay, const Cell& c, Nbr& nb) {
    nb.ax.init(c.lx, c.bx, lay.tx, lay.ntx, 1u, 1u);
    nb.ay.init(c.ly, c.by, lay.ty, lay.nty, (uint32_t)lay.tx, (uint32_t)lay.ntx);
    if constexpr (L::D == 3)
        nb.az.init(c.lz, c.bz, lay.tz, lay.ntz, (uint32_t)(lay.tx * lay.ty), (uint32_t)(lay.ntx * lay.nty));
    else {
        nb.az.loc[0] = nb.az.loc[1] = nb.az.loc[2] = 0u;
        nb.az.til[0] = nb.az.til[1] = nb.az.til[2] = 0u;
    }
}

// The bricks of a grid.  A warp's 32 lanes are 2^sbx cells along x times 2^sby along y.  3D: a
// brick has 2^sp planes along z, field row g = lx 2^sby + ly, fast index z.  2D: its planes follow
// each other along y, row g = lx, fast index y (2^(sp + sby) of them).
struct Brick {
    uint32_t sbx, sby;        // sbx + sby = 5
    uint32_t sp, sf;          // log2 of the planes and of a field row's length
    uint32_t nbx, nby, nbz;   // bricks per axis
    uint32_t rx, ry, rz;      // the brick with its one-cell rim
    FastDiv d_tz;
};

// Resident blocks per SM the field kernels are built for: 4 (64 registers, some 30 bytes spilled for
// D3Q19) against 3 took rho and u from 452 to 391 us together with the cheaper addressing; D3Q27 3.
#ifndef LBM_FIELDS_MIN_BLOCKS
#define LBM_FIELDS_MIN_BLOCKS 4
#endif

constexpr uint32_t kBrickThreads = 256;
constexpr uint32_t kBrickPlanes = 32;  // at most
// 1024 cells and one pad word per field row (at most 32 rows)
constexpr uint32_t kBrickField = 32u * kBrickPlanes + 32u;
// flag bytes of a brick with its rim: 34 x 3 x 34 (32 lanes along one axis, 3D) is the largest
constexpr uint32_t kBrickFlags = 3472;

// x extent: the largest power of two up to min(tx, 32) whose last brick of a row is not mostly empty
// (a quarter of the cells at most lie outside the grid), else 8 (or tx's power of two below it): a
// warp then reads runs of 2^sbx consecutive cells of the tile.
// Planes: 32 (whole 128-byte lines of the fields) on grids that give every resident block one such
// brick, else 8, one per warp: on a small grid the number of blocks and the serial planes of a warp
// count, not the width of a store (rho and u of 256^2 D2Q9 cells: 8.5 us with 64 blocks of 32 planes, 6.3
// with 256 blocks of 8).  So do 3D grids of up to 8 planes (512 x 512 x 8: 103 / 81 us, x 12: 136 / 158).
inline Brick make_brick(const LayoutDesc& l, int D) {
    Brick b;
    b.sp = l.ncells >= 1024u * 4u * 152u && (D == 2 || l.nz > 8) ? 5u : 3u;
    uint32_t sx = 0;
    while (sx < 5u && (2u << sx) <= (uint32_t)l.tx) ++sx;
    auto waste = [&](uint32_t s) {
        const uint64_t w = 1ull << s, full = (l.nx + w - 1) / w * w;
        return full * 4 > (uint64_t)l.nx * 5;
    };
    while (sx > 3u && waste(sx)) --sx;
    b.sbx = sx;
    b.sby = 5u - sx;
    const uint32_t ex = 1u << b.sbx, ey = 1u << (D == 3 ? b.sby : b.sby + b.sp), ez = D == 3 ? 1u << b.sp : 1u;
    b.sf = D == 3 ? b.sp : b.sp + b.sby;
    b.nbx = ((uint32_t)l.nx + ex - 1u) / ex;
    b.nby = ((uint32_t)l.ny + ey - 1u) / ey;
    b.nbz = ((uint32_t)l.nz + ez - 1u) / ez;
    b.rx = ex + 2u;
    b.ry = ey + 2u;
    b.rz = D == 3 ? ez + 2u : 1u;
    b.d_tz = FastDiv((uint32_t)l.tz);
    return b;
}

// Does one thread per cell, in tile order, do without bricks?  us per call, cell / brick (D3Q19 float32 where
// nothing else is said):
//   few cells, where a brick's barriers and serial planes count: rho and u of 16^3 6.4 / 6.8, 32^3 6.5 / 8.3, 48^3
//     10.6 / 8.6, D2Q9 64^2 4.4 / 6.3, 256^2 6.3 / 6.3; Q of 24^3 6.5 / 8.4, 40^3 9.3 / 10.0, 48^3 13.5 / 10.6 (the
//     initial state gains nothing: 32^3 4.4 / 4.4, with u and grad 6.6 / 6.3)
//   few planes: rho and u of 512 x 512 x 2 28.9 / 49.5, x 4 55.0 / 64.1, x 6 88.9 / 74.2; in 2D rows of a brick past
//     the grid's end: rho and u of 65536 x 16 D2Q9 22.7 / 24.9, Q of x 40 69.9 / 86.5, initial state of x 4 6.3 / 8.4,
//     x 24 16.7 / 14.6
//   short runs of a warp's cells in the tile, where the stores of the cell's order, or all of it, are the better
//     ones: 128^3 in tiles of 1 x 1 x 1 initial state 160 / 293, in place 197 / 357, rho and u 134 / 188, in place
//     Float16C 112 / 186; 2 x 1 x 1 in place 82 / 198, rho and u 111 / 116; 2 x 2 x 2 initial state 41 / 78, in place 51 / 104
//     (with u and grad 97 / 81 and 113 / 123), rho and u 113 / 87; 8 x 1 x 1 and 4 x 4 x 4 40 / 28
// A 2D lattice on a grid that extends along z has its neighbours in another plane (CellDeltas).
enum FieldOp { kInitOp, kRhoUOp, kQOp };
inline bool by_cell(const LayoutDesc& l, const Brick& b, int D, FieldOp op, bool eso, bool reads = false) {
    const uint32_t tx = (uint32_t)l.tx, ty = (uint32_t)l.ty, wx = 1u << b.sbx, wy = 1u << b.sby;
    const uint32_t run = wx < tx ? wx : tx * (ty < wy ? ty : wy);  // consecutive cells of a tile in a warp
    const uint64_t rows = D == 2 ? (uint64_t)b.nby << (b.sby + b.sp) : 0u, ny = (uint64_t)l.ny;
    if (D == 2 ? l.nz > 1 : l.nz <= 4) return true;
    if (op == kInitOp) return rows > 2u * ny || run == 1u || (run <= 4u && (eso || !reads));
    return l.ncells <= 1u << 16 || rows * 4u > ny * 5u || run <= (op == kRhoUOp ? 2u : 1u);
}

// First cell of brick blockIdx.x.
__device__ __forceinline__ void brick_origin(const Brick& b, int D, int32_t& x0, int32_t& y0, int32_t& z0) {
    const uint32_t k = blockIdx.x, r = k / b.nbx;
    x0 = (int32_t)((k - r * b.nbx) << b.sbx);
    y0 = (int32_t)((r % b.nby) << (D == 3 ? b.sby : b.sby + b.sp));
    z0 = (int32_t)((r / b.nby) << b.sp);
}

__device__ __forceinline__ Cell locate_cell(const LayoutDesc& l, const Brick& b, int32_t x, int32_t y, int32_t z) {
    Cell c;
    c.x = x;
    c.y = y;
    c.z = z;
    c.bx = l.d_tx.div((uint32_t)x);
    c.by = l.d_ty.div((uint32_t)y);
    c.bz = b.d_tz.div((uint32_t)z);
    c.lx = (uint32_t)x - c.bx * (uint32_t)l.tx;
    c.ly = (uint32_t)y - c.by * (uint32_t)l.ty;
    c.lz = (uint32_t)z - c.bz * (uint32_t)l.tz;
    c.loc = c.lx + (uint32_t)l.tx * (c.ly + (uint32_t)l.ty * c.lz);
    c.tile = c.bx + (uint32_t)l.ntx * (c.by + (uint32_t)l.nty * c.bz);
    c.n = c.loc + l.T * c.tile;
    c.r = ((uint32_t)x * (uint32_t)l.ny + (uint32_t)y) * (uint32_t)l.nz + (uint32_t)z;
    return c;
}

// Per plane of a 3D brick and its rim (index 0: the plane below the brick): the plane's part of a
// cell's flag index and of its population offset (periodic; planes past the neighbour of the grid's
// last one are nobody's neighbour and repeat it).
template <class Off>
struct PlaneTable {
    uint32_t n[kBrickPlanes + 2];
    Off own[kBrickPlanes + 2];
};
template <class Off>
__device__ __forceinline__ void fill_planes(const LayoutDesc& l, const Brick& b, int32_t z0, Off TQ, PlaneTable<Off>& t) {
    if (threadIdx.x < (1u << b.sp) + 2u) {
        int32_t z = min(z0 + (int32_t)threadIdx.x - 1, l.nz);
        z = z < 0 ? l.nz - 1 : (z == l.nz ? 0 : z);
        const uint32_t bz = b.d_tz.div((uint32_t)z), lz = (uint32_t)z - bz * (uint32_t)l.tz;
        const uint32_t in = lz * (uint32_t)(l.tx * l.ty), til = bz * (uint32_t)(l.ntx * l.nty);
        t.n[threadIdx.x] = in + l.T * til;
        t.own[threadIdx.x] = (Off)in + TQ * (Off)til;
    }
    __syncthreads();
}

// The flags of the brick and its rim (periodic) into fl[rx + RX (ry + RY rz)] (2D: rz = 0); cells more
// than one past the grid's end are nobody's neighbour and read 0.  Returns (block-wide) whether any
// is not 0.  Each thread keeps one (x, y) of the rim's cross-section (3D) or one x (2D) and walks the
// planes or rows, so the layout is decoded once per thread.
template <int D, class Off>
__device__ __forceinline__ bool stage_brick_flags(const uint8_t* __restrict__ flags, const LayoutDesc& l,
                                                  const Brick& b, int32_t x0, int32_t y0, int32_t z0,
                                                  const PlaneTable<Off>& planes, uint8_t* fl) {
    const uint32_t S = D == 3 ? b.rx * b.ry : b.rx, groups = kBrickThreads / S;
    const uint32_t grp = threadIdx.x / S, s = threadIdx.x - grp * S;
    bool any = false;
    auto col = [&](int32_t v, int32_t n) { return v < 0 ? n - 1 : (v == n ? 0 : v); };
    if (grp < groups) {
        const uint32_t sy = D == 3 ? s / b.rx : 0u, sx = s - sy * b.rx;
        const int32_t x = x0 + (int32_t)sx - 1;
        const uint32_t wx = (uint32_t)col(x, l.nx), bx = l.d_tx.div(wx), nx = wx - bx * (uint32_t)l.tx + l.T * bx;
        if constexpr (D == 3) {
            const int32_t y = y0 + (int32_t)sy - 1;
            const uint32_t wy = (uint32_t)col(y, l.ny), by = l.d_ty.div(wy);
            const uint32_t nxy = nx + (wy - by * (uint32_t)l.ty) * (uint32_t)l.tx + l.T * by * (uint32_t)l.ntx;
            const bool in = x <= l.nx && y <= l.ny;
            const uint32_t last = (uint32_t)min((1 << b.sp) + 1, l.nz - z0 + 1);
            for (uint32_t k = grp; k < (1u << b.sp) + 2u; k += groups) {
                const uint8_t v = in && k <= last ? __ldg(flags + nxy + planes.n[k]) : (uint8_t)0;
                fl[s + S * k] = v;
                any = any || v != 0;
            }
        } else {
            for (uint32_t k = grp; k < b.ry; k += groups) {
                const int32_t y = y0 + (int32_t)k - 1;
                const uint32_t wy = (uint32_t)col(y, l.ny), by = l.d_ty.div(wy);
                uint8_t v = 0;
                if (x <= l.nx && y <= l.ny)
                    v = __ldg(flags + nx + (wy - by * (uint32_t)l.ty) * (uint32_t)l.tx + l.T * by * (uint32_t)l.ntx);
                fl[s + S * k] = v;
                any = any || v != 0;
            }
        }
    }
    return __syncthreads_or(any) != 0;
}

struct RhoUArgs {
    LayoutDesc lay;
    Brick brick;
    const void* f;
    const float* bc;
    const uint8_t* flags;
    float* rho;
    float* u;        // [D][nx][ny][nz]: written by the rho/u pass, read by the Q-criterion pass
    float* q;        // [nx][ny][nz]: Q-criterion output
    float tau;       // Q-criterion: the tau of the strain-rate reconstruction
    int32_t ddf, moving, eqbc, even;
};

// get_velocity_gradient (src/lbm/kernels/utils/finite_difference.mojo:14-90), dx = 1, along one
// axis.  Each neighbour inside the grid gives a one-sided difference over a spacing of 1, or 1/2
// when it is SOLID (raw flag compare), weighted (1 - own spacing / sum of spacings).  A neighbour
// outside the grid gives spacing 0, which gives the other side weight 0: the reference's weighting,
// kept as it is, returns 0 across a non-periodic domain edge.
struct AxisGradient {
    bool vl, vr;
    float kl, kr, lw, rw;  // 1 / spacing and weight of the two sides
    // g: coordinate, n: extent; fm, fp: flags of the two neighbours (those outside the grid unused)
    __device__ __forceinline__ void init(int32_t g, int32_t n, uint8_t fm, uint8_t fp) {
        vl = g - 1 >= 0;
        vr = g + 1 < n;
        const float ldx = !vl ? 0.f : fm == LBM_FLAG_SOLID ? 0.5f : 1.f;
        const float rdx = !vr ? 0.f : fp == LBM_FLAG_SOLID ? 0.5f : 1.f;
        kl = fm == LBM_FLAG_SOLID ? 2.f : 1.f;
        kr = fp == LBM_FLAG_SOLID ? 2.f : 1.f;
        // 1 - ldx / (ldx + rdx): the quotients of the spacings 0, 1/2 and 1
        const float total = ldx + rdx;
        const float frac = !vl ? 0.f : !vr ? 1.f : ldx == rdx ? 0.5f : ldx / total;
        lw = 1.f - frac;
        rw = 1.f - lw;
    }
    // u: the component at the cell, s: the element stride of the axis
    __device__ __forceinline__ float of(const float* u, size_t s) const {
        const float u2 = u[0];
        const float lgrad = vl ? (u2 - *(u - s)) * kl : 0.f;
        const float rgrad = vr ? (u[s] - u2) * kr : 0.f;
        return vl || vr ? rgrad * rw + lgrad * lw : 0.f;
    }
};

// calculate_vorticity (Q_criterion.mojo:26-85) and Vector.norm_squared (sequential sum); u0: the cell's first
// component of the stored velocity.
template <int D>
__device__ __forceinline__ float vorticity_squared(const LayoutDesc& l, const float* u0, const AxisGradient& gx,
                                                   const AxisGradient& gy, const AxisGradient& gz) {
    const size_t N = l.ncells, sx = (size_t)l.ny * (size_t)l.nz, sy = (size_t)l.nz;
    const float *u1 = u0 + N, *u2 = u1 + N;
    float w2 = 0.f;
    if constexpr (D == 2) {
        const float wz = gx.of(u1, sx) - gy.of(u0, sy);
        w2 += wz * wz;
    } else {
        const float wx = gy.of(u2, sy) - gz.of(u1, 1);
        const float wy = gz.of(u0, 1) - gx.of(u2, sx);
        const float wz = gx.of(u1, sx) - gy.of(u0, sy);
        w2 += wx * wx;
        w2 += wy * wy;
        w2 += wz * wz;
    }
    return w2;
}

// Density and velocity of a cell's streamed populations.
template <class L>
__device__ __forceinline__ void cell_moments(const float (&f)[L::Q], bool ddf, float& rho, float (&u)[3]) {
    rho = 0.f;
    static_for<0, L::Q>([&](auto qc) { rho += f[qc.value]; });
    if (ddf) rho += 1.f;
    float mom[3] = {0.f, 0.f, 0.f};
    static_for<0, L::Q>([&](auto qc) {
        constexpr int q = qc.value;
        static_for<0, L::D>([&](auto dc) {
            constexpr int d = dc.value;
            if constexpr (L::c(q, d) > 0) mom[d] += f[q];
            else if constexpr (L::c(q, d) < 0) mom[d] -= f[q];
        });
    });
    u[0] = u[1] = u[2] = 0.f;
    static_for<0, L::D>([&](auto dc) { u[dc.value] = mom[dc.value] / rho; });
}

// get_f_noneq_vec (post_collision False), get_non_eq_second_order_moment, get_strain_rate_tensor and its
// norm (kernels/utils/{equilibrium,moment}.mojo), as collide: |S|^2.
template <class L>
__device__ __forceinline__ float strain_norm_squared(const float (&f)[L::Q], float rho, const float (&u)[3], bool ddf,
                                                     float tau) {
    float uu = 0.f;
    static_for<0, L::D>([&](auto dc) { uu += u[dc.value] * u[dc.value]; });
    float Pi[L::NS];
    static_for<0, L::NS>([&](auto nc) { Pi[nc.value] = 0.f; });
    for_each_feq<L>(rho, u, uu, ddf, [&](auto qc, float e) {
        constexpr int q = decltype(qc)::value;
        const float fn = f[q] - e;
        static_for<0, L::NS>([&](auto nc) {
            constexpr int n = nc.value;
            constexpr int cc = L::c(q, sa<L>(n)) * L::c(q, sb<L>(n));
            if constexpr (cc > 0) Pi[n] += fn;
            else if constexpr (cc < 0) Pi[n] -= fn;
        });
    });
    const float k = -1.f / (2.f * rho * (float)(1.0 / 3.0) * tau);
    float s2 = 0.f;
    static_for<0, L::NS>([&](auto nc) {
        constexpr int n = nc.value;
        const float Sn = Pi[n] * k;
        if constexpr (sa<L>(n) != sb<L>(n)) s2 += (Sn * Sn) * 2.f;
        else s2 += Sn * Sn;
    });
    return s2;
}

// calculate_rho_and_velocity (src/lbm/output/velocity.mojo:25-125): the next step's stream and
// boundary conditions, then density and velocity; SOLID cells (raw compare) report their bc.
// With QCRIT, calculate_Q_criterion (src/lbm/output/Q_criterion.mojo:90-216) instead: the same
// stream and boundary conditions, the strain rate from the non-equilibrium second moment (tau of
// the call), the vorticity from finite differences of the stored velocity a.u, and
// Q = |omega|^2 / 4 - |S|^2 / 2 at every cell whose raw flag is not SOLID (others untouched).
//
// One block per brick.  A brick whose flags, rim included, are all plain FLUID skips the
// neighbour-flag gather; the others gather from the staged bytes.  The velocity gradients of the
// Q-criterion are taken after the block has left its strain norms in shared memory, in the order of
// the fields, so their loads are contiguous too.
template <class L, bool F16C, bool ESO, bool QCRIT, class Off>
__global__ void __launch_bounds__(kBrickThreads, L::Q == 27 ? 3 : LBM_FIELDS_MIN_BLOCKS) rho_u_kernel(const __grid_constant__ RhoUArgs a) {
    using P = Pop<F16C>;
    using S = typename P::T;
    constexpr int Q = L::Q, D = L::D, K = D + 1;
    constexpr int NF = QCRIT ? 1 : D + 1;  // staged fields: |S|^2, or u and rho
    __shared__ float field[NF][kBrickField];
    __shared__ uint8_t fl[kBrickFlags];
    __shared__ PlaneTable<Off> planes;
    const Brick& b = a.brick;
    const uint32_t N = a.lay.ncells, T = a.lay.T;
    const Off oT = (Off)T, TQ = oT * Q;
    int32_t x0, y0, z0;
    brick_origin(b, D, x0, y0, z0);
    if constexpr (D == 3) fill_planes<Off>(a.lay, b, z0, TQ, planes);
    const bool flagged = stage_brick_flags<D, Off>(a.flags, a.lay, b, x0, y0, z0, planes, fl);

    const uint32_t lane = threadIdx.x & 31u;
    const int32_t lx = (int32_t)(lane & ((1u << b.sbx) - 1u)), ly = (int32_t)(lane >> b.sbx);
    const uint32_t sf = b.sf;
    const S* fin = (const S*)a.f;
    const bool ddf = a.ddf != 0;
    const int32_t x = x0 + lx;
    CellDeltas<Off, D> d;
    Off own_xy;  // the cell's population offset without the planes' (3D) or rows' (2D) part
    auto row_deltas = [&](int32_t y) -> Off {
        const uint32_t by = a.lay.d_ty.div((uint32_t)y), iy = (uint32_t)y - by * (uint32_t)a.lay.ty;
        axis_deltas<Off>(iy, (uint32_t)a.lay.ty, by, (uint32_t)a.lay.nty, (Off)a.lay.tx, TQ * (Off)a.lay.ntx, d.y);
        return (Off)iy * (Off)a.lay.tx + TQ * (Off)a.lay.ntx * (Off)by;
    };
    {
        const uint32_t bx = a.lay.d_tx.div((uint32_t)x), ix = (uint32_t)x - bx * (uint32_t)a.lay.tx;
        axis_deltas<Off>(ix, (uint32_t)a.lay.tx, bx, (uint32_t)a.lay.ntx, 1, TQ, d.x);
        own_xy = (Off)ix + TQ * (Off)bx;
        if constexpr (D == 3) own_xy += row_deltas(y0 + ly);
    }
#pragma unroll 1
    for (int32_t p = (int32_t)(threadIdx.x >> 5); p < (1 << b.sp); p += (int32_t)(kBrickThreads / 32u)) {
        const int32_t y = D == 3 ? y0 + ly : y0 + (p << b.sby) + ly, z = D == 3 ? z0 + p : 0;
        if (x >= a.lay.nx || y >= a.lay.ny || z >= a.lay.nz) continue;
        const uint32_t slot = D == 3 ? ((uint32_t)((lx << b.sby) + ly) * ((1u << sf) + 1u) + (uint32_t)p)
                                     : (uint32_t)lx * ((1u << sf) + 1u) + (uint32_t)((p << b.sby) + ly);
        const uint32_t at = (uint32_t)(lx + 1) + b.rx * ((uint32_t)(y - y0 + 1) + (D == 3 ? b.ry * (uint32_t)(p + 1) : 0u));
        if constexpr (D == 3) {
            const Off oz = planes.own[p + 1];
            d.own = own_xy + oz;
            d.z[0] = planes.own[p] - oz;
            d.z[2] = planes.own[p + 2] - oz;
        } else {
            d.own = d.flat = own_xy + row_deltas(y);  // (2D bricks lie in the plane z = 0)
        }
        if (flagged && fl[at] == LBM_FLAG_SOLID) {
            if constexpr (!QCRIT) {
                const Cell c = locate_cell(a.lay, b, x, y, z);
                const uint64_t own_bc = c.loc + (uint64_t)T * K * c.tile;
                static_for<0, D>([&](auto dc) { field[dc.value][slot] = a.bc[own_bc + (uint64_t)T * dc.value]; });
                field[D][slot] = a.bc[own_bc + (uint64_t)T * D];
            }
            continue;
        }

        // ---- stream (the loads do not wait for the flags)
        float f[Q];
        if constexpr (!ESO) {
            static_for<0, Q>([&](auto qc) {
                constexpr int q = qc.value;
                f[q] = P::ld(fin + (d.template at<-L::c(q, 0), -L::c(q, 1), -L::c(q, 2)>() + oT * q));
            });
        } else {
            // slot pos + 1 = neg: the parity folds into two base pointers
            const bool ev = a.even != 0;
            const S* fA = fin + (ev ? 0u : T);
            const S* fB = fin + (ev ? T : 0u);
            f[0] = P::ld(fin + d.own);
            static_for<1, Q - 1, 2>([&](auto qc) {
                constexpr int pos = qc.value, neg = pos + 1;
                f[pos] = P::ld(fA + (d.own + oT * pos));
                f[neg] = P::ld(fB + (d.template at<L::c(pos, 0), L::c(pos, 1), L::c(pos, 2)>() + oT * pos));
            });
        }
        if (flagged) {
            uint32_t raw_solid = 0u, nib_solid = 0u;
            static_for<1, Q>([&](auto qc) {
                constexpr int q = qc.value;
                const int32_t o = -L::c(q, 0) - (int32_t)b.rx * (L::c(q, 1) + (int32_t)b.ry * L::c(q, 2));
                const uint8_t pf = fl[(int32_t)at + o];
                if (pf == LBM_FLAG_SOLID) raw_solid |= 1u << q;
                if ((pf & 0x0F) == LBM_FLAG_SOLID) nib_solid |= 1u << q;
            });
            if constexpr (!ESO) {
                if (raw_solid)
                    static_for<1, Q>([&](auto qc) {
                        constexpr int q = qc.value;
                        if ((raw_solid >> q) & 1u) f[q] = P::ld(fin + (d.own + oT * opp<L>(q)));
                    });
            }
            if (a.moving && nib_solid) {
                Nbr nb;
                cell_nbr<L>(a.lay, locate_cell(a.lay, b, x, y, z), nb);
                const uint64_t TK = (uint64_t)T * K;
                moving_wall<L>(f, nib_solid, a.bc, T, [&](auto qc) -> uint64_t {
                    constexpr int q = decltype(qc)::value;
                    constexpr int sx = -L::c(q, 0), sy = -L::c(q, 1), sz = -L::c(q, 2);
                    return nb.template loc<sx, sy, sz>() + TK * nb.template til<sx, sy, sz>();
                });
            }
            if (a.eqbc && (fl[at] & 0x0F) == LBM_FLAG_EQUILIBRIUM) {
                const Cell c = locate_cell(a.lay, b, x, y, z);
                equilibrium_bc<L>(f, a.bc, c.loc + (uint64_t)T * K * c.tile, T, x, y, z, a.lay, ddf);
            }
        }
        float rho, u[3];
        cell_moments<L>(f, ddf, rho, u);
        if constexpr (!QCRIT) {
            static_for<0, D>([&](auto dc) { field[dc.value][slot] = u[dc.value]; });
            field[D][slot] = rho;
        } else {
            field[0][slot] = strain_norm_squared<L>(f, rho, u, ddf, a.tau);
        }
    }
    __syncthreads();

    // ---- out in the fields' order
#pragma unroll 1
    for (uint32_t i = threadIdx.x; i < (32u << b.sp); i += kBrickThreads) {
        const uint32_t fast = i & ((1u << sf) - 1u), g = i >> sf;
        const int32_t cx = (int32_t)(D == 3 ? g >> b.sby : g);
        const int32_t fx = x0 + cx;
        const int32_t y = y0 + (int32_t)(D == 3 ? g & ((1u << b.sby) - 1u) : fast), z = D == 3 ? z0 + (int32_t)fast : 0;
        if (fx >= a.lay.nx || y >= a.lay.ny || z >= a.lay.nz) continue;
        const uint32_t slot = g * ((1u << sf) + 1u) + fast;
        const uint32_t r = ((uint32_t)fx * (uint32_t)a.lay.ny + (uint32_t)y) * (uint32_t)a.lay.nz + (uint32_t)z;
        if constexpr (!QCRIT) {
            static_for<0, D>([&](auto dc) { a.u[(size_t)N * dc.value + r] = field[dc.value][slot]; });
            a.rho[r] = field[D][slot];
        } else {
            const uint32_t at = (uint32_t)(cx + 1) + b.rx * ((uint32_t)(y - y0 + 1) + (D == 3 ? b.ry * (fast + 1u) : 0u));
            if (fl[at] == LBM_FLAG_SOLID) continue;
            AxisGradient gx, gy, gz;
            gx.init(fx, a.lay.nx, fl[at - 1u], fl[at + 1u]);
            gy.init(y, a.lay.ny, fl[at - b.rx], fl[at + b.rx]);
            if constexpr (D == 3) gz.init(z, a.lay.nz, fl[at - b.rx * b.ry], fl[at + b.rx * b.ry]);
            a.q[r] = 0.25f * vorticity_squared<D>(a.lay, a.u + r, gx, gy, gz) - 0.5f * field[0][slot];
        }
    }
}

// The same, one thread per cell in tile order (by_cell).
template <class L, bool F16C, bool ESO, bool QCRIT, class Off>
__global__ void __launch_bounds__(256) rho_u_cell_kernel(const __grid_constant__ RhoUArgs a) {
    using P = Pop<F16C>;
    using S = typename P::T;
    constexpr int Q = L::Q, D = L::D, K = D + 1;
    const LayoutDesc& l = a.lay;
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x, N = l.ncells, T = l.T;
    if (n >= N) return;
    const AnyCell<L, Off> c(l, n);
    const uint32_t r = c.row(l);
    const uint64_t own_bc = c.loc + (uint64_t)T * K * c.tile;
    const uint8_t flag = a.flags[n];
    if (flag == LBM_FLAG_SOLID) {
        if constexpr (!QCRIT) {
            static_for<0, D>([&](auto dc) { a.u[(size_t)N * dc.value + r] = a.bc[own_bc + (uint64_t)T * dc.value]; });
            a.rho[r] = a.bc[own_bc + (uint64_t)T * D];
        }
        return;
    }
    Nbr nb;
    c.nbr(l, nb);
    [[maybe_unused]] uint32_t any;
    uint2 m = make_uint2(0u, 0u);
    if constexpr (!ESO) m = any_solid_masks<L, false>(a.flags, 0u, l, nb, any);
    [[maybe_unused]] const uint32_t raw_solid = m.x;
    const Off oT = (Off)T;
    const S* fin = (const S*)a.f;
    float f[Q];
    if constexpr (!ESO) {
        static_for<0, Q>([&](auto qc) {
            constexpr int q = qc.value;
            Off o = c.d.template at<-L::c(q, 0), -L::c(q, 1), -L::c(q, 2)>();
            if constexpr (q > 0) {
                if ((raw_solid >> q) & 1u) o = c.d.own + (opp<L>(q) > q ? oT : -oT);  // slot q +- 1
            }
            f[q] = P::ld(fin + (o + oT * q));
        });
    } else {
        const bool ev = a.even != 0;
        const S* fA = fin + (ev ? 0u : T);
        const S* fB = fin + (ev ? T : 0u);
        f[0] = P::ld(fin + c.d.own);
        static_for<1, Q - 1, 2>([&](auto qc) {
            constexpr int pos = qc.value, neg = pos + 1;
            f[pos] = P::ld(fA + (c.d.own + oT * pos));
            f[neg] = P::ld(fB + (c.d.template at<L::c(pos, 0), L::c(pos, 1), L::c(pos, 2)>() + oT * pos));
        });
        if (a.moving) m = any_solid_masks<L, false>(a.flags, 0u, l, nb, any);
    }
    const uint32_t nib_solid = a.moving ? m.y & ~1u : 0u;
    if (nib_solid) {
        const uint64_t TK = (uint64_t)T * K;
        moving_wall<L>(f, nib_solid, a.bc, T, [&](auto qc) -> uint64_t {
            constexpr int q = decltype(qc)::value;
            constexpr int sx = -L::c(q, 0), sy = -L::c(q, 1), sz = -L::c(q, 2);
            return nb.template loc<sx, sy, sz>() + TK * nb.template til<sx, sy, sz>();
        });
    }
    const int32_t x = (int32_t)(c.bx * l.tx + c.lx), y = (int32_t)(c.by * l.ty + c.ly), z = (int32_t)(c.bz * l.tz + c.lz);
    if (a.eqbc && (flag & 0x0F) == LBM_FLAG_EQUILIBRIUM) equilibrium_bc<L>(f, a.bc, own_bc, T, x, y, z, l, a.ddf != 0);
    float rho, u[3];
    cell_moments<L>(f, a.ddf != 0, rho, u);
    if constexpr (!QCRIT) {
        static_for<0, D>([&](auto dc) { a.u[(size_t)N * dc.value + r] = u[dc.value]; });
        a.rho[r] = rho;
    } else {
        const float s2 = strain_norm_squared<L>(f, rho, u, a.ddf != 0, a.tau);
        // the flags of the neighbours in the cell's own plane
        const uint32_t own_z = D == 2 ? c.lz * (uint32_t)(l.tx * l.ty) + T * c.bz * (uint32_t)(l.ntx * l.nty) : 0u;
        auto flag_at = [&](auto sx, auto sy, auto sz) {
            constexpr int X = decltype(sx)::value, Y = decltype(sy)::value, Z = decltype(sz)::value;
            return a.flags[own_z + nb.template loc<X, Y, Z>() + T * nb.template til<X, Y, Z>()];
        };
        constexpr std::integral_constant<int, 0> O{};
        constexpr std::integral_constant<int, 1> up{};
        constexpr std::integral_constant<int, -1> down{};
        AxisGradient gx, gy, gz;
        gx.init(x, l.nx, flag_at(down, O, O), flag_at(up, O, O));
        gy.init(y, l.ny, flag_at(O, down, O), flag_at(O, up, O));
        if constexpr (D == 3) gz.init(z, l.nz, flag_at(O, O, down), flag_at(O, O, up));
        a.q[r] = 0.25f * vorticity_squared<D>(l, a.u + r, gx, gy, gz) - 0.5f * s2;
    }
}

struct InitArgs {
    LayoutDesc lay;
    Brick brick;
    void* f;
    const float* u;     // D * ncells, row-major per component, or null
    const float* grad;  // D*D * ncells, or null
    float rho, tau;
    int32_t ddf, esoteric;
};

// The initial populations of a cell with velocity u and symmetric velocity gradient S_, stored.
template <class L, bool F16C, class Off>
__device__ __forceinline__ void store_initial(const InitArgs& a, typename Pop<F16C>::T* fs, const CellDeltas<Off, L::D>& d,
                                              const float (&u)[3], const float (&S_)[3][3]) {
    using P = Pop<F16C>;
    constexpr int Q = L::Q, D = L::D;
    const Off oT = (Off)a.lay.T;
    float uu = 0.f;
    static_for<0, D>([&](auto dc) { uu += u[dc.value] * u[dc.value]; });
    auto population = [&](auto qc) -> float {
        constexpr int q = decltype(qc)::value;
        float fi = feq<L, q>(a.rho, u, uu, a.ddf != 0);
        if (a.grad) {
            float neq = 0.f;
            static_for<0, D>([&](auto ac) {
                static_for<0, D>([&](auto bc) {
                    constexpr int A = ac.value, B = bc.value;
                    constexpr float Qab = (float)(L::c(q, A) * L::c(q, B)) - (A == B ? (float)(1.0 / 3.0) : 0.f);
                    neq += Qab * S_[A][B];
                });
            });
            neq *= (-wf<L>(q) * a.rho * a.tau * 3.f) * ((a.tau - 1.f) / a.tau);
            fi += neq;
        }
        return fi;
    };
    if (!a.esoteric) {
        static_for<0, Q>([&](auto qc) { P::st(fs + (d.own + oT * qc.value), population(qc)); });
    } else {
        P::st(fs + d.own, population(std::integral_constant<int, 0>{}));
        static_for<1, Q - 1, 2>([&](auto qc) {
            constexpr int pos = qc.value, neg = pos + 1;
            P::st(fs + (d.template at<L::c(pos, 0), L::c(pos, 1), L::c(pos, 2)>() + oT * pos), population(qc));
            P::st(fs + (d.own + oT * neg), population(std::integral_constant<int, neg>{}));
        });
    }
}

// initialize_f_from_func (src/lbm/preprocess/initial_condition.mojo:86-179) with fi_neq
// (:182-234); esoteric pull stores with the odd-step pattern (:172-174).
// One block per brick: u and the symmetric part of grad come in in the fields' order and wait in
// shared memory (38 KB in 3D), then the populations are computed and stored plane by plane in the
// lattice's order.  256^3 D3Q19 float32 with u and grad (2.07 GB, floor 305 us): 1080 us with one
// thread per cell in tile order, 428 us with bricks (at rest, 1.27 GB: 376 and 260 us); bound by the
// arithmetic of the non-equilibrium part (issue-active 68 %).
template <class L, bool F16C, class Off>
__global__ void __launch_bounds__(kBrickThreads) init_kernel(const __grid_constant__ InitArgs a) {
    using P = Pop<F16C>;
    using S = typename P::T;
    constexpr int Q = L::Q, D = L::D, NS = L::NS;
    __shared__ float field[D + NS][kBrickField];
    __shared__ PlaneTable<Off> planes;
    const Brick& b = a.brick;
    const uint32_t N = a.lay.ncells;
    const Off oT = (Off)a.lay.T, TQ = oT * Q;
    int32_t x0, y0, z0;
    brick_origin(b, D, x0, y0, z0);
    if constexpr (D == 3) fill_planes<Off>(a.lay, b, z0, TQ, planes);
    const uint32_t sf = b.sf;
    if (a.u || a.grad) {
#pragma unroll 2
        for (uint32_t i = threadIdx.x; i < (32u << b.sp); i += kBrickThreads) {
            const uint32_t fast = i & ((1u << sf) - 1u), g = i >> sf;
            const int32_t x = x0 + (int32_t)(D == 3 ? g >> b.sby : g);
            const int32_t y = y0 + (int32_t)(D == 3 ? g & ((1u << b.sby) - 1u) : fast), z = D == 3 ? z0 + (int32_t)fast : 0;
            if (x >= a.lay.nx || y >= a.lay.ny || z >= a.lay.nz) continue;
            const uint32_t slot = g * ((1u << sf) + 1u) + fast;
            const uint32_t r = ((uint32_t)x * (uint32_t)a.lay.ny + (uint32_t)y) * (uint32_t)a.lay.nz + (uint32_t)z;
            if (a.u) static_for<0, D>([&](auto dc) { field[dc.value][slot] = __ldg(a.u + (size_t)N * dc.value + r); });
            if (a.grad)
                static_for<0, NS>([&](auto nc) {
                    constexpr int n = nc.value, A = sa<L>(n), B = sb<L>(n);
                    field[D + n][slot] = 0.5f * (__ldg(a.grad + (size_t)N * (A * D + B) + r) +
                                                 __ldg(a.grad + (size_t)N * (B * D + A) + r));
                });
        }
        __syncthreads();
    }

    const uint32_t lane = threadIdx.x & 31u;
    const int32_t lx = (int32_t)(lane & ((1u << b.sbx) - 1u)), ly = (int32_t)(lane >> b.sbx);
    const int32_t x = x0 + lx;
    S* fs = (S*)a.f;
    CellDeltas<Off, D> d;
    Off own_xy;
    auto row_deltas = [&](int32_t y) -> Off {
        const uint32_t by = a.lay.d_ty.div((uint32_t)y), iy = (uint32_t)y - by * (uint32_t)a.lay.ty;
        axis_deltas<Off>(iy, (uint32_t)a.lay.ty, by, (uint32_t)a.lay.nty, (Off)a.lay.tx, TQ * (Off)a.lay.ntx, d.y);
        return (Off)iy * (Off)a.lay.tx + TQ * (Off)a.lay.ntx * (Off)by;
    };
    {
        const uint32_t bx = a.lay.d_tx.div((uint32_t)x), ix = (uint32_t)x - bx * (uint32_t)a.lay.tx;
        axis_deltas<Off>(ix, (uint32_t)a.lay.tx, bx, (uint32_t)a.lay.ntx, 1, TQ, d.x);
        own_xy = (Off)ix + TQ * (Off)bx;
        if constexpr (D == 3) own_xy += row_deltas(y0 + ly);
    }
#pragma unroll 1
    for (int32_t p = (int32_t)(threadIdx.x >> 5); p < (1 << b.sp); p += (int32_t)(kBrickThreads / 32u)) {
        const int32_t y = D == 3 ? y0 + ly : y0 + (p << b.sby) + ly, z = D == 3 ? z0 + p : 0;
        if (x >= a.lay.nx || y >= a.lay.ny || z >= a.lay.nz) continue;
        const uint32_t slot = D == 3 ? ((uint32_t)((lx << b.sby) + ly) * ((1u << sf) + 1u) + (uint32_t)p)
                                     : (uint32_t)lx * ((1u << sf) + 1u) + (uint32_t)((p << b.sby) + ly);
        if constexpr (D == 3) {
            const Off oz = planes.own[p + 1];
            d.own = own_xy + oz;
            d.z[0] = planes.own[p] - oz;
            d.z[2] = planes.own[p + 2] - oz;
        } else {
            d.own = d.flat = own_xy + row_deltas(y);  // (2D bricks lie in the plane z = 0)
        }
        float u[3] = {0.f, 0.f, 0.f};
        if (a.u) static_for<0, D>([&](auto dc) { u[dc.value] = field[dc.value][slot]; });
        float S_[3][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
        if (a.grad)
            static_for<0, NS>([&](auto nc) {
                constexpr int n = nc.value, A = sa<L>(n), B = sb<L>(n);
                S_[A][B] = S_[B][A] = field[D + n][slot];
            });
        store_initial<L, F16C>(a, fs, d, u, S_);
    }
}

// The same, one thread per cell in tile order (by_cell).
template <class L, bool F16C, class Off>
__global__ void __launch_bounds__(256) init_cell_kernel(const __grid_constant__ InitArgs a) {
    constexpr int D = L::D;
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x, N = a.lay.ncells;
    if (n >= N) return;
    const AnyCell<L, Off> c(a.lay, n);
    const uint32_t r = c.row(a.lay);
    float u[3] = {0.f, 0.f, 0.f}, S_[3][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
    if (a.u) static_for<0, D>([&](auto dc) { u[dc.value] = __ldg(a.u + (size_t)N * dc.value + r); });
    if (a.grad)
        static_for<0, L::NS>([&](auto nc) {
            constexpr int k = nc.value, A = sa<L>(k), B = sb<L>(k);
            S_[A][B] = S_[B][A] = 0.5f * (__ldg(a.grad + (size_t)N * (A * D + B) + r) + __ldg(a.grad + (size_t)N * (B * D + A) + r));
        });
    store_initial<L, F16C>(a, (typename Pop<F16C>::T*)a.f, c.d, u, S_);
}

template <class L>
cudaError_t launch_init(const InitArgs& a, bool f16, cudaStream_t s) {
    const bool narrow = offsets32<L>(a.lay);
    const bool cells = by_cell(a.lay, a.brick, L::D, kInitOp, a.esoteric != 0, a.u || a.grad);
    const uint32_t blocks = cells ? (a.lay.ncells - 1u) / 256u + 1u : a.brick.nbx * a.brick.nby * a.brick.nbz;
    auto go = [&](auto f16c, auto off) {
        constexpr bool F = decltype(f16c)::value;
        using Off = decltype(off);
        if (cells) init_cell_kernel<L, F, Off><<<blocks, 256, 0, s>>>(a);
        else init_kernel<L, F, Off><<<blocks, kBrickThreads, 0, s>>>(a);
        return cudaGetLastError();
    };
    if (f16) return narrow ? go(std::true_type{}, int32_t{}) : go(std::true_type{}, int64_t{});
    return narrow ? go(std::false_type{}, int32_t{}) : go(std::false_type{}, int64_t{});
}

// Launches the outputs of one lattice (lbm_fields_*.cu): rho and u, or with qcrit the Q-criterion.
template <class L, bool F16C, bool ESO, bool QCRIT>
cudaError_t launch_rho_u_impl(const RhoUArgs& a, cudaStream_t s) {
    const bool narrow = offsets32<L>(a.lay);
    if (by_cell(a.lay, a.brick, L::D, QCRIT ? kQOp : kRhoUOp, ESO)) {
        const uint32_t blocks = (a.lay.ncells - 1u) / 256u + 1u;
        if (narrow) rho_u_cell_kernel<L, F16C, ESO, QCRIT, int32_t><<<blocks, 256, 0, s>>>(a);
        else rho_u_cell_kernel<L, F16C, ESO, QCRIT, int64_t><<<blocks, 256, 0, s>>>(a);
    } else {
        const uint32_t blocks = a.brick.nbx * a.brick.nby * a.brick.nbz;
        if (narrow) rho_u_kernel<L, F16C, ESO, QCRIT, int32_t><<<blocks, kBrickThreads, 0, s>>>(a);
        else rho_u_kernel<L, F16C, ESO, QCRIT, int64_t><<<blocks, kBrickThreads, 0, s>>>(a);
    }
    return cudaGetLastError();
}
template <class L>
cudaError_t launch_rho_u(const RhoUArgs& a, bool f16, bool eso, bool qcrit, cudaStream_t s) {
    if (f16) {
        if (eso) return qcrit ? launch_rho_u_impl<L, true, true, true>(a, s) : launch_rho_u_impl<L, true, true, false>(a, s);
        return qcrit ? launch_rho_u_impl<L, true, false, true>(a, s) : launch_rho_u_impl<L, true, false, false>(a, s);
    }
    if (eso) return qcrit ? launch_rho_u_impl<L, false, true, true>(a, s) : launch_rho_u_impl<L, false, true, false>(a, s);
    return qcrit ? launch_rho_u_impl<L, false, false, true>(a, s) : launch_rho_u_impl<L, false, false, false>(a, s);
}

}  // namespace lbm
