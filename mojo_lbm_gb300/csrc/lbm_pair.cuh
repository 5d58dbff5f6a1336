// The cell-pair form of the block-per-tile step: one thread streams and collides two cells that are
// neighbours along x, so that half of the population traffic moves as 64-bit (float32) or 32-bit
// (Float16C) words, half of the neighbour address arithmetic is shared, and the fast arithmetic runs as
// packed two-value instructions.  Double buffer, and in the fast arithmetic also the in-place method.
//
// A 256-cell tile with power-of-two sides and tx >= 2 is one CTA of 128 threads; thread t owns the
// cells tA = 2t and tB = 2t + 1 of the tile, which sit at x_A (even) and x_A + 1 of one tile row.
// For a direction q the pull source of A is x_A - c_q and that of B is one cell further along x:
//   c_q.x =  0: the two sources are the aligned pair (x_A, x_A + 1) of the source row: one word;
//   c_q.x = +1: A from x_A - 1 (the west tile's last cell when x_A = 0), B from x_A;
//   c_q.x = -1: A from x_A + 1, B from x_A + 2 (the east tile's first cell when x_A + 2 = tx).
// The source row (y - c_q.y, z - c_q.z) is shared by up to three directions, so a D3Q19 pair
// computes 9 row addresses and 10 west/east addresses for its 38 populations.  Every own-cell
// access (the stores, the mid-grid bounce-back reload) is one word per direction.  In place, the own
// slots are words and the slots at x + c_q (the positive direction of each pair) are found the same
// way, for the loads and for the stores.
//
// Everything else is the per-cell code of tile_step (lbm_step.cuh), applied to A and B in turn or to
// both at once with the same operations: the results are those of step_kernel_tile bit for bit (the
// exact build) or word for word (the fast build).  A warp owns the warp boxes 2w and 2w + 1 of the
// tile (its 64 cells); it takes the all-fluid branch when both boxes' mask bits are clear, otherwise the pair
// body's general form or two passes of the per-cell body (pair_by_cell).
//
// Requirements: the population buffers 8-byte aligned (the host falls back to the per-cell kernel
// otherwise), tx >= 2, no learned closure.
#pragma once

#include "lbm_step.cuh"

namespace lbm {

constexpr uint32_t kPairThreads = kTileCells / 2;

// Word access to the aligned pair (A, B) of one population slot.
template <bool F16C, bool SCALED> struct PairWord;
template <bool SCALED> struct PairWord<false, SCALED> {
    static __device__ __forceinline__ void ld(const float* p, float& a, float& b) {
        const float2 v = __ldg(reinterpret_cast<const float2*>(p));
        a = v.x;
        b = v.y;
    }
    static __device__ __forceinline__ void ld_rw(const float* p, float& a, float& b) {
        const float2 v = *reinterpret_cast<const float2*>(p);
        a = v.x;
        b = v.y;
    }
    static __device__ __forceinline__ void st(float* p, float a, float b) {
        *reinterpret_cast<float2*>(p) = make_float2(a, b);
    }
};
template <bool SCALED> struct PairWord<true, SCALED> {
    // low half: A's code, high half: B's (little-endian)
    static __device__ __forceinline__ void decode(uint32_t w, float& a, float& b) {
        if constexpr (SCALED) {
            // an arithmetic shift by 4 puts a code's magnitude at bits 12..26 and leaves its sign at 31
            a = as_f32((uint32_t)((int32_t)(w << 16) >> 4) & 0x87FFF000u);
            b = as_f32((uint32_t)((int32_t)w >> 4) & 0x87FFF000u);
        } else {
            a = f16c_decode_sx((int32_t)(w << 16) >> 16);
            b = f16c_decode_sx((int32_t)w >> 16);
        }
    }
    static __device__ __forceinline__ void ld(const uint16_t* p, float& a, float& b) {
        decode(__ldg(reinterpret_cast<const uint32_t*>(p)), a, b);
    }
    static __device__ __forceinline__ void ld_rw(const uint16_t* p, float& a, float& b) {
        decode(*reinterpret_cast<const uint32_t*>(p), a, b);
    }
    static __device__ __forceinline__ void st(uint16_t* p, float a, float b) {
        uint32_t w;
        if constexpr (SCALED) {
            // f16c_encode_scaled of both: the two magnitudes side by side, then both signs (the top
            // bytes of a and b moved to bytes 1 and 3, bits 15 and 31 kept) in one bitwise select
            constexpr float kSatScaled = 0x1.ffdp-112f;
            const uint32_t ma = round_shift12(as_u32(fminf(fabsf(a), kSatScaled)));
            const uint32_t mb = round_shift12(as_u32(fminf(fabsf(b), kSatScaled)));
            const uint32_t signs = __byte_perm(as_u32(a), as_u32(b), 0x7430);
            w = (signs & 0x80008000u) | __byte_perm(ma, mb, 0x5410);
        } else {
            w = __byte_perm(f16c_encode(a), f16c_encode(b), 0x5410);
        }
        *reinterpret_cast<uint32_t*>(p) = w;
    }
};

// Element deltas of the pair: y and z as in tile_deltas (shifts -1, 0, +1), and along x the
// delta from A to x_A - 1 and from B to x_B + 1 (-1 / +1 inside the tile, the periodic jump to
// the neighbouring tile at its edge).
template <int D>
__device__ __forceinline__ void pair_deltas(const StepArgs& a, uint32_t bx, uint32_t by, uint32_t bz, uint32_t lxA,
                                            uint32_t ly, uint32_t lz, int32_t TQ, int32_t& dxm, int32_t& dxp,
                                            int32_t (&dy)[3], int32_t (&dz)[3]) {
    const int32_t tx = a.lay.tx, ty = a.lay.ty, tz = a.lay.tz, txy = tx * ty;
    const int32_t ntx = a.lay.ntx, nty = a.lay.nty, ntz = a.lay.ntz;
    const int32_t jxm = bx > 0 ? -1 : ntx - 1, jxp = (int32_t)bx + 1 < ntx ? 1 : 1 - ntx;
    const int32_t jym = by > 0 ? -ntx : (nty - 1) * ntx, jyp = (int32_t)by + 1 < nty ? ntx : (1 - nty) * ntx;
    dxm = lxA > 0 ? -1 : (tx - 1) + TQ * jxm;
    dxp = (int32_t)lxA + 2 < tx ? 1 : (1 - tx) + TQ * jxp;
    dy[1] = dz[1] = 0;
    dy[0] = ly > 0 ? -tx : (ty - 1) * tx + TQ * jym;
    dy[2] = (int32_t)ly + 1 < ty ? tx : (1 - ty) * tx + TQ * jyp;
    if constexpr (D == 3) {
        const int32_t ntxy = ntx * nty;
        const int32_t jzm = bz > 0 ? -ntxy : (ntz - 1) * ntxy, jzp = (int32_t)bz + 1 < ntz ? ntxy : (1 - ntz) * ntxy;
        dz[0] = lz > 0 ? -txy : (tz - 1) * txy + TQ * jzm;
        dz[2] = (int32_t)lz + 1 < tz ? txy : (1 - tz) * txy + TQ * jzp;
    } else {
        dz[0] = dz[2] = 0;
    }
}

// Does the fast arithmetic work on both cells at once (F2)?  In lockstep they need the registers of two
// collisions at a time: TRT in double buffer or on D3Q19, and Smagorinsky SRT on D3Q19, spill at any
// occupancy that pays and take the cells in turn.  Float16C, us a step, packed / in turn: 160^3 D3Q19
// double buffer SRT 66.5 / 70.5, SRT with LES 81.7 / 80.1, TRT 81.4 / 77.3; 2048^2 D2Q9 double buffer SRT
// 36.5 / 38.5, SRT with LES 40.6 / 44.9, TRT 39.6 / 38.7; 144^3 D3Q27 in place, SRT with LES 93.9 / 100.1,
// TRT 86.7 / 90.7; 2048^2 D2Q9 in place TRT 32.3 / 35.4.
template <class L, int METHOD, int COLL, int LES, bool FAST>
constexpr bool pair_packed() {
    if (!FAST) return false;
    if (L::Q == 19) return COLL != LBM_TRT && (!LES || COLL != LBM_SRT);
    return COLL != LBM_TRT || METHOD == LBM_ESOTERIC_PULL;
}

// The two cells of one thread.  GENERAL = false is the all-fluid form (the warp's two boxes hold
// no flag and pull from no flagged cell): no flag is read, both cells are active and the code is
// straight-line from the loads to the stores, so the scheduler interleaves the two collisions.
// GENERAL = true takes the masks of both cells, m (x, y of A, z, w of B; 0 in a box without a flag), and
// handles them as tile_step does.
template <class L, int METHOD, bool F16C, int COLL, int LES, bool FAST, bool GENERAL>
__device__ __forceinline__ void pair_cells(const StepArgs& a, const uint32_t tile, const uint32_t t,
                                           const uint4 m, const uint32_t bx, const uint32_t by,
                                           const uint32_t bz) {
    using P = Pop<F16C>;
    using S = typename P::T;
    constexpr int Q = L::Q, D = L::D, K = D + 1;
    constexpr uint32_t T = kTileCells;
    constexpr bool ESO = METHOD == LBM_ESOTERIC_PULL;
    constexpr bool SCALED = FAST && F16C && !LES && COLL != LBM_KBC;
    using W = PairWord<F16C, SCALED>;
    auto ld = [](const S* p) -> float {
        if constexpr (ESO) {
            if constexpr (SCALED) return P::ld_rw_scaled(p);
            else return P::ld_rw(p);
        } else {
            if constexpr (SCALED) return P::ld_scaled(p);
            else return P::ld(p);
        }
    };
    auto st = [](S* p, float v) {
        if constexpr (SCALED) P::st_scaled(p, v);
        else P::st(p, v);
    };

    const uint32_t tA = 2u * t;         // cell A; B = tA + 1
    const uint32_t nA = tA + T * tile;  // flag offset of A

    uint8_t flagA = 0, flagB = 0;
    bool actA = true, actB = true;
    if constexpr (GENERAL) {
        actA = (m.x & 1u) == 0u;
        actB = (m.z & 1u) == 0u;
        if (!actA && !actB) return;
        if (m.y & 1u) flagA = __ldg(a.flags + nA);
        if (m.w & 1u) flagB = __ldg(a.flags + nA + 1u);
    }

    const uint32_t lxA = tA & a.mx, ly = (tA >> a.shx) & a.my, lz = tA >> a.shxy;
    const int32_t TQ = (int32_t)(T * Q);
    int32_t dxm, dxp, dy[3], dz[3];
    pair_deltas<D>(a, bx, by, bz, lxA, ly, lz, TQ, dxm, dxp, dy, dz);
    const int32_t own = (int32_t)tA + TQ * (int32_t)tile;
    const S* fin = after_wait<S>(a.f_in);
    S* fout = (S*)a.f_out;

    // ---- stream: pull loads of both cells
    float fa[Q], fb[Q];
    // a population slot of both cells at the neighbour (SX, .., ..) of the row `p` (at x_A)
    auto ld2 = [&](const S* p, auto sxc, float& va, float& vb) {
        constexpr int sx = decltype(sxc)::value;
        if constexpr (sx == 0) {
            if constexpr (ESO) W::ld_rw(p, va, vb);
            else W::ld(p, va, vb);
        } else if constexpr (sx < 0) {
            va = ld(p + dxm);
            vb = ld(p);
        } else {
            va = ld(p + 1);
            vb = ld(p + dxp + 1);
        }
    };
    // even: pos from (x, pos), neg from (x + c_pos, neg); odd: pos from (x, neg), neg from
    // (x + c_pos, pos).  Slot pos + 1 = neg, so the parity folds into two base pointers.
    [[maybe_unused]] const bool ev = a.even != 0;
    if constexpr (!ESO) {
        static_for<0, Q>([&](auto qc) {
            constexpr int q = qc.value;
            constexpr int sx = -L::c(q, 0), sy = -L::c(q, 1), sz = -L::c(q, 2);
            // the source row at x_A: one 64-bit address per row (shared by its directions, whose q*T
            // are immediate offsets) and one per x edge
            ld2(fin + (own + dy[sy + 1] + dz[sz + 1]) + (int32_t)(T * q), std::integral_constant<int, sx>{}, fa[q], fb[q]);
        });
    } else {
        const S* finA = fin + (ev ? 0u : T);
        const S* finB = fin + (ev ? T : 0u);
        W::ld_rw(fin + own, fa[0], fb[0]);
        static_for<1, Q - 1, 2>([&](auto qc) {
            constexpr int pos = qc.value, neg = pos + 1;
            constexpr int sx = L::c(pos, 0), sy = L::c(pos, 1), sz = L::c(pos, 2);
            W::ld_rw(finA + own + (int32_t)(T * pos), fa[pos], fb[pos]);
            ld2(finB + (own + dy[sy + 1] + dz[sz + 1]) + (int32_t)(T * pos), std::integral_constant<int, sx>{}, fa[neg], fb[neg]);
        });
    }

    if constexpr (GENERAL && !ESO) {
        // mid-grid bounce-back on a raw SOLID compare (ops/load_and_store.mojo:216); selecting the
        // address before the pull, as the per-cell kernels do, was slower here (393.3 against 389.8 us a
        // step of the 256^3 float32 cavity, 269.9 against 262.1 in Float16C)
        const uint32_t backA = m.x & ~1u, backB = m.z & ~1u;
        if (backA)
            static_for<1, Q>([&](auto qc) {
                constexpr int q = qc.value;
                if ((backA >> q) & 1u) fa[q] = ld(fin + own + (int32_t)(T * opp<L>(q)));
            });
        if (backB)
            static_for<1, Q>([&](auto qc) {
                constexpr int q = qc.value;
                if ((backB >> q) & 1u) fb[q] = ld(fin + own + 1 + (int32_t)(T * opp<L>(q)));
            });
    }

    if constexpr (GENERAL) {
        const uint32_t wallA = m.y & ~1u, wallB = m.w & ~1u;
        if constexpr (!FAST) {
            if (a.moving) {
                add_resting_walls<L>(fa, m.x & ~(m.y | 1u));
                add_resting_walls<L>(fb, m.z & ~(m.w | 1u));
            }
        }
        if (a.moving && (wallA | wallB)) {
            // moving_wall_bc with the bc of each cell's SOLID pull neighbours
            auto wall = [&](float (&f)[Q], uint32_t nib, uint32_t tc) {
                int32_t dc[3][3], dp[3][3];
                tile_deltas<D>(a, bx, by, bz, tc & a.mx, ly, lz, TQ, dc, dp);
                const uint32_t n = tc + T * tile;
                moving_wall<L, SCALED>(f, nib, a.bc, T, [&](auto qc) -> uint64_t {
                    constexpr int q = decltype(qc)::value;
                    constexpr int sx = -L::c(q, 0), sy = -L::c(q, 1), sz = -L::c(q, 2);
                    const uint32_t mm = (uint32_t)((int32_t)n + dc[0][sx + 1] + dc[1][sy + 1] + dc[2][sz + 1]);
                    const uint32_t mt = mm / T;
                    return (uint64_t)(mm - mt * T) + (uint64_t)T * K * mt;
                });
            };
            if (wallA) wall(fa, wallA, tA);
            if (wallB) wall(fb, wallB, tA + 1u);
        }
        if (a.eqbc) {
            const int32_t gx = (int32_t)(bx * (uint32_t)a.lay.tx + lxA), gy = (int32_t)(by * (uint32_t)a.lay.ty + ly),
                          gz = (int32_t)(bz * (uint32_t)a.lay.tz + lz);
            auto eq = [&](float (&f)[Q], uint32_t tc, int32_t x) {
                if constexpr (SCALED) static_for<0, Q>([&](auto qc) { f[qc.value] *= 0x1p112f; });
                equilibrium_bc<L>(f, a.bc, tc + (uint64_t)T * K * tile, T, x, gy, gz, a.lay, a.ddf != 0);
                if constexpr (SCALED) static_for<0, Q>([&](auto qc) { f[qc.value] *= 0x1p-112f; });
            };
            if ((flagA & 0x0F) == LBM_FLAG_EQUILIBRIUM) eq(fa, tA, gx);
            if ((flagB & 0x0F) == LBM_FLAG_EQUILIBRIUM) eq(fb, tA + 1u, gx + 1);
        }
    }

    // ---- collide: both cells at once by packed instructions (a cell that is not stepped goes along and is
    // not stored), or one after the other
    float* bcA = a.bc + (tA + (uint64_t)T * K * tile);
    if constexpr (pair_packed<L, METHOD, COLL, LES, FAST>()) {
        F2 f[Q];
        static_for<0, Q>([&](auto qc) { f[qc.value] = F2{fa[qc.value], fb[qc.value]}; });
        collide_fast_v<L, COLL, LES, SCALED, F2>(f, a, [&](F2 rho, const F2* u) {
            if constexpr (GENERAL) {
                auto keep = [&](bool act, uint32_t flag, float* bc, float r, auto&& comp) {
                    if (act && a.cap_rho && (flag & LBM_FLAG_CAPTURE_DENSITY)) bc[(size_t)T * D] = r;
                    if (act && a.cap_u && (flag & LBM_FLAG_CAPTURE_VELOCITY))
                        static_for<0, D>([&](auto dc) { bc[(size_t)T * dc.value] = comp(dc); });
                };
                keep(actA, flagA, bcA, rho.x, [&](auto dc) { return u[decltype(dc)::value].x; });
                keep(actB, flagB, bcA + 1, rho.y, [&](auto dc) { return u[decltype(dc)::value].y; });
            }
        });
        static_for<0, Q>([&](auto qc) {
            fa[qc.value] = f[qc.value].x;
            fb[qc.value] = f[qc.value].y;
        });
    } else if constexpr (FAST) {
        if (!GENERAL || actA) collide_fast<L, COLL, LES, SCALED>(fa, a, bcA, T, flagA);
        if (!GENERAL || actB) collide_fast<L, COLL, LES, SCALED>(fb, a, bcA + 1, T, flagB);
    } else {
        if (!GENERAL || actA) collide<L, COLL, LES>(fa, a.tau, a, bcA, T, flagA);
        if (!GENERAL || actB) collide<L, COLL, LES>(fb, a.tau, a, bcA + 1, T, flagB);
    }

    // ---- store: one word per direction, or the active cell's half (mode 0: both, 1: A, 2: B)
    auto store = [&](auto mode) {
        constexpr int MODE = decltype(mode)::value;
        auto st2 = [&](S* p, auto sxc, float va, float vb) {
            constexpr int sx = decltype(sxc)::value;
            if constexpr (sx == 0 && MODE == 0) {
                W::st(p, va, vb);
            } else {
                if constexpr (MODE != 2) st(sx == 0 ? p : sx < 0 ? p + dxm : p + 1, va);
                if constexpr (MODE != 1) st(sx == 0 ? p + 1 : sx < 0 ? p : p + dxp + 1, vb);
            }
        };
        constexpr std::integral_constant<int, 0> here{};
        if constexpr (!ESO) {
            static_for<0, Q>([&](auto qc) { st2(fout + own + (int32_t)(T * qc.value), here, fa[qc.value], fb[qc.value]); });
        } else {
            // the slots that were loaded, pos and neg exchanged
            S* foA = fout + (ev ? 0u : T);
            S* foB = fout + (ev ? T : 0u);
            st2(fout + own, here, fa[0], fb[0]);
            static_for<1, Q - 1, 2>([&](auto qc) {
                constexpr int pos = qc.value, neg = pos + 1;
                constexpr int sx = L::c(pos, 0), sy = L::c(pos, 1), sz = L::c(pos, 2);
                st2(foB + (own + dy[sy + 1] + dz[sz + 1]) + (int32_t)(T * pos), std::integral_constant<int, sx>{}, fa[pos], fb[pos]);
                st2(foA + own + (int32_t)(T * pos), here, fa[neg], fb[neg]);
            });
        }
    };
    if (!GENERAL || (actA && actB)) store(std::integral_constant<int, 0>{});
    else if (actA) store(std::integral_constant<int, 1>{});
    else store(std::integral_constant<int, 2>{});
}

// Does a warp with a flag in or next to its 64 cells step them by two passes of the per-cell body (tile_cell,
// which folds the bounce-back into the pull addresses), instead of the pair body's general form (which pulls
// both cells by words and then reloads direction by direction)?  us a step, general form / by cell:
//   exact double buffer   192^3 D3Q19 cavity SRT 164.0 / 162.7, Float16C 161.3 / 147.6, TRT 176.6 / 170.7, RLBM
//                         171.7 / 163.5, Float16C with LES 238 / 213; 1024^2 D2Q9 11.8 / 11.0, TRT 13.7 / 12.8
//   fast double buffer    1024^2 D2Q9 10.75 / 9.46, Float16C 9.42 / 8.85; D3Q19 Float16C cavity 128^3 37.5 / 36.0,
//                         256^3 240.7 / 236.3 (a periodic box without a flag 29.7 / 30.1: the compiler's code for
//                         the pairs differs), TRT 44.0 / 40.1; not RLBM (38.3 / 38.0, box 30.8 / 31.7) and SRT
//                         with LES (45.9 / 43.7, box 38.6 / 40.5)
//   in place              256^3 D3Q27 Float16C TRT with LES 491 / 456, RLBM 430 / 421, SRT 421.5 / 409.9; not SRT
//                         with LES (448 / 472) nor the other lattices (192^3 D3Q19 112.9 / 120.1, D2Q9 9.87 / 9.97)
// KBC keeps the general form (256^3 D3Q19 in place 387 / 396), and so does the batch, whose narrow domains have
// such warps everywhere (128 channels 190 / 202).
template <class L, int METHOD, bool F16C, int COLL, int LES, bool FAST>
constexpr bool pair_by_cell() {
    if (COLL == LBM_KBC) return false;
    if (METHOD == LBM_ESOTERIC_PULL) return L::Q == 27 && !(COLL == LBM_SRT && LES);
    return !FAST || L::Q != 19 || COLL == LBM_TRT || (COLL == LBM_SRT && !LES);
}

// What a warp of the pair kernel knows before it steps its 64 cells.  near: the tile's mask byte.
struct PairMasks {
    bool general;  // a flag in or next to one of its two boxes
    uint4 m;       // the masks of the thread's two cells (0 in a box without): its pair, or by cell those of
                   // cells cell(t) and cell(t) + 32
    template <bool BY_CELL>
    __device__ __forceinline__ void load(uint32_t near, const uint2* masks, uint32_t tile, uint32_t t) {
        const uint32_t boxes = (near >> ((t >> 5) * 2u)) & 3u;
        general = !__all_sync(0xffffffffu, boxes == 0u);
        m = make_uint4(0u, 0u, 0u, 0u);
        if (!general) return;
        // (masks are written for every cell of a box with its bit set)
        if constexpr (BY_CELL) {
            const uint2* p = masks + (kTileCells * tile + cell(t));
            if (boxes & 1u) {
                const uint2 v = load_masks(p);
                m.x = v.x;
                m.y = v.y;
            }
            if (boxes & 2u) {
                const uint2 v = load_masks(p + 32);
                m.z = v.x;
                m.w = v.y;
            }
        } else {
            if ((near >> (t >> 4)) & 1u) m = load_masks2(masks + (2u * t + kTileCells * tile));
        }
    }
    static __device__ __forceinline__ uint32_t cell(uint32_t t) { return 2u * (t & ~31u) + (t & 31u); }
};

// The 256 cells of a tile by 128 threads.  (BY_CELL: pair_by_cell, or false.)
template <class L, int METHOD, bool F16C, int COLL, int LES, bool FAST, bool BY_CELL>
__device__ __forceinline__ void pair_step(const StepArgs& a, const uint32_t tile, const uint32_t t, const PairMasks& pm) {
    if (BY_CELL && pm.general) {
        uint32_t tl = tile;
        asm volatile("" : "+r"(tl));  // (nothing of this form is computed ahead of the branch)
#pragma unroll 1
        for (uint32_t b = 0; b < 2u; ++b)
            tile_cell<L, METHOD, F16C, COLL, LES, FAST, false, false, true, kPairThreads>(
                a, tl, PairMasks::cell(t) + 32u * b, b ? make_uint2(pm.m.z, pm.m.w) : make_uint2(pm.m.x, pm.m.y),
                nullptr, nullptr, nullptr);
        return;
    }
    const uint32_t byz = a.lay.d_ntx.div(tile);
    const uint32_t bx = tile - byz * (uint32_t)a.lay.ntx;
    const uint32_t bz = a.lay.d_nty.div(byz);
    const uint32_t by = byz - bz * (uint32_t)a.lay.nty;
    if (BY_CELL || !pm.general) pair_cells<L, METHOD, F16C, COLL, LES, FAST, false>(a, tile, t, pm.m, bx, by, bz);
    else pair_cells<L, METHOD, F16C, COLL, LES, FAST, true>(a, tile, t, pm.m, bx, by, bz);
}

// Resident CTAs (of 128 threads) per SM the pair kernels are built for: the populations of two
// cells stay in registers across both collisions, so the budget is wider than the per-cell
// kernel's.  Float16C in the fast arithmetic 8 (64 registers: 63.7 GLUPs on the 256^3 Float16C
// cavity against 60.0 at 9, 61.2 at 7 and 58.0 at 6), float32 8 (64 registers, a few spilled
// bytes in the wall warps' form only: 43.05 GLUPs on the float32 cavity against 42.46 at 7), the
// exact Float16C build 7 (72 registers; at 64 it spills), float32 D3Q19 SRT with LES 7 (64 registers spill 76
// bytes; 128^3 cavity 62.3 -> 60.4 us a step, vortex 53.4 -> 49.5), TRT 6 (80), KBC and D3Q27 4 (128).
#ifndef LBM_PAIR_MIN_BLOCKS_F16C_FAST
#define LBM_PAIR_MIN_BLOCKS_F16C_FAST 8
#endif
#ifndef LBM_PAIR_MIN_BLOCKS_F16C
#define LBM_PAIR_MIN_BLOCKS_F16C 7
#endif
#ifndef LBM_PAIR_MIN_BLOCKS
#define LBM_PAIR_MIN_BLOCKS 8
#endif
#ifndef LBM_PAIR_MIN_BLOCKS_HEAVY
#define LBM_PAIR_MIN_BLOCKS_HEAVY 4
#endif
template <class L, int METHOD, bool F16C, int COLL, int LES, bool FAST>
constexpr int pair_min_blocks() {
    if constexpr (FAST) {
        if (COLL == LBM_KBC || L::Q == 27) return LBM_PAIR_MIN_BLOCKS_HEAVY;
        if (COLL == LBM_TRT) return L::Q == 9 && METHOD == LBM_ESOTERIC_PULL ? 7 : 6;
        return L::Q == 19 && METHOD == LBM_ESOTERIC_PULL ? 7 : LBM_PAIR_MIN_BLOCKS_F16C_FAST;
    }
    return (COLL == LBM_KBC || L::Q == 27) ? LBM_PAIR_MIN_BLOCKS_HEAVY
           : COLL == LBM_TRT               ? 6
           : F16C                          ? LBM_PAIR_MIN_BLOCKS_F16C
           : L::Q == 19 && COLL == LBM_SRT && LES ? 7
                                                  : LBM_PAIR_MIN_BLOCKS;
}

template <class L, int METHOD, bool F16C, int COLL, int LES, bool FAST>
__global__ void __launch_bounds__(kPairThreads, (pair_min_blocks<L, METHOD, F16C, COLL, LES, FAST>())) step_kernel_pair(const StepArgs a) {
    static_assert(LES != kLesLearned, "the learned closure runs in step_kernel_learned");
    const uint32_t tile = blockIdx.x, t = threadIdx.x;
    pdl_wait_before_masks(a);
    constexpr bool BY_CELL = pair_by_cell<L, METHOD, F16C, COLL, LES, FAST>();
    PairMasks pm;
    pm.load<BY_CELL>(load_byte(a.tile_near + tile), a.cell_masks, tile, t);
    pdl_wait_after_masks(a);
    pair_step<L, METHOD, F16C, COLL, LES, FAST, BY_CELL>(a, tile, t, pm);
}

template <class L, int METHOD, bool F16C, int COLL, int LES>
cudaError_t launch_step_pair(const StepArgs& a, int, cudaStream_t s) {
    return launch_pdl(step_kernel_pair<L, METHOD, F16C, COLL, LES, false>, a.lay.ncells / kTileCells, kPairThreads, s, a);
}
template <class L, int METHOD, bool F16C, int COLL, int LES>
cudaError_t launch_step_pair_fast(const StepArgs& a, int, cudaStream_t s) {
    return launch_pdl(step_kernel_pair<L, METHOD, F16C, COLL, LES, true>, a.lay.ncells / kTileCells, kPairThreads, s, a);
}

}  // namespace lbm
