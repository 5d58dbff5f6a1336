// The collision of the fast-arithmetic build (LBM_ARITH_FAST): the same operators as collide()
// in lbm_step.cuh (src/lbm/kernels/steps/collide.mojo:23-90), rearranged for the FMA pipe and
// held to a float32 tolerance instead of the reference's operation order.
//
//  - Moments from the sums and differences of opposite pairs (q, q+1): rho = f0 + sum s_p,
//    m_d = sum +-d_p, Pi_ab = sum c_a c_b s_p (the reference sums f_q over q one by one,
//    src/utils/vector.mojo:205-224).
//  - One approximate reciprocal of rho (rcp.approx), u = m / rho as three products.
//  - Equilibria per opposite pair: f_eq(q), f_eq(q+1) = (A + C45 (e.u)^2) +- C3 (e.u) with the
//    weight, rho and the relaxation rate folded into A, C3, C45, so SRT is two FMAs per
//    population after three per pair (src/lbm/kernels/ops/collisions/collision.mojo:12-46).
//  - The non-equilibrium stress as the raw second moment less the equilibrium's,
//    rho u_a u_b + cs^2 (rho - ddf) delta_ab (algebraically the reference's sum of
//    (f - f_eq) c_a c_b, src/lbm/kernels/utils/moment.mojo:111-150).
//  - KBC (src/lbm/kernels/ops/collisions/KBC_.mojo:180-238) evaluates each f_eq once per pass and
//    takes 1/f_eq by rcp.approx in place of two IEEE divisions per direction.
//  - Float16C storage with a linear collision (SRT, TRT, RLBM without LES) works on "scaled"
//    populations: a code's bits shifted into float32 position are the population times 2^-112
//    (f16c_decode_sx without its final multiplication), the 2^112 is folded into the
//    coefficients, and the result is encoded straight from its scaled value
//    (f16c_encode_scaled).  Everything linear in f is exact under that scaling up to float32
//    rounding at the scaled magnitudes (float32 denormals below 2^-126, i.e. populations below
//    2^-14, keep an absolute resolution of 2^-37, far below a code's).
//
// Included by lbm_step.cuh after StepArgs, kbc_shear and collide.
#pragma once

#include "lbm_device.cuh"

namespace lbm {

// 1/x to within 1 ulp (PTX rcp.approx; subnormal inputs flush to zero, which rho and f_eq never are)
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ F2 rcp_approx(F2 a) { return F2{rcp_approx(a.x), rcp_approx(a.y)}; }
__device__ __forceinline__ F2 sqrt_approx(F2 a) { return F2{sqrt_approx(a.x), sqrt_approx(a.y)}; }

// e_q . u with the first positive component taken as is (no 0 + x), for the fast build (q odd: a
// direction with a positive component)
template <class L, int q, class V>
__device__ __forceinline__ V edot_fast(const V* u) {
    constexpr int d0 = L::c(q, 0) > 0 ? 0 : (L::c(q, 1) > 0 ? 1 : 2);
    static_assert(L::c(q, d0) > 0, "odd directions have a positive component");
    V o = u[d0];
    static_for<0, L::D>([&](auto dc) {
        constexpr int d = dc.value;
        if constexpr (d != d0 && L::c(q, d) > 0) o = o + u[d];
        else if constexpr (d != d0 && L::c(q, d) < 0) o = o - u[d];
    });
    return o;
}

template <class L, int q>
constexpr int nnz_of() { return (L::c(q, 0) != 0) + (L::c(q, 1) != 0) + (L::c(q, 2) != 0); }

// (e_q . u)^2; uc2: the squares of the components
template <class L, int q, class V>
__device__ __forceinline__ V edot2_fast(V eu, const V* uc2) {
    if constexpr (nnz_of<L, q>() == 1) return uc2[L::c(q, 0) != 0 ? 0 : (L::c(q, 1) != 0 ? 1 : 2)];
    else return eu * eu;
}

// The pair (q, q+1) of r * f_eq in units s: (plus, minus) = (A + C45 e2) +- C3 eu with
// A = w a0, C3 = 3 w r0, C45 = 4.5 w r0, where the caller passes a0 = r s (rho (1 - 1.5 uu) - ddf)
// and r0 = r s rho.  With ddf this is the shifted equilibrium
// w rho (3 eu + 4.5 eu^2 - 1.5 uu) + w (rho - 1) (src/lbm/kernels/utils/equilibrium.mojo:10-39).
template <class L, int q, class V>
__device__ __forceinline__ void feq_pair_fast(V a0, V r0, const V* u, const V* uc2, V& plus, V& minus) {
    constexpr float w = wf<L>(q);
    const V eu = edot_fast<L, q>(u);
    const V e2 = edot2_fast<L, q>(eu, uc2);
    const V base = vfma(r0 * (4.5f * w), e2, a0 * w);
    const V c3 = r0 * (3.f * w);
    plus = vfma(c3, eu, base);
    if constexpr (std::is_same_v<V, float>) minus = vfma(-c3, eu, base);
    else minus = vfma(r0 * (-3.f * w), eu, base);
}

// The collision of the fast build, in place on f (in units of 2^-112 when SCALED).  V: float, one cell,
// or F2, two cells by packed instructions, with the same operations on each.  capture(rho, u) is called
// with the density and velocity.
template <class L, int COLL, int LES, bool SCALED, class V, int NT = 256, class Capture>
__device__ __forceinline__ void collide_fast_v(V (&f)[L::Q], const StepArgs& a, Capture&& capture) {
    static_assert(!(SCALED && (LES || COLL == LBM_KBC)), "scaled populations need a collision linear in f");
    constexpr int Q = L::Q, D = L::D, NP = (Q - 1) / 2, NS = L::NS;
    constexpr float S = SCALED ? 0x1p-112f : 1.f;  // stored units per population unit
    constexpr float IS = SCALED ? 0x1p112f : 1.f;
    auto stored = [](V v) { if constexpr (SCALED) return v * S; else return v; };
    auto units = [](V v) { if constexpr (SCALED) return v * IS; else return v; };
    constexpr float cs2 = (float)(1.0 / 3.0);
    const float ddf = a.ddf ? 1.f : 0.f;

    // ---- moments from opposite pairs (the first direction with a component has it positive)
    V ps[NP], pd[NP];
    static_for<0, NP>([&](auto pc) {
        constexpr int p = pc.value, q = 2 * p + 1;
        ps[p] = f[q] + f[q + 1];
        pd[p] = f[q] - f[q + 1];
    });
    V rs = f[0];
    static_for<0, NP>([&](auto pc) { rs = rs + ps[pc.value]; });
    V ms[3] = {splat<V>(0.f), splat<V>(0.f), splat<V>(0.f)};
    static_for<0, D>([&](auto dc) {
        constexpr int d = dc.value;
        static_for<0, NP>([&](auto pc) {
            constexpr int p = pc.value, q = 2 * p + 1;
            if constexpr (p == d) ms[d] = pd[p];  // (the axis directions come first)
            else if constexpr (L::c(q, d) > 0) ms[d] = ms[d] + pd[p];
            else if constexpr (L::c(q, d) < 0) ms[d] = ms[d] - pd[p];
        });
    });
    const V rho = vfma(rs, IS, ddf);
    const V k = units(rcp_approx(rho));
    V u[3] = {splat<V>(0.f), splat<V>(0.f), splat<V>(0.f)}, uc2[3] = {splat<V>(0.f), splat<V>(0.f), splat<V>(0.f)};
    static_for<0, D>([&](auto dc) {
        u[dc.value] = ms[dc.value] * k;
        uc2[dc.value] = mul_apart(u[dc.value], u[dc.value]);
    });
    V uu = uc2[0] + uc2[1];
    if constexpr (D == 3) uu = uu + uc2[2];
    capture(rho, u);

    // rho (1 - 1.5 uu) - ddf: the part of f_eq / w without e.u
    const V r1 = vfma(rho, vfma(uu, -1.5f, 1.f), -ddf);

    // ---- non-equilibrium stress and the local relaxation time
    V tau_l = splat<V>(a.tau);
    [[maybe_unused]] V P[NS];
    constexpr bool NEED_NEQ = LES || COLL == LBM_KBC || COLL == LBM_RLBM;
    if constexpr (NEED_NEQ) {
        V nu_[3];  // -u
        static_for<0, D>([&](auto dc) { nu_[dc.value] = u[dc.value] * -1.f; });
        static_for<0, NS>([&](auto nc) {
            constexpr int n = nc.value, A = sa<L>(n), B = sb<L>(n);
            V raw = splat<V>(0.f);
            bool first = true;
            static_for<0, NP>([&](auto pc) {
                constexpr int p = pc.value, q = 2 * p + 1;
                constexpr int cc = L::c(q, A) * L::c(q, B);
                if constexpr (cc != 0) {
                    raw = first ? ps[p] : cc > 0 ? raw + ps[p] : raw - ps[p];
                    first = false;
                }
            });
            // Pi_ab = IS (raw - m_a u_b) - cs^2 (rho - ddf) delta_ab, with m_a = IS ms_a = rho u_a
            const V t = vfma(ms[A], nu_[B], raw);
            if constexpr (A == B) P[n] = vfma(t, IS, mul_apart(rho - ddf, -cs2));
            else P[n] = units(t);
        });
        if constexpr (LES) {
            // get_strain_rate_tensor / _norm_squared (moment.mojo:154-215),
            // get_Smagorinsky_LES_tau (src/lbm/kernels/ops/turbulence.mojo:12-38):
            // S = -Pi / (2 rho cs^2 tau), tau_l = tau + 3 Cs^2 sqrt(2 |S|^2)
            const V kS = rcp_approx(rho * (2.f * cs2) * a.tau);
            V s2 = splat<V>(0.f);
            static_for<0, NS>([&](auto nc) {
                constexpr int n = nc.value;
                const V pn = P[n];
                if constexpr (sa<L>(n) != sb<L>(n)) s2 = vfma(pn * 2.f, pn, s2);
                else s2 = vfma(pn, pn, s2);
            });
            // |S| = |Pi| kS
            tau_l = vfma(sqrt_approx(s2 * 2.f) * kS, 3.f * (a.Cs * a.Cs), a.tau);
        }
    }

    if constexpr (COLL == LBM_SRT) {
        // SRT: f' = (1 - w) f + w f_eq
        V om1, a0, r0;
        if constexpr (LES) {
            const V om = rcp_approx(tau_l);
            om1 = splat<V>(1.f) - om;
            a0 = stored(om) * r1;
            r0 = stored(om) * rho;
        } else {
            const float om = a.inv_tau;
            om1 = splat<V>(1.f - om);
            a0 = r1 * (om * S);
            r0 = rho * (om * S);
        }
        f[0] = vfma(om1, f[0], a0 * wf<L>(0));
        static_for<0, NP>([&](auto pc) {
            constexpr int q = 2 * pc.value + 1;
            V p, m;
            feq_pair_fast<L, q>(a0, r0, u, uc2, p, m);
            f[q] = vfma(om1, f[q], p);
            f[q + 1] = vfma(om1, f[q + 1], m);
        });
    } else if constexpr (COLL == LBM_TRT) {
        // TRT (collision.mojo:49-113), tau_asymm = 1/2 + Lambda / (tau - 1/2)
        // (steps/collide.mojo:214-215): symmetric part relaxed at 1/tau, antisymmetric at 1/tau_a
        const V os = rcp_approx(tau_l);
        const V tm = tau_l - 0.5f;
        const V oa = tm * rcp_approx(vfma(tm, 0.5f, a.trt_lambda));  // 1 / (1/2 + Lambda / tm)
        const V a0 = stored(os) * r1, r0s = stored(os) * rho, r0a = stored(oa) * rho;
        const V hs = os * 0.5f, ha = oa * 0.5f;
        f[0] = vfma(splat<V>(1.f) - os, f[0], a0 * wf<L>(0));
        static_for<0, NP>([&](auto pc) {
            constexpr int q = 2 * pc.value + 1;
            constexpr float w = wf<L>(q);
            const V eu = edot_fast<L, q>(u);
            const V e2 = edot2_fast<L, q>(eu, uc2);
            // os (f_s - feq_s) with f_s = (f_q + f_o) / 2, feq_s = w (r1 + 4.5 rho e2);
            // oa (f_a - feq_a) with f_a = (f_q - f_o) / 2, feq_a = 3 w rho eu
            const V sym = vfma(hs, ps[pc.value], vfma(r0s * (-4.5f * w), e2, a0 * -w));
            const V asy = vfma(ha, pd[pc.value], r0a * (-3.f * w) * eu);
            f[q] = (f[q] - sym) - asy;
            f[q + 1] = (f[q + 1] - sym) + asy;
        });
    } else if constexpr (COLL == LBM_RLBM) {
        // RLBM (collision.mojo:168-223): f' = f_eq + (1 - 1/tau) w / (2 cs^4) H : Pi_neq
        V g;
        if constexpr (LES) g = stored(splat<V>(1.f) - rcp_approx(tau_l));
        else g = splat<V>((1.f - a.inv_tau) * S);
        const V a0 = stored(r1), r0 = stored(rho);
        // rest direction: H = -cs^2 delta: H : Pi = -(Pxx + Pyy (+ Pzz)) / 3
        {
            V tr = P[0] + P[L::D == 2 ? 2 : 3];
            if constexpr (L::D == 3) tr = tr + P[5];
            constexpr float k0 = (float)(L::wd(0) / (2.0 / 9.0));
            f[0] = vfma(g * k0 * (float)(-1.0 / 3.0), tr, a0 * wf<L>(0));
        }
        static_for<0, NP>([&](auto pc) {
            constexpr int q = 2 * pc.value + 1;
            V dot = splat<V>(0.f);
            bool first = true;
            static_for<0, NS>([&](auto nc) {
                constexpr int n = nc.value, A = sa<L>(n), B = sb<L>(n);
                constexpr float Qn = (A == B) ? (float)(L::c(q, A) * L::c(q, B)) - (float)(1.0 / 3.0)
                                              : (float)(2 * L::c(q, A) * L::c(q, B));
                if constexpr (Qn != 0.f) {
                    dot = first ? P[n] * Qn : vfma(P[n], Qn, dot);
                    first = false;
                }
            });
            constexpr float kq = (float)(L::wd(q) / (2.0 / 9.0));
            V p, m;
            feq_pair_fast<L, q>(a0, r0, u, uc2, p, m);
            const V t = mul_apart(g * kq, dot);
            f[q] = p + t;
            f[q + 1] = m + t;
        });
    } else if constexpr (COLL == LBM_KBC) {
        // KBC (KBC_.mojo:180-238), gamma not clamped: beta = 1 / (2 tau_l),
        // dh = f - f_eq - ds, gamma = 2 tau_l - (2 - 2 tau_l) <ds, dh> / (<dh, dh> + 1e-32),
        // <x, y> = sum x y / f_eq (unshifted); f' = f - beta (2 ds + gamma dh)
        //       = f_eq + (1 - 2 beta) ds + (1 - beta gamma) dh.
        // One pass over the directions computes f_eq and ds once: dh goes to this thread's
        // lane-fastest slots of shared memory, f_eq + (1 - 2 beta) ds stays in f; once gamma is
        // known the update adds (1 - beta gamma) dh.  A single cell (V float) takes the two directions of an
        // opposite pair, whose ds is the same, by packed instructions (256^3 D3Q27 Float16C cavity, with
        // LES, us a step, one direction at a time / packed: in place 614.7 / 598.2, double buffer 603.7 /
        // 571.3; bound by issue, 1061 instructions a warp at 66 % issue activity).
        constexpr bool IN_CELL = std::is_same_v<V, float>;
        __shared__ V dh_keep[IN_CELL ? 1 : Q][NT * sizeof(float) / sizeof(V)];
        __shared__ F2 dh_pair[IN_CELL ? NP : 1][IN_CELL ? NT : 1];
        const uint32_t slot = threadIdx.x;
        const V beta = rcp_approx(tau_l) * 0.5f;
        const V inv_beta = tau_l * 2.f;
        const V cds = vfma(beta, -2.f, 1.f);
        const V a0u = rho * vfma(uu, -1.5f, 1.f);  // unshifted: rho (1 - 1.5 uu)
        V sp1 = splat<V>(0.f), sp2 = splat<V>(0.f);
        auto visit = [&](auto qc, V fe0) {
            constexpr int q = decltype(qc)::value;
            constexpr float w = wf<L>(q);
            const V ds = kbc_shear<L, q>(P);
            const V fe = fe0 - w * ddf;  // shifted: f_eq - w
            const V dh = (f[q] - fe) - ds;
            const V t = dh * rcp_approx(fe0);
            sp1 = vfma(ds, t, sp1);
            sp2 = vfma(dh, t, sp2);
            dh_keep[IN_CELL ? 0 : q][slot] = dh;
            f[q] = vfma(cds, ds, fe);
        };
        visit(std::integral_constant<int, 0>{}, mul_apart(a0u, wf<L>(0)));
        if constexpr (IN_CELL) {
            static_for<0, NP>([&](auto pc) {
                constexpr int p = pc.value, q = 2 * p + 1;
                constexpr float w = wf<L>(q);
                const float eu = edot_fast<L, q>(u);
                const float base = vfma(rho * (4.5f * w), edot2_fast<L, q>(eu, uc2), a0u * w);
                const float c3 = rho * (3.f * w), ds = kbc_shear<L, q>(P);
                const F2 fe0 = vfma(F2{c3, -c3}, F2{eu, eu}, F2{base, base});
                const F2 fe = fe0 - w * ddf;  // shifted: f_eq - w
                const F2 dh = (F2{f[q], f[q + 1]} - fe) - ds;
                const F2 t = dh * rcp_approx(fe0);
                sp1 = vfma(ds, t.y, vfma(ds, t.x, sp1));
                sp2 = vfma(dh.y, t.y, vfma(dh.x, t.x, sp2));
                dh_pair[p][slot] = dh;
                const F2 g = vfma(F2{cds, cds}, F2{ds, ds}, fe);
                f[q] = g.x;
                f[q + 1] = g.y;
            });
        } else {
            static_for<0, NP>([&](auto pc) {
                constexpr int q = 2 * pc.value + 1;
                V p, m;
                feq_pair_fast<L, q>(a0u, rho, u, uc2, p, m);
                visit(std::integral_constant<int, q>{}, p);
                visit(std::integral_constant<int, q + 1>{}, m);
            });
        }
        const V gamma = inv_beta - mul_apart((splat<V>(2.f) - inv_beta) * sp1, rcp_approx(sp2 + 1e-32f));
        const V cdh = vfma(beta * -1.f, gamma, splat<V>(1.f));
        if constexpr (IN_CELL) {
            f[0] = vfma(cdh, dh_keep[0][slot], f[0]);
            static_for<0, NP>([&](auto pc) {
                constexpr int p = pc.value, q = 2 * p + 1;
                const F2 g = vfma(F2{cdh, cdh}, dh_pair[p][slot], F2{f[q], f[q + 1]});
                f[q] = g.x;
                f[q + 1] = g.y;
            });
        } else {
            static_for<0, Q>([&](auto qc) { f[qc.value] = vfma(cdh, dh_keep[qc.value][slot], f[qc.value]); });
        }
    }
}

// One cell.  bc_own_base, T, own_flag: the capture outputs, as collide() writes them.
template <class L, int COLL, int LES, bool SCALED, int NT = 256>
__device__ __forceinline__ void collide_fast(float (&f)[L::Q], const StepArgs& a, float* bc_own_base, uint32_t T,
                                             uint8_t own_flag, bool active = true) {
    collide_fast_v<L, COLL, LES, SCALED, float, NT>(f, a, [&](float rho, const float* u) {
        if (active && a.cap_rho && (own_flag & LBM_FLAG_CAPTURE_DENSITY)) bc_own_base[(size_t)T * L::D] = rho;
        if (active && a.cap_u && (own_flag & LBM_FLAG_CAPTURE_VELOCITY))
            static_for<0, L::D>([&](auto dc) { bc_own_base[(size_t)T * dc.value] = u[dc.value]; });
    });
}

}  // namespace lbm
