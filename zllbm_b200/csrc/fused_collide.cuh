// The fused D3Q19 collisions of FP32 storage and of the learned step, written once for one node (F1) and for a
// pair of nodes in packed FP32 registers (F2 of pair_value.cuh), and those of the 16-bit pair and row kernels.
// The 16-bit one-node kernel and forced MRT levels keep the contracted forms of aa_kernel.cuh, which their
// results have always been rounded with.
//
// Every operation is explicit (no product and sum left for the compiler to contract), so a node's
// result has the same bits whether a kernel updates it alone or as half of a pair, and step kernels
// of different widths can stand in for one another.
#pragma once
#include <cuda_runtime.h>
#include "level_params.cuh"

namespace zl {

struct F1 {
    float v;
};
__device__ __forceinline__ F1 operator+(F1 a, F1 b) { return {__fadd_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 operator-(F1 a, F1 b) { return {__fsub_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 operator*(F1 a, F1 b) { return {__fmul_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 vfma(F1 a, F1 b, F1 c) { return {__fmaf_rn(a.v, b.v, c.v)}; }

__device__ __forceinline__ F1 neg(F1 a) { return {-a.v}; }

template <class V> __device__ __forceinline__ V splat_as(float s);
template <> __device__ __forceinline__ F1 splat_as<F1>(float s) { return {s}; }

// fn applied to every element
template <class Fn> __device__ __forceinline__ F1 each(F1 a, Fn fn) { return {fn(a.v)}; }

// Relaxation frequency of the Smagorinsky model from the stress norm: tau = tau0 + tau_sgs,
// tau_sgs = (sqrt(tau0^2 + C sqrt(2 Pi:Pi)) - tau0) / 2 (lbm_les_smagorinsky.cpp:22-94).
__device__ __forceinline__ float smag_omega(float pi2, float c, float tau0) {
    const float s = __fsqrt_rn(__fmaf_rn(c, __fsqrt_rn(__fmul_rn(2.f, pi2)), __fmul_rn(tau0, tau0)));
    return __frcp_rn(__fmaf_rn(0.5f, __fsub_rn(s, tau0), tau0));
}
__device__ __forceinline__ F1 smag_omega(F1 pi2, F1 c, float tau0) { return {smag_omega(pi2.v, c.v, tau0)}; }

// D3Q19 SRT (also with a body force) or MRT, on the deviations d (scaled units), in one pass: the pair
// sums and differences of opposite directions give the density, the momentum, the stress and the
// relaxed moments, and every opposite pair's output is formed from its sum and difference.
//
// f* = f - omega neq - sum_k lambda_k m_k M_k over the moments whose rate is not the shear rate,
// lambda_k = (s_k - omega) / |M_k|^2 (SRT: none).  The relaxed moments of neq are the moments of d
// minus their equilibrium values, closed forms in (rho, j) for the reference's second-order
// equilibrium (lbm_solver_interface.cpp:374-435): with drho = scale (rho - 1), G = scale rho,
// m1 = 19 (Sd - d0 - G u^2), m2 = 9 d0 - 7 Sa - 2 Sd + 5.5 G u^2, m4 = -(10/3) D1 + (5/3)(X1 + X2)
// (likewise m6, m8), m10 = M10.d + G (3 ux^2 - u^2) / 2, m12 = M12.d + G (uy^2 - uz^2) / 2,
// m16..18 = M.d.
//
// Les: omega per node from the non-equilibrium stress Pi_ab = sum_q c_a c_b d_q - drho / 3 delta_ab -
// G u_a u_b and the Smagorinsky constant les_c; otherwise omega is the level's.
// Forced (SRT): the Guo force F (CalMacroForce*, CalForcingTerming3D: lbm_solver_interface.cpp:443-470,
// 541-592) shifts the velocity by F dt / (2 rho), j is G u, the stress gains dt (F_a u_b + F_b u_a) / 2,
// and the term Fq_q = w [3 (c - u).F + 9 (c.u)(c.F)] splits into an even part w (9 (c.u)(c.F) - 3 u.F)
// and an odd part 3 w (c.F) per pair.
// 1 / rho is correctly rounded in the MRT + Smagorinsky and the forced collisions and the caller's where it has
// it (inv_rho: the learned SRT step, rounded too), which have always divided so; otherwise the fast reciprocal,
// two ulps.
// mac (optional): rho, ux, uy, uz.
// Planes: the two diagonal pairs of a coordinate plane share the even part that is symmetric in them, which
// MRT corrects once for both.  An SRT pair from its own (c.u)^2 instead is as many operations in a shorter
// chain, which the one-node kernel is bound by (us per step, 64^3 6.73 -> 6.61, between walls 256^3 546 -> 535,
// Smagorinsky 161 x 97 x 81 36.8 -> 36.1, between walls 37.2 -> 36.5; pairs with Smagorinsky, 256^3, within
// 0.7 %).  The 16-bit storages keep the bits of the shared form.
template <bool Mrt, bool Les, bool Forced, class V, bool Planes = Mrt>
__device__ __forceinline__ void fused_collide(const V* d, V* out, const StepParams& p, V les_c, const V* F, V* mac,
                                              const V* inv_rho = nullptr) {
    static_assert(!(Mrt && Forced), "the forced MRT collision has no fused form");
    auto S = [](float s) { return splat_as<V>(s); };
    const float* lam = p.mrt_coef;
    const V S1 = d[1] + d[2], D1 = d[1] - d[2];
    const V S2 = d[3] + d[4], D2 = d[3] - d[4];
    const V S3 = d[5] + d[6], D3 = d[5] - d[6];
    const V S4 = d[7] + d[10], D4 = d[7] - d[10];
    const V S5 = d[8] + d[9], D5 = d[8] - d[9];
    const V S6 = d[11] + d[14], D6 = d[11] - d[14];
    const V S7 = d[12] + d[13], D7 = d[12] - d[13];
    const V S8 = d[15] + d[18], D8 = d[15] - d[18];
    const V S9 = d[16] + d[17], D9 = d[16] - d[17];
    const V S23 = S2 + S3;
    const V Sa = S1 + S23;
    const V Sxy = S4 + S5, Sxz = S6 + S7, Syz = S8 + S9;
    const V Sd = (Sxy + Sxz) + Syz;
    const V drho = (d[0] + Sa) + Sd;
    const V X1 = D4 - D5, X2 = D6 - D7;
    const V Y1 = D4 + D5, Y2 = D8 - D9;
    const V Z1 = D6 + D7, Z2 = D8 + D9;
    const V X12 = X1 + X2, Y12 = Y1 + Y2, Z12 = Z1 + Z2;
    V jx = D1 + X12, jy = D2 + Y12, jz = D3 + Z12;
    const V rho = vfma(drho, S(p.inv_scale), S(1.f));
    const float is = p.inv_scale;
    V ux, uy, uz;
    if constexpr (Forced) {
        const V r = each(rho, [](float x) { return __frcp_rn(x); });
        const V k = S(is) * r, hf = S(0.5f * (float)p.dt) * r;
        ux = vfma(hf, F[0], jx * k);
        uy = vfma(hf, F[1], jy * k);
        uz = vfma(hf, F[2], jz * k);
    } else {
        V k;
        if (inv_rho) k = S(is) * *inv_rho;
        else if constexpr (Mrt && Les) k = S(is) * each(rho, [](float r) { return __frcp_rn(r); });
        else k = each(rho, [is](float r) { return __fdividef(is, r); });
        ux = jx * k;
        uy = jy * k;
        uz = jz * k;
    }
    if (mac) {
        mac[0] = rho;
        mac[1] = ux;
        mac[2] = uy;
        mac[3] = uz;
    }
    const V ux2 = ux * ux, uy2 = uy * uy, uz2 = uz * uz;
    const V usq = (ux2 + uy2) + uz2;
    const V G = S(p.scale) * rho;
    const V Gu = G * usq;
    const V zero = S(0.f);
    if constexpr (Forced) {
        // the momentum of the shifted equilibrium
        jx = G * ux;
        jy = G * uy;
        jz = G * uz;
    }
    V om = S(p.omega32);
    if constexpr (Les) {
        const V t = drho * S(1.f / 3.f), nG = neg(G);
        V pxx = vfma(nG, ux2, (S1 + (Sxy + Sxz)) - t);
        V pyy = vfma(nG, uy2, (S2 + (Sxy + Syz)) - t);
        V pzz = vfma(nG, uz2, (S3 + (Sxz + Syz)) - t);
        V pxy = vfma(nG, ux * uy, S4 - S5);
        V pxz = vfma(nG, ux * uz, S6 - S7);
        V pyz = vfma(nG, uy * uz, S8 - S9);
        if constexpr (Forced) {
            const V ds = S((float)p.dt * p.scale), half = S(0.5f);
            const V fx = (ds * F[0]) * ux, fy = (ds * F[1]) * uy, fz = (ds * F[2]) * uz;
            pxx = pxx + fx;
            pyy = pyy + fy;
            pzz = pzz + fz;
            pxy = vfma(half, fx + fy, pxy);
            pxz = vfma(half, fx + fz, pxz);
            pyz = vfma(half, fy + fz, pyz);
        }
        const V dia = vfma(pzz, pzz, vfma(pyy, pyy, pxx * pxx));
        const V off = vfma(pyz, pyz, vfma(pxz, pxz, pxy * pxy));
        const V pi2 = S(is * is) * vfma(S(2.f), off, dia);
        om = smag_omega(pi2, les_c, (float)p.tau);
    }
    // lambda_k times a factor: with Les from the node's own omega
    auto rate = [&](int m, float factor) -> V {
        if constexpr (Les) {
            const float w = factor / (float)row_norm2<D3Q19>(m);
            return vfma(om, S(-w), S((float)Tables<D3Q19>::s(m) * w));
        } else {
            return S(factor * lam[m]);
        }
    };
    V c0 = zero, cx = zero, cy = zero, cz = zero, c_xy = zero, c_xz = zero, c_yz = zero;
    V a4x4 = zero, a6x4 = zero, a8x4 = zero, u1 = zero, u2 = zero, v1 = zero, v2 = zero, t1 = zero, t2 = zero;
    if constexpr (Mrt) {
        // relaxed moments of neq, times lambda_k
        const V a1 = rate(1, 19.f) * ((Sd - d[0]) - Gu);
        const V a2 = rate(2, 1.f) * vfma(S(5.5f), Gu, vfma(S(9.f), d[0], vfma(S(-7.f), Sa, S(-2.f) * Sd)));
        const V a4 = rate(4, 1.f) * vfma(S(-10.f / 3.f), D1, S(5.f / 3.f) * X12);
        const V a6 = rate(6, 1.f) * vfma(S(-10.f / 3.f), D2, S(5.f / 3.f) * Y12);
        const V a8 = rate(8, 1.f) * vfma(S(-10.f / 3.f), D3, S(5.f / 3.f) * Z12);
        const V hG = S(0.5f) * G;
        const V a10 = rate(10, 1.f) * vfma(hG, vfma(S(3.f), ux2, neg(usq)),
                                           vfma(S(-4.f), S1, vfma(S(2.f), S23, (Sxy + Sxz) - S(2.f) * Syz)));
        const V a12 = rate(12, 1.f) * vfma(hG, uy2 - uz2, vfma(S(2.f), S3 - S2, Sxy - Sxz));
        const V a16 = rate(16, 1.f) * (X1 - X2), a17 = rate(17, 1.f) * (Y2 - Y1), a18 = rate(18, 1.f) * (Z1 - Z2);
        const V e_ax = vfma(S(-11.f), a1, S(-4.f) * a2);
        const V e_dg = vfma(S(8.f), a1, a2);
        c0 = vfma(S(-30.f), a1, S(12.f) * a2);
        cx = vfma(S(-4.f), a10, e_ax);
        cy = vfma(S(2.f), a10 - a12, e_ax);
        cz = vfma(S(2.f), a10 + a12, e_ax);
        c_xy = e_dg + (a10 + a12);
        c_xz = e_dg + (a10 - a12);
        c_yz = vfma(S(-2.f), a10, e_dg);
        a4x4 = S(4.f) * a4;
        a6x4 = S(4.f) * a6;
        a8x4 = S(4.f) * a8;
        u1 = a4 + a16;  // q7: u1 + u2, q8: u2 - u1
        u2 = a6 - a17;
        v1 = a4 - a16;  // q11: v1 + v2, q12: v2 - v1
        v2 = a8 + a18;
        t1 = a6 + a17;  // q15: t1 + t2, q16: t2 - t1
        t2 = a8 - a18;
    }
    // corrections: x - c (nothing to subtract for SRT) and fma(a, b, c)
    auto less = [](V x, V c) -> V {
        if constexpr (Mrt) return x - c;
        else return x;
    };
    auto odd = [](V a, V b, V c) -> V {
        if constexpr (Mrt) return vfma(a, b, c);
        else return a * b;
    };
    // omega feq: w (B + 4.5 G (c.u)^2) even, 3 w (c.j) odd, B = drho - 1.5 G u^2
    const V B = vfma(S(-1.5f), Gu, drho);
    V ow0, K1, L1, K2, L2, o1, o2, h, keep;
    if constexpr (Les) {
        const V ow1 = om * S(1.f / 18.f), ow2 = om * S(1.f / 36.f);
        ow0 = om * S(1.f / 3.f);
        K1 = (S(4.5f) * ow1) * G;
        L1 = ow1 * B;
        K2 = (S(4.5f) * ow2) * G;
        L2 = ow2 * B;
        o1 = ow1 * S(3.f);
        o2 = ow2 * S(3.f);
        keep = S(1.f) - om;
        h = S(0.5f) * keep;
    } else {
        const float omega = p.omega32;
        const float w1 = omega * (1.f / 18.f), w2 = omega * (1.f / 36.f);
        ow0 = S(omega * (1.f / 3.f));
        K1 = S(4.5f * w1) * G;
        L1 = S(w1) * B;
        K2 = S(4.5f * w2) * G;
        L2 = S(w2) * B;
        o1 = S(w1 * 3.f);
        o2 = S(w2 * 3.f);
        h = S(0.5f * (1.f - omega));
        keep = S(1.f - omega);
    }
    // (1 - omega) d_q of a pair of opposite directions from their sum and difference
    auto pair = [&](int q, int o, V Sq, V Dq, V A, V Bo) {
        const V e = vfma(h, Sq, A), od = vfma(h, Dq, Bo);
        out[q] = e + od;
        out[o] = e - od;
    };
    if constexpr (Forced) {
        // Guo parts, scaled: g_w = (1 - omega/2) dt scale w
        const V g = vfma(om, S(-0.5f), S(1.f)) * S((float)p.dt * p.scale);
        const V g1 = g * S(1.f / 18.f), g2 = g * S(1.f / 36.f), three = S(3.f), nine = S(9.f);
        const V uF3 = three * vfma(uz, F[2], vfma(uy, F[1], ux * F[0]));
        out[0] = vfma(keep, d[0], vfma(ow0, B, neg(g * S(1.f / 3.f)) * uF3));
        // a pair with c.u = cu, c.j = cj, c.F = cF, weight factors K, L, o and gw
        auto forced = [&](int q, int o, V Sq, V Dq, V K, V Lw, V ow, V gw, V cu, V cj, V cF) {
            const V ev = vfma(gw, vfma(nine * cu, cF, neg(uF3)), vfma(K, cu * cu, Lw));
            pair(q, o, Sq, Dq, ev, vfma(gw * three, cF, ow * cj));
        };
        forced(1, 2, S1, D1, K1, L1, o1, g1, ux, jx, F[0]);
        forced(3, 4, S2, D2, K1, L1, o1, g1, uy, jy, F[1]);
        forced(5, 6, S3, D3, K1, L1, o1, g1, uz, jz, F[2]);
        forced(7, 10, S4, D4, K2, L2, o2, g2, ux + uy, jx + jy, F[0] + F[1]);
        forced(8, 9, S5, D5, K2, L2, o2, g2, uy - ux, jy - jx, F[1] - F[0]);
        forced(11, 14, S6, D6, K2, L2, o2, g2, ux + uz, jx + jz, F[0] + F[2]);
        forced(12, 13, S7, D7, K2, L2, o2, g2, uz - ux, jz - jx, F[2] - F[0]);
        forced(15, 18, S8, D8, K2, L2, o2, g2, uy + uz, jy + jz, F[1] + F[2]);
        forced(16, 17, S9, D9, K2, L2, o2, g2, uz - uy, jz - jy, F[2] - F[1]);
        return;
    }
    if constexpr (Mrt) out[0] = vfma(keep, d[0], vfma(ow0, B, neg(c0)));
    else out[0] = vfma(keep, d[0], ow0 * B);
    pair(1, 2, S1, D1, less(vfma(K1, ux2, L1), cx), odd(o1, jx, a4x4));
    pair(3, 4, S2, D2, less(vfma(K1, uy2, L1), cy), odd(o1, jy, a6x4));
    pair(5, 6, S3, D3, less(vfma(K1, uz2, L1), cz), odd(o1, jz, a8x4));
    if constexpr (Planes) {
        const V K2x2 = K2 + K2;
        {
            const V P = less(vfma(K2, ux2 + uy2, L2), c_xy), Q = K2x2 * (ux * uy);
            pair(7, 10, S4, D4, P + Q, odd(o2, jx + jy, neg(u1 + u2)));
            pair(8, 9, S5, D5, P - Q, odd(o2, jy - jx, u1 - u2));
        }
        {
            const V P = less(vfma(K2, ux2 + uz2, L2), c_xz), Q = K2x2 * (ux * uz);
            pair(11, 14, S6, D6, P + Q, odd(o2, jx + jz, neg(v1 + v2)));
            pair(12, 13, S7, D7, P - Q, odd(o2, jz - jx, v1 - v2));
        }
        {
            const V P = less(vfma(K2, uy2 + uz2, L2), c_yz), Q = K2x2 * (uy * uz);
            pair(15, 18, S8, D8, P + Q, odd(o2, jy + jz, neg(t1 + t2)));
            pair(16, 17, S9, D9, P - Q, odd(o2, jz - jy, t1 - t2));
        }
    } else {
        auto diagonal = [&](int q, int o, V Sq, V Dq, V cu, V cj) { pair(q, o, Sq, Dq, vfma(K2, cu * cu, L2), o2 * cj); };
        diagonal(7, 10, S4, D4, ux + uy, jx + jy);
        diagonal(8, 9, S5, D5, uy - ux, jy - jx);
        diagonal(11, 14, S6, D6, ux + uz, jx + jz);
        diagonal(12, 13, S7, D7, uz - ux, jz - jx);
        diagonal(15, 18, S8, D8, uy + uz, jy + jz);
        diagonal(16, 17, S9, D9, uz - uy, jz - jy);
    }
}

}  // namespace zl
