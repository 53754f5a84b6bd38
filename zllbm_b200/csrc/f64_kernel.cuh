// The fused collide + stream step in FP64 storage: the reference's arithmetic, operation for
// operation (the unit is compiled with -fmad=false; collide_exact of aa_kernel.cuh is the same sequence
// in one function per node).
//
// What bounds it: a D3Q19 MRT node needs 722 FP64 multiplies and adds for its dense M^-1 S M (the
// reference's summation order admits no shortcut) plus about 250 for moments and equilibria, so at 64
// FP64 operations per SM and cycle the node costs 15 cycles of an SM against 14 for its 304 bytes of
// HBM traffic: everything else has to stay out of the way.  Hence
//  * the matrix travels in the kernel's parameters (constant bank, read through the uniform path)
//    instead of 361 global loads per node;
//  * every row of the matrix is formed and stored at once, so that the node holds its populations and
//    f - feq in registers and no post-collision array (no local-memory traffic);
//  * SRT divides by the level's relaxation time through a precomputed reciprocal (DivByConstant).
// MRT on periodic boxes on B200, per step: 128^3 333 us with the one-node kernel of aa_kernel.cuh at 80
// registers, 135 us here (15.5 k MLUPS; 4.7 TB/s); 64^3 43 -> 18 us; 256^3 1163 us.
#pragma once
#include "aa_kernel.cuh"

namespace zl {

// M^-1 S M of a level, and M^-1 (I - S/2) M when it is forced, as a kernel argument.
template <int Q, bool Mrt, bool Forced> struct MrtArg {};
template <int Q> struct MrtArg<Q, true, false> {
    double a[Q * Q];
};
template <int Q> struct MrtArg<Q, true, true> {
    double a[Q * Q], b[Q * Q];
};

// x / b for a divisor known in advance, correctly rounded: with the reciprocal as an unevaluated sum
// zh + zl, fma(x, zh, x zl) is within one ulp of the quotient (N. Brisebarre, J.-M. Muller and
// S. K. Raina, "Accelerating correctly rounded floating-point division when the divisor is known in
// advance", IEEE Trans. Computers 53, 2004), and a residual step with the correctly rounded zh then
// gives the rounded quotient (P. Markstein, IBM J. Res. Dev. 34, 1990).  The residual is exact for
// quotients well inside the normal range; smaller (and non-finite) ones take the division.
struct DivByConstant {
    double b, zh, zl;
    __device__ __forceinline__ double operator()(double x) const {
        const double q = __fma_rn(x, zh, x * zl);
        const double r = __fma_rn(-q, b, x);
        const uint32_t hi = (uint32_t)__double2hiint(q) & 0x7fffffffu;
        // 2^-960 <= |q| < 2^992, or a zero
        if (hi - 0x03f00000u < 0x7a000000u || (hi | (uint32_t)__double2loint(q)) == 0u) return __fma_rn(r, zh, q);
        return x / b;
    }
};

// Guo forcing term of direction q (CalForcingTerming2D / 3D, lbm_solver_interface.cpp:443-470); the
// products with a zero lattice component are left out.
template <class L>
__device__ __forceinline__ double guo_term(int q, const double* F, double ux, double uy, double uz) {
    using Tb = Tables<L>;
    auto dot = [&](double x, double y, double z) -> double {
        double s = 0.;
        bool first = true;
        if (Tb::cx(q)) { s = Tb::cx(q) > 0 ? x : -x; first = false; }
        if (Tb::cy(q)) { const double t = Tb::cy(q) > 0 ? y : -y; s = first ? t : s + t; first = false; }
        if (L::kDims == 3 && Tb::cz(q)) { const double t = Tb::cz(q) > 0 ? z : -z; s = first ? t : s + t; }
        return s;
    };
    const double cx = Tb::cx(q), cy = Tb::cy(q), cz = Tb::cz(q);
    double lin = (cx - ux) * F[0] + (cy - uy) * F[1];
    if (L::kDims == 3) lin = lin + (cz - uz) * F[2];
    return Tb::w(q) * (3. * lin + 9. * dot(ux, uy, uz) * dot(F[0], F[1], F[2]));
}

template <class L, int Coll, bool Odd, bool Bnd, bool Masked, int Ext>
__global__ void __launch_bounds__(256, 2)
    aa_step_f64_kernel(double* f, LevelGeom geo, StepParams p,
                       const __grid_constant__ MrtArg<L::kQ, Coll == kMrt, (Ext & kExtForce) != 0> m) {
    constexpr bool Forced = (Ext & kExtForce) != 0, Les = (Ext & kExtLes) != 0;
    static_assert(!(Les && Coll == kMrt), "MRT with a relaxation time per node builds its matrix per node");
    using Tb = Tables<L>;
    constexpr int Q = L::kQ;
    pdl_wait();
    pdl_trigger();
    const Coord c = step_coord(geo);
    if (c.x[0] >= geo.n[0] || c.x[1] >= geo.n[1]) return;

    const NodeCells<L> cell(geo, c);
    const int self = cell(0, 0, 0);
    const long long st = geo.stride;
    auto read_slot = [&](int q) -> double* {
        if (Odd && q != 0) return f + Tb::opp(q) * st + cell(-Tb::cx(q), -Tb::cy(q), -Tb::cz(q));
        return f + q * st + self;
    };
    auto write_slot = [&](int q) -> double* {
        if (Odd && q != 0) return f + q * st + cell(Tb::cx(q), Tb::cy(q), Tb::cz(q));
        return f + Tb::opp(q) * st + self;
    };
    const uint32_t info = Masked ? __ldg(geo.info + self) : 0u;
    double pre[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) pre[q] = *read_slot(q);
    if (Masked && !(info & kInfoPresent)) return;

    // a node whose force is exactly zero takes the unforced operations: every term the force would
    // add is a zero, which changes no value
    double F[3] = {0., 0., 0.};
    bool forced = false;
    if (Forced) {
        const bool node_force = p.force && (!Masked || (info & kInfoForce));
#pragma unroll
        for (int a = 0; a < 3; ++a) F[a] = p.const_force[a] + (node_force ? p.force[(long long)self * 3 + a] : 0.);
        forced = !(F[0] == 0. && F[1] == 0. && F[2] == 0.);
    }
    double rho, ux, uy, uz;
    macro_exact<L>(pre, rho, ux, uy, uz, Forced && forced ? F : nullptr, p.dt);
    if (Masked && (info & kInfoSaveMacro)) {
        double* mac = p.macro + (long long)self * 4;
        mac[0] = rho;
        mac[1] = ux;
        mac[2] = uy;
        mac[3] = uz;
    }
    double d[Q];  // feq, then f - feq
    feq_exact<L>(rho, ux, uy, uz, d);
    double tau = p.tau;
    if constexpr (Les)
        tau = p.tau + smag_tau_sgs_exact<L>(pre, d, p.tau, p.les_c, Forced && forced, F, p.dt, ux, uy, uz);
#pragma unroll
    for (int q = 0; q < Q; ++q) d[q] = pre[q] - d[q];

    // D2Q9 has the registers to keep its post-collision values for the patch below
    constexpr bool kKeepPost = Q == 9;
    double post[kKeepPost ? Q : 1];
    auto put = [&](int q, double v) {
        *write_slot(q) = v;
        if (kKeepPost) post[kKeepPost ? q : 0] = v;
    };
    if constexpr (Coll == kSrt) {
        const DivByConstant by_tau{p.tau, p.inv_tau_hi, p.inv_tau_lo};
        const double keep = Forced && forced ? 1. - 0.5 / tau : 0.;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            double v = pre[q] - (Les ? d[q] / tau : by_tau(d[q]));
            if (Forced && forced) v = v + keep * guo_term<L>(q, F, ux, uy, uz) * p.dt;
            put(q, v);
        }
    } else {
        bool done = false;
        if constexpr (Forced) {
            if (forced) {
                double t[Q];
#pragma unroll
                for (int q = 0; q < Q; ++q) t[q] = guo_term<L>(q, F, ux, uy, uz);
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    double acc = 0.;
#pragma unroll
                    for (int s = 0; s < Q; ++s) acc = acc + (m.a[q * Q + s] * d[s] - m.b[q * Q + s] * t[s] * p.dt);
                    put(q, pre[q] - acc);
                }
                done = true;
            }
        }
        if (!done) {
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                double acc = 0.;
#pragma unroll
                for (int s = 0; s < Q; ++s) acc = acc + m.a[q * Q + s] * d[s];
                put(q, pre[q] - acc);
            }
        }
    }

    // stale values and fused bounce back where the upstream node is missing (as in aa_node); D3Q19 reads
    // the post-collision values a bounce back needs back from the slots this node just wrote, which
    // no patch overwrites: a patch goes to the slot that holds f(x, q) in the next layout, off this
    // node's own writes
    bool patch = false;
    if (Masked) {
        patch = (info & ((1u << Q) - 2u)) != 0u;
    } else if (Bnd) {
#pragma unroll
        for (int a = 0; a < L::kDims; ++a)
            if (!geo.periodic[a] && (c.x[a] == 0 || c.x[a] == geo.n[a] - 1)) patch = true;
    }
    if (!patch) return;
    const int faces = Bnd ? (Masked ? (int)((info >> kInfoFaceShift) & 63u) : on_faces(geo, c, L::kDims)) : 0;
#pragma unroll
    for (int q = 1; q < Q; ++q) {
        const bool miss = Masked ? ((info >> q) & 1u) : upstream_missing<L>(geo, c, q);
        if (!miss) continue;
        double v = pre[q];
        if (faces && p.fuse_bb) {
            // the last bounce-back face in the reference's order the node lies on and q enters through
#pragma unroll
            for (int k = 0; k < 2 * L::kDims; ++k) {
                const int face = k < L::kDims ? 2 * k : 2 * (k - L::kDims) + 1;
                if (((faces >> face) & 1) && p.face_kind[face] == kBcBounceBack && enters_through<L>(q, face)) {
                    const int o = bb_source<L>(q, face);
                    v = (kKeepPost ? post[kKeepPost ? o : 0] : *write_slot(o)) - p.bb_term[face][o];
                }
            }
        }
        if (Odd) f[q * st + self] = v;
        else f[Tb::opp(q) * st + cell(-Tb::cx(q), -Tb::cy(q), -Tb::cz(q))] = v;
    }
}

}  // namespace zl
