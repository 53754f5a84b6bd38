// The per-level description that every kernel takes by value: box geometry, per-cell info bits and
// physical parameters.
#pragma once
#include <cstdint>
#include "lattice.cuh"

namespace zl {

enum BcKind : int { kBcNone = 0, kBcBounceBack = 1, kBcPeriodic = 2, kBcNeq = 3, kBcConvective = 4 };
enum Collision : int { kSrt = 0, kMrt = 1 };

// Per-cell information for levels whose node set does not fill its box.
constexpr uint32_t kInfoPresent = 1u << 31;
constexpr uint32_t kInfoSaveMacro = 1u << 30;  // keep rho, u of the last collision (coarse/fine transfer source)
constexpr uint32_t kInfoForce = 1u << 23;  // node force may be non-zero (a stencil node of the immersed boundary)
constexpr int kInfoFaceShift = 24;  // 6 bits: on face xmin..zmax (reference boundary node sets)

// extended-physics bits of the step kernel's Ext template argument
constexpr int kExtForce = 1;
constexpr int kExtLes = 2;

// Division of 31-bit unsigned integers by a fixed divisor through one widening multiply and a
// shift (Granlund and Montgomery, "Division by invariant integers using multiplication", PLDI
// 1994, the round-up method): with l = ceil(log2 d) and m = floor(2^(31 + l) / d) + 1,
// floor(n / d) = floor(n m / 2^(31 + l)) for every 0 <= n < 2^31; m < 2^32 for d >= 2.
struct FastDiv {
    uint32_t d = 1, m = 0, shift = 0;
    ZL_HD static FastDiv make(uint32_t divisor) {
        FastDiv f;
        f.d = divisor;
        if (divisor <= 1) return f;
        uint32_t l = 0;
        while ((1ull << l) < divisor) ++l;
        f.shift = 31 + l;
        f.m = (uint32_t)((1ull << f.shift) / divisor + 1);
        return f;
    }
    ZL_HD uint32_t div(uint32_t n) const {
        return d <= 1 ? n : (uint32_t)(((unsigned long long)n * m) >> shift);
    }
};

struct LevelGeom {
    int n[3];          // nodes per axis (periodic axes hold each plane once)
    int g[3];          // ghost frame width per axis (0 on periodic axes, 1 otherwise)
    int a[3];          // allocated extents, n + 2 g
    int periodic[3];   // wrap-around per axis
    long long stride;  // elements between population planes (>= a0 a1 a2)
    int face_on_box;   // bit f: box edge f lies on domain face f (non-periodic faces only)
    int block[2];      // thread-block shape of the step kernel (x, y); {0, 0}: default
    const uint32_t* info;  // per-cell info (masked levels), nullptr for full boxes
    // 1: a full D3Q19 box, periodic along x and y, whose two z faces are halo faces (a slab of a
    // sharded lattice): every upstream node is present, the z ones in the ghost planes, so the
    // kernels of full periodic boxes apply with z addressed through the ghost frame
    int ring;
    int full;  // every cell of the box holds a node (also where info is kept for forcing or Smagorinsky)
    FastDiv fa0, fa1;  // division by a[0] and a[1] (cell index -> box coordinates)
    // D3Q19 step launches: planes [z0, z0 + zn) of the last axis; zn = 0: every plane
    int z0, zn;
    // one-node step launches: 1 = threads numbered over each x-y plane (x fastest) instead of per
    // row, so that rows whose length is not a multiple of 32 share warps; fn0 divides by n[0].
    // 2 = the same with each plane's row-inner nodes (x = 1 .. n[0] - 2) first and the rows' end
    // nodes (x = 0, n[0] - 1) last; fn0 divides by n[0] - 2
    int flat;
    FastDiv fn0;
};

struct StepParams {
    double tau;             // relaxation time at this level
    double rho0;            // default density
    int face_kind[6];       // BcKind per face
    double bb_term[6][19];  // 6 rho0 w_o (c_o . U_face) for outgoing direction o
    const double* mrt64;    // dense M^-1 S M, reference construction order (FP64 mode)
    const double* mrt64_host;    // the same on the host (the FP64 step passes it as a kernel argument)
    const double* mrt64_d_host;  // M^-1 (I - S/2) M on the host
    double inv_tau_hi, inv_tau_lo;  // 1 / tau as an unevaluated sum (FP64 SRT: division by tau)
    float mrt_coef[19];     // (s_k - 1/tau) / |M_k|^2 per non-shear moment, 0 elsewhere (fast path)
    float omega32;          // 1/tau in FP32 (fast path)
    float inv_scale;        // reduced storage: deviation = stored * inv_scale
    float scale;
    double scale_d;         // the same scale in FP64 (1 for FP64 / FP32 storage)
    int fuse_bb;            // bounce back applied inside the step kernel (no ordered face passes needed)
    double* macro;          // rho, ux, uy, uz per cell for nodes flagged kInfoSaveMacro (else unused)
    // body forces (Guo forcing): F = const_force + force[cell] (GetAllForcesForANode,
    // lbm_solver_interface.cpp:132-144); force is dims-strided by 3, or nullptr
    const double* force;
    double const_force[3];
    int forced;             // the level collides with forcing (requires the masked layout)
    double dt;              // time step of the level, 2^-level
    const double* mrt64_d;  // dense M^-1 (I - S/2) M (FP64 forced MRT)
    // Smagorinsky: tau = tau + tau_sgs with tau_sgs from the non-equilibrium stress
    int les;
    double les_c;           // 18 Cs^2
    const float* c_node;    // learned closure: per-cell constant c (C = 18 c), or nullptr
    double conv_u[6];       // convective outflow: convection speed per face
    // FP16 / BF16 stochastic rounding: two step seeds of the level in device memory (the even
    // step reads [0] and its first thread writes [1] = [0] + 1, the odd step the other way round,
    // so no launch reads a word another thread of it writes); nullptr: round to nearest
    uint32_t* sr_seed;
};

}  // namespace zl
