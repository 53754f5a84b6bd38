// Launchers of the fused step (one parity of the AA pattern) and of the batched multi-level
// step (one set of extensions) for one (storage, lattice, collision).  Only step_inst.cu includes this file: it is
// compiled once per combination, each with an explicit instantiation, so the build compiles the
// step kernel variants in parallel translation units.  The launch sets of launch.cuh call them
// through the declarations there.
#pragma once
#include <cstring>
#include "f64_kernel.cuh"
#include "launch.cuh"

namespace zl {
namespace step_impl {

// D3Q19 with the default block shape and rows whose length is not a multiple of 32: the threads
// are numbered over each x-y plane (no warp holds the few nodes left at a row's end on its own),
// rows' end nodes last when the x axis is bounded; a level of a few thousand nodes takes one-warp
// blocks, so that its launch still reaches every SM.
// (Measured: the flow past a cube 3 % faster.)  D2Q9 levels take blocks of 32 x 4 nodes: 257^2 is 771
// blocks of 128 along its rows, a wave and a bit of the FP64 step, and 585 of 32 x 4 (FP64, per step:
// 257^2 5.0 -> 3.8 us, 385^2 6.5 -> 5.8, 1025^2 27.7 -> 26.0; numbering threads over the plane 4.1, 6.3, 25.6,
// but 3.6 instead of 3.2 at 33^2).
template <class S, class L, int C, bool O, bool B, bool M, int X>
cudaError_t launch_one(S* f, const LevelGeom& geo, const StepParams& p, dim3 g, dim3 b, cudaStream_t s) {
    // FP64 MRT with Smagorinsky keeps the general kernel, which builds the matrix node by node
    if constexpr (sizeof(S) == 8 && !(C == kMrt && (X & kExtLes))) {
        MrtArg<L::kQ, C == kMrt, (X & kExtForce) != 0> m;
        if constexpr (C == kMrt) std::memcpy(m.a, p.mrt64_host, sizeof(m.a));
        if constexpr (C == kMrt && (X & kExtForce)) std::memcpy(m.b, p.mrt64_d_host, sizeof(m.b));
        ZL_LAUNCH_DEP(aa_step_f64_kernel<L, C, O, B, M, X>, g, b, 0, s, f, geo, p, m);
    } else {
        ZL_LAUNCH_DEP(aa_step_kernel<L, S, C, O, B, M, X>, g, b, 0, s, f, geo, p);
    }
    return cudaGetLastError();
}

template <class S, class L, int C, bool O, bool B, bool M, int X = 0>
cudaError_t step_one(S* f, const LevelGeom& level, const StepParams& p, cudaStream_t s) {
    LevelGeom geo = level;
    // a shape of pairs chosen before the level stopped being one for the pair kernel
    if (geo.block[0] < 0) geo.block[0] = geo.block[1] = 0;
    dim3 g, b;
    step_shape(geo, L::kDims, g, b);
    const bool default_shape = geo.block[0] == 0 || geo.block[0] == kRowKernelBlockX;
    const long long plane = (long long)geo.n[0] * geo.n[1];
    if (L::kDims == 2 && default_shape) {
        b = dim3(32, 4);
        g = dim3((geo.n[0] + 31) / 32, (geo.n[1] + 3) / 4);
    }
    if (L::kDims == 3 && default_shape && (geo.n[0] & 31) && plane < (1ll << 31)) {
        LevelGeom fg = geo;
        // a non-periodic x axis: every row's two end nodes patch missing upstream values, and
        // numbered in row order they would put the patch path into most warps of a plane; the
        // threads take the rows' inner nodes first and the end nodes last (a few warps per plane)
        const bool ends_last = (B || M) && !geo.periodic[0] && geo.n[0] >= 3;
        fg.flat = ends_last ? 2 : 1;
        fg.fn0 = FastDiv::make((uint32_t)(ends_last ? geo.n[0] - 2 : geo.n[0]));
        const unsigned bs = plane * g.z >= 148ll * 128 * 8 ? 128u : 32u;
        return launch_one<S, L, C, O, B, M, X>(f, fg, p, dim3((unsigned)((plane + bs - 1) / bs), 1, g.z), dim3(bs), s);
    }
    return launch_one<S, L, C, O, B, M, X>(f, geo, p, g, b, s);
}

// Two nodes per thread; Les: Smagorinsky.  The default shape is 128 threads, as wide as leaves the fewest lanes
// idle past a row's n0 / 2 pairs (264 x 160 x 128 MRT: 163 us per step with 128 x 1, 154 with 32 x 4).
template <class S, int C, bool O, bool Les>
cudaError_t step_pair(S* f, const LevelGeom& geo, const StepParams& p, cudaStream_t s) {
    if constexpr (Storage<S>::kDeviation) {
        if ((geo.n[0] & 1) || (geo.stride & 1)) {
            // pair accesses need an even row length and plane stride: scalar kernel instead
            LevelGeom g1 = geo;
            g1.block[0] = g1.block[1] = 0;
            return step_one<S, D3Q19, C, O, false, false>(f, g1, p, s);
        }
        LevelGeom pg = geo;
        if (geo.block[0] == 0) {
            const int bx = pair_block_x(geo.n[0]);
            pg.block[0] = -bx;
            pg.block[1] = 128 / bx;
        }
        dim3 g, b;
        step_shape(pg, 3, g, b);
        ZL_LAUNCH_DEP(aa_pair_kernel<S, C, O, Les>, g, b, 0, s, f, geo, p);
        return cudaGetLastError();
    }
    return cudaErrorInvalidValue;
}

template <class S, int C, bool O>
cudaError_t step_row(S* f, const LevelGeom& geo, const StepParams& p, cudaStream_t s) {
    if constexpr (sizeof(S) == 2) {
        const int v = row_kernel_width(geo);
        const int rows = geo.block[1];
        if (v == 0 || rows < 1 || rows > 4) return cudaErrorInvalidValue;
        const dim3 b(32 * rows), g((geo.n[1] + rows - 1) / rows, geo.zn > 0 ? geo.zn : geo.n[2]);
        if (v == 8) ZL_LAUNCH_DEP(aa_row_kernel<S, C, O, 8>, g, b, 0, s, f, geo, p);
        else ZL_LAUNCH_DEP(aa_row_kernel<S, C, O, 4>, g, b, 0, s, f, geo, p);
        return cudaGetLastError();
    }
    return cudaErrorInvalidValue;
}

}  // namespace step_impl

template <class S, class L, int C, bool O>
cudaError_t step_lco(bool bnd, bool masked, S* f, const LevelGeom& geo, const StepParams& p, cudaStream_t s) {
    using namespace step_impl;
    if constexpr (L::kDims == 3) {
        if (geo.block[0] == kRowKernelBlockX && row_eligible(3, bnd, masked, p, (int)sizeof(S), geo))
            return step_row<S, C, O>(f, geo, p, s);
        if (geo.block[0] < 0 && pair_eligible(3, bnd, masked, p, (int)sizeof(S), geo))
            return step_pair<S, C, O, false>(f, geo, p, s);
        if constexpr (sizeof(S) == 4) {
            if (pair_default(3, C == kMrt, p, (int)sizeof(S), geo) ||
                (geo.block[0] < 0 && pair_les_eligible(3, p, (int)sizeof(S), geo)))
                return p.les ? step_pair<S, C, O, true>(f, geo, p, s) : step_pair<S, C, O, false>(f, geo, p, s);
        }
    }
    if (p.forced || p.les) {
        if (!masked) return cudaErrorInvalidValue;
        if (p.forced && p.les) return step_one<S, L, C, O, true, true, kExtForce | kExtLes>(f, geo, p, s);
        if (p.forced) return step_one<S, L, C, O, true, true, kExtForce>(f, geo, p, s);
        return step_one<S, L, C, O, true, true, kExtLes>(f, geo, p, s);
    }
    if (masked) return step_one<S, L, C, O, true, true>(f, geo, p, s);
    if (bnd) return step_one<S, L, C, O, true, false>(f, geo, p, s);
    return step_one<S, L, C, O, false, false>(f, geo, p, s);
}

template <class S, class L, int C, int X>
cudaError_t batch_lcx(const LevelBatch& b, cudaStream_t s) {
    const long long total = b.first[b.count];
    if (total <= 0) return cudaSuccess;
    const long long want = (total + kBatchThreads - 1) / kBatchThreads, cap = 148 * 6;
    const unsigned blocks = (unsigned)(want < cap ? want : cap);
    aa_batch_kernel<L, S, C, X><<<blocks, kBatchThreads, 0, s>>>(b);
    return cudaGetLastError();
}

}  // namespace zl
