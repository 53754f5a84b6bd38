// Two nodes per thread with packed FP32 pairs (fma.rn.f32x2 and friends, sm_100): the D3Q19 step
// of a full periodic box in deviation storage.  Thread t updates nodes x0 = 2t and x0 + 1 of a
// row.  Populations of the two nodes that sit side by side in a plane move as one 32-bit (FP16 /
// BF16) or 64-bit (FP32) access; the collision runs once on (node a, node b) pairs in the form of
// fused_collide.cuh, which halves its arithmetic instructions.  FP32: the one-node kernel's bits; FP16 / BF16:
// its formulas, in roundings that can differ where the one-node build contracts a product and a sum.  Requires an even row length (x0, x0 + 1 in one row, pair accesses aligned).
#pragma once
#include "aa_kernel.cuh"
#include "pair_value.cuh"

namespace zl {

// Two neighbouring slots of a plane as one access.
template <class S> struct PairIO;
template <> struct PairIO<float> {
    __device__ __forceinline__ static F2 load(const float* p) { return {__ldg(reinterpret_cast<const float2*>(p))}; }
    __device__ __forceinline__ static void store(float* p, F2 v) { *reinterpret_cast<float2*>(p) = v.v; }
    __device__ __forceinline__ static void store_sr(float* p, F2 v, uint32_t) { store(p, v); }
};
template <> struct PairIO<__half> {
    __device__ __forceinline__ static F2 load(const __half* p) {
        return {__half22float2(__ldg(reinterpret_cast<const __half2*>(p)))};
    }
    __device__ __forceinline__ static void store(__half* p, F2 v) {
        *reinterpret_cast<__half2*>(p) = __float22half2_rn(v.v);
    }
    __device__ __forceinline__ static void store_sr(__half* p, F2 v, uint32_t rbits) {
        *reinterpret_cast<uint32_t*>(p) = cvt_rs_f16x2(v.v.y, v.v.x, rbits);
    }
};
template <> struct PairIO<__nv_bfloat16> {
    __device__ __forceinline__ static F2 load(const __nv_bfloat16* p) {
        return {__bfloat1622float2(__ldg(reinterpret_cast<const __nv_bfloat162*>(p)))};
    }
    __device__ __forceinline__ static void store(__nv_bfloat16* p, F2 v) {
        *reinterpret_cast<__nv_bfloat162*>(p) = __float22bfloat162_rn(v.v);
    }
    __device__ __forceinline__ static void store_sr(__nv_bfloat16* p, F2 v, uint32_t rbits) {
        *reinterpret_cast<uint32_t*>(p) = cvt_rs_bf16x2(v.v.y, v.v.x, rbits);
    }
};

// The unforced collision of a node pair in storage S.
template <bool Mrt, class S>
__device__ __forceinline__ void fused_pair(const F2* d, F2* out, const StepParams& p) {
    fused_collide<Mrt, false, false, F2, Mrt || sizeof(S) == 2>(d, out, p, splat(0.f), (const F2*)nullptr, (F2*)nullptr);
}

// Nodes x0 and x0 + 1 of a row of a full periodic box (or a slab of one, geo.ring: z neighbours
// in the ghost planes) with an even row length.  Rows whose y or z neighbours wrap take the scalar
// node update twice.  Les: Smagorinsky (FP32 storage), the constant C per node where the learned
// closure left one.  The Smagorinsky step of one node per thread is bound by its instructions, which
// the packed collision halves.
template <class S, int Coll, bool Odd, bool Les = false>
__global__ void __launch_bounds__(256, 2) aa_pair_kernel(S* __restrict__ f, LevelGeom geo, StepParams p) {
    pdl_wait();
    pdl_trigger();
    static_assert(!Les || sizeof(S) == 4, "Smagorinsky pairs are FP32");
    using Tb = Tables<D3Q19>;
    using St = Storage<S>;
    using IO = PairIO<S>;
    constexpr int Ext = Les ? kExtLes : 0;
    const int x0 = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int y = blockIdx.y * blockDim.y + threadIdx.y, z = blockIdx.z + geo.z0;
    if (sizeof(S) == 2 && (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x | threadIdx.y) == 0)
        sr_advance(p, Odd, sr_seed(p, Odd), true);
    if (x0 >= geo.n[0] || y >= geo.n[1]) return;
    const int gz = geo.g[2];  // 1 on a slab: z rows never wrap
    if (!(y > 0 && y < geo.n[1] - 1 && (gz || (z > 0 && z < geo.n[2] - 1)))) {
        Coord c;
        c.x[0] = x0;
        c.x[1] = y;
        c.x[2] = z;
        aa_node<D3Q19, S, Coll, Odd, false, false, Ext>(f, geo, p, c);
        c.x[0] = x0 + 1;
        aa_node<D3Q19, S, Coll, Odd, false, false, Ext>(f, geo, p, c);
        return;
    }
    const int n0 = geo.n[0];
    const int row = geo.a[0] * (y + geo.a[1] * (z + gz));
    // columns x0 - 1, x0, x0 + 1, x0 + 2 of the row (x wrapped)
    S* const pc[4] = {f + (row + (x0 == 0 ? n0 - 1 : x0 - 1)), f + (row + x0), f + (row + x0 + 1),
                      f + (row + (x0 + 2 == n0 ? 0 : x0 + 2))};
    const long long st = geo.stride;
    const int a0 = geo.a[0], a01 = geo.a[0] * geo.a[1];
    auto off = [&](int q, int dy, int dz) -> long long { return q * st + (long long)(dy * a0 + dz * a01); };
    F2 pre[19], post[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        if (!Odd || q == 0) {
            pre[q] = IO::load(pc[1] + off(q, 0, 0));
        } else if (Tb::cx(q) == 0) {
            pre[q] = IO::load(pc[1] + off(Tb::opp(q), -Tb::cy(q), -Tb::cz(q)));
        } else {
            const long long o = off(Tb::opp(q), -Tb::cy(q), -Tb::cz(q));
            pre[q] = {make_float2(St::load_raw(pc[1 - Tb::cx(q)] + o), St::load_raw(pc[2 - Tb::cx(q)] + o))};
        }
    }
    if constexpr (Les) {
        F2 les_c = splat((float)p.les_c);
        if (p.c_node) {
            const float* c = p.c_node + row + x0;
            les_c = {make_float2(18.f * __ldg(c), 18.f * __ldg(c + 1))};
        }
        fused_collide<Coll == kMrt, true, false>(pre, post, p, les_c, (const F2*)nullptr, (F2*)nullptr);
    } else {
        fused_pair<Coll == kMrt, S>(pre, post, p);
    }
    if (sizeof(S) == 2 && p.sr_seed) {
        // stochastic rounding of the 16-bit stores, one random stream per node pair
        SrBits rng(sr_seed(p, Odd), (uint32_t)((row + x0) >> 1));
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            const uint32_t r = rng.next();
            if (!Odd || q == 0) {
                IO::store_sr(pc[1] + off(Tb::opp(q), 0, 0), post[q], r);
            } else if (Tb::cx(q) == 0) {
                IO::store_sr(pc[1] + off(q, Tb::cy(q), Tb::cz(q)), post[q], r);
            } else {
                const long long o = off(q, Tb::cy(q), Tb::cz(q));
                St::store_raw_sr(pc[1 + Tb::cx(q)] + o, post[q].v.x, r);
                St::store_raw_sr(pc[2 + Tb::cx(q)] + o, post[q].v.y, r ^ 0x9e3779b9u);
            }
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        if (!Odd || q == 0) {
            IO::store(pc[1] + off(Tb::opp(q), 0, 0), post[q]);
        } else if (Tb::cx(q) == 0) {
            IO::store(pc[1] + off(q, Tb::cy(q), Tb::cz(q)), post[q]);
        } else {
            const long long o = off(q, Tb::cy(q), Tb::cz(q));
            St::store_raw(pc[1 + Tb::cx(q)] + o, post[q].v.x);
            St::store_raw(pc[2 + Tb::cx(q)] + o, post[q].v.y);
        }
    }
}

}  // namespace zl
