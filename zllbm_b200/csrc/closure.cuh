// Learned LES closure: node features, the 24 -> 64 -> 64 -> 1 network on tcgen05 tensor cores,
// and the shared-memory tile layout its kernels use.
//
// The closure has no counterpart in the reference, which hard-wires Smagorinsky
// (lbm_project/les_models/lbm_les_smagorinsky.cpp:22-94).  It keeps that model's relaxation
// formula and replaces the constant: C = 18 c with c = 0.01 clamp(y, 0, 8) from the network, so
// y = 1 is Smagorinsky with Cs = 0.1 and a network that is not set (or a non-finite y) falls
// back to the configured Smagorinsky constant.
//
// Layers: Z1 = W1 x_hat + b1, A1 = gelu(Z1), Z2 = W2 A1 + b2, A2 = gelu(Z2), y = w3 . A2 + b3, with
// x_hat = (x - mean) * inv_std and gelu the tanh form 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3))).
// x_hat, W1, A1, W2 (and in training dZ2, dZ1) are BF16 tensor-core operands; everything else is FP32.
#pragma once
#include "aa_kernel.cuh"
#include "tc.cuh"

namespace zl {
namespace closure {

constexpr int kIn = 24, kHid = 64, kTile = 128;
// offsets in the flat parameter array (the zl_mlp struct)
constexpr int oW1 = 0, oB1 = oW1 + kHid * kIn, oW2 = oB1 + kHid, oB2 = oW2 + kHid * kHid, oW3 = oB2 + kHid,
              oB3 = oW3 + kHid, oMean = oB3 + 1, oInvStd = oMean + kIn, kFlat = oInvStd + kIn;
constexpr int kTrainable = oMean;
static_assert(kTrainable == 5825, "parameter count");
static_assert(oW1 % 4 == 0 && oW2 % 4 == 0 && kIn % 8 == 0 && kHid % 8 == 0, "16-byte rows of weights");

constexpr float kGeluK = 0.7978845608028654f;  // sqrt(2 / pi)
constexpr float kGeluA = 0.044715f;
constexpr float kCUnit = 0.01f;
constexpr float kYMax = 8.f;
constexpr uint32_t kWaitLimit = 1u << 22;  // mbarrier polls before a wait gives up

// ---------------------------------------------------------------- tiles (bytes, no swizzle)
// X  [128 samples x 32]: x_hat (24), a ones column (24), zeros        row groups 512 B apart
// A1 [128 samples x 80]: A1 (64), a ones column (64), zeros           1280 B
// DZ [128 samples x 128]: dZ (64), zeros (the M = 128 padding of the weight-gradient products)
// W1 [64 x 32]: W1 (24), b1 (24), zeros;  W2 [64 x 80]: W2 (64), b2 (64), zeros
// The ones columns carry the biases through the products: Z1 = [X | 1] [W1 | b1]^T, likewise Z2.
constexpr uint32_t kSboX = 512, kSboA1 = 1280, kSboDz = 2048, kSboW1 = 512, kSboW2 = 1280;
constexpr uint32_t kBytesX = 128 * kSboX / 8, kBytesA1 = 128 * kSboA1 / 8, kBytesDz = 128 * kSboDz / 8,
                   kBytesW1 = 64 * kSboW1 / 8, kBytesW2 = 64 * kSboW2 / 8;
// every descriptor stays inside its buffer
static_assert(tc::extent_kmajor(128, kSboX, 2) <= kBytesX, "X as A (K = 32)");
static_assert(tc::extent_mnmajor(32, kSboX, 8) <= kBytesX, "X as B of dW1 (N = 32, K = 128)");
static_assert(tc::extent_kmajor(128, kSboA1, 5) <= kBytesA1, "[A1 | 1] as A (K = 80)");
static_assert(tc::extent_mnmajor(80, kSboA1, 8) <= kBytesA1, "A1 as B of dW2 (N = 80, K = 128)");
static_assert(tc::extent_kmajor(128, kSboDz, 4) <= kBytesDz, "dZ2 as A of dA1 (K = 64)");
static_assert(tc::extent_mnmajor(128, kSboDz, 8) <= kBytesDz, "dZ as A of dW (M = 128, K = 128)");
static_assert(tc::extent_kmajor(64, kSboW1, 2) <= kBytesW1, "W1 as B (N = 64, K = 32)");
static_assert(tc::extent_kmajor(64, kSboW2, 5) <= kBytesW2, "[W2 | b2] as B (N = 64, K = 80)");
static_assert(tc::extent_mnmajor(64, kSboW2, 4) <= kBytesW2, "W2^T as B of dA1 (N = 64, K = 64)");

constexpr uint32_t kIdescFwd = tc::idesc_bf16(128, 64, false, false);   // X W1^T, A1 W2^T
constexpr uint32_t kIdescDa1 = tc::idesc_bf16(128, 64, false, true);    // dZ2 W2
constexpr uint32_t kIdescDw2 = tc::idesc_bf16(128, 80, true, true);     // dZ2^T [A1 | 1]
constexpr uint32_t kIdescDw1 = tc::idesc_bf16(128, 32, true, true);     // dZ1^T [X | 1]

__device__ __forceinline__ float gelu(float z, float& t) {
    t = tanhf(kGeluK * fmaf(kGeluA * z, z * z, z));
    return 0.5f * z * (1.f + t);
}
// Inference: twice the same GELU on packed BF16 pairs (the result is a BF16 operand anyway):
// z^2, 1 + a z^2, k z, k z (1 + a z^2), tanh.approx.bf16x2, z + z t -- every step rounds to BF16
// (constants a, k rounded to BF16 too).  The factor 1/2 that is missing sits in the next layer's
// weights (W2, w3), where halving is exact.
// The constants are BF16 bit patterns (a = 0x3d37, k = 0x3f4c, 1 = 0x3f80, each in both halves), so that
// no conversion runs per call.
__device__ __forceinline__ __nv_bfloat162 bf16x2_bits(uint32_t b) {
    __nv_bfloat162 v;
    memcpy(&v, &b, 4);
    return v;
}
__device__ __forceinline__ uint32_t gelu2_bf16x2(float z0, float z1) {
    const __nv_bfloat162 z = __floats2bfloat162_rn(z0, z1);
    const __nv_bfloat162 a = bf16x2_bits(0x3d373d37u), k = bf16x2_bits(0x3f4c3f4cu), one = bf16x2_bits(0x3f803f80u);
    const __nv_bfloat162 p = __hfma2(__hmul2(z, z), a, one);
    const __nv_bfloat162 arg = __hmul2(__hmul2(z, k), p);
    uint32_t t;
    asm("tanh.approx.bf16x2 %0, %1;" : "=r"(t) : "r"(*reinterpret_cast<const uint32_t*>(&arg)));
    const __nv_bfloat162 out = __hfma2(z, *reinterpret_cast<const __nv_bfloat162*>(&t), z);
    return *reinterpret_cast<const uint32_t*>(&out);
}
__device__ __forceinline__ float gelu_grad(float z, float t) {
    return fmaf(0.5f, 1.f + t, 0.5f * z * (1.f - t * t) * kGeluK * fmaf(3.f * kGeluA, z * z, 1.f));
}

__device__ __forceinline__ void st_row_chunk(uint8_t* tile, uint32_t row, uint32_t col, uint32_t sbo, const float* v) {
    *reinterpret_cast<uint4*>(tile + tc::tile_offset(row, col, sbo)) = tc::pack_bf16x8(v);
}

// Stage [W1 | b1] and [W2 | b2] as BF16 tiles and the FP32 vectors.  Eight weights of a row are two 16-byte
// loads and one core-matrix row (net comes from cudaMalloc and the rows are 96 and 256 bytes).
// Loaded past L1: a trainer's update kernel may still run when its next step's launch begins.
// scale multiplies W2 and w3 (inference: 1/2, the factor its GELU leaves out).
__device__ __forceinline__ void stage_weights(const float* __restrict__ net, uint8_t* w1s, uint8_t* w2s, float* w3,
                                              float* b3, float* mean, float* istd, float scale) {
    const int tid = threadIdx.x, nt = blockDim.x;
    auto chunk = [&](uint8_t* tile, uint32_t sbo, int row, int col, const float* src, float k) {
        const float4 lo = __ldcg(reinterpret_cast<const float4*>(src)), hi = __ldcg(reinterpret_cast<const float4*>(src) + 1);
        const float v[8] = {k * lo.x, k * lo.y, k * lo.z, k * lo.w, k * hi.x, k * hi.y, k * hi.z, k * hi.w};
        st_row_chunk(tile, row, col, sbo, v);
    };
#pragma unroll 4
    for (int e = tid; e < kHid * 8; e += nt) chunk(w2s, kSboW2, e >> 3, 8 * (e & 7), net + oW2 + 8 * e, scale);
    for (int e = tid; e < kHid * 3; e += nt) {
        const int j = e / 3, c = e - 3 * j;
        chunk(w1s, kSboW1, j, 8 * c, net + oW1 + 8 * e, 1.f);
    }
    for (int j = tid; j < kHid; j += nt) {
        float v[8] = {__ldcg(net + oB1 + j), 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        st_row_chunk(w1s, j, kIn, kSboW1, v);
        v[0] = __ldcg(net + oB2 + j);
        st_row_chunk(w2s, j, kHid, kSboW2, v);
        v[0] = 0.f;
        st_row_chunk(w2s, j, kHid + 8, kSboW2, v);
    }
    for (int e = tid; e < kHid; e += nt) w3[e] = scale * __ldcg(net + oW3 + e);
    for (int e = tid; e < kIn; e += nt) {
        mean[e] = __ldcg(net + oMean + e);
        istd[e] = __ldcg(net + oInvStd + e);
    }
    if (tid == 0) *b3 = __ldcg(net + oB3);
}

// This thread's row of an A1 tile's constant columns (the ones column and the zero padding).
__device__ __forceinline__ void stage_ones(uint8_t* a1s) {
    const int tid = threadIdx.x & (kTile - 1);
    float v[8] = {1.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    st_row_chunk(a1s, tid, 64, kSboA1, v);
    v[0] = 0.f;
    st_row_chunk(a1s, tid, 72, kSboA1, v);
}

// One warp polls the MMA's mbarrier; the others wait at the block barrier, which issues nothing
// while it waits (polling from every warp takes issue slots from the other resident blocks).
__device__ __forceinline__ bool wait_mma(uint64_t* bar, uint32_t& phase, int* err) {
    bool ok = true;
    if (threadIdx.x < 32) ok = tc::mbar_wait(bar, phase, kWaitLimit);
    const bool failed = __syncthreads_or(!ok) != 0;
    if (!failed) phase ^= 1u;
    if (failed && threadIdx.x == 0) atomicExch(err, 1);
    tc::fence_after_sync();
    return !failed;
}

// Inference of N tiles of 128 rows: X (this thread's row written by the caller) -> y of this thread's
// row.  64 TMEM columns per tile (Z1, then Z2).  A tile's X occupies the first 32 columns of its
// A1 tile, whose constant columns lie beyond: X is dead once the first product is done, so the tile
// needs no memory of its own.  Returns false if a tensor-core wait gave up.
static_assert(tc::extent_kmajor(128, kSboA1, 2) <= kBytesA1, "X in the A1 tile as A (K = 32)");
struct InferTile {
    uint8_t* a1s;
    uint32_t sA1, sW1, sW2, tmem, lane_addr;
    uint64_t* bar;
    const float* w3;  // halved
    float b3;
};

// 128 N threads, a row each.
template <int N>
__device__ __forceinline__ bool infer_tiles(const InferTile& it, uint32_t& phase, int* err, float& y) {
    const int tid = threadIdx.x, row = tid & (kTile - 1), tile = tid / kTile;
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0) {
        tc::fence_after_sync();
        for (int t = 0; t < N; ++t)
            for (int s = 0; s < 2; ++s)
                tc::mma_bf16(it.tmem + kHid * t, tc::desc_kmajor(it.sA1 + kBytesA1 * t, kSboA1, s),
                             tc::desc_kmajor(it.sW1, kSboW1, s), kIdescFwd, s > 0);
        tc::commit(it.bar);
    }
    if (!wait_mma(it.bar, phase, err)) return false;
    // (the loops over column halves stay loops: unrolled, the step kernel's body outgrows the instruction
    // cache)
#pragma unroll 1
    for (int h = 2 * tile; h < 2 * tile + 2; ++h) {  // half h: tile h / 2, columns 32 (h % 2) ..
        float v[32];
        tc::tmem_ld32(it.tmem + it.lane_addr + 32 * h, v);
        uint8_t* dst = it.a1s + kBytesA1 * (h >> 1) + tc::tile_offset(row, 32 * (h & 1), kSboA1);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint4 o;
            o.x = gelu2_bf16x2(v[8 * k], v[8 * k + 1]);
            o.y = gelu2_bf16x2(v[8 * k + 2], v[8 * k + 3]);
            o.z = gelu2_bf16x2(v[8 * k + 4], v[8 * k + 5]);
            o.w = gelu2_bf16x2(v[8 * k + 6], v[8 * k + 7]);
            *reinterpret_cast<uint4*>(dst + 128 * k) = o;
        }
    }
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0) {
        tc::fence_after_sync();
        for (int t = 0; t < N; ++t)
            for (int s = 0; s < 5; ++s)
                tc::mma_bf16(it.tmem + kHid * t, tc::desc_kmajor(it.sA1 + kBytesA1 * t, kSboA1, s),
                             tc::desc_kmajor(it.sW2, kSboW2, s), kIdescFwd, s > 0);
        tc::commit(it.bar);
    }
    if (!wait_mma(it.bar, phase, err)) return false;
    float2 acc = make_float2(it.b3, 0.f);
#pragma unroll 1
    for (int h = 2 * tile; h < 2 * tile + 2; ++h) {
        float v[32];
        tc::tmem_ld32(it.tmem + it.lane_addr + 32 * h, v);
        const float* w3 = it.w3 + 32 * (h & 1);
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            // w3 four at a time (one 128-bit shared load, the same address for every thread)
            const float4 w = *reinterpret_cast<const float4*>(w3 + i);
            const uint32_t g0 = gelu2_bf16x2(v[i], v[i + 1]), g1 = gelu2_bf16x2(v[i + 2], v[i + 3]);
            const float2 a0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g0));
            const float2 a1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g1));
            acc = __ffma2_rn(a0, make_float2(w.x, w.y), acc);
            acc = __ffma2_rn(a1, make_float2(w.z, w.w), acc);
        }
    }
    y = acc.x + acc.y;
    return true;
}

// ---------------------------------------------------------------- features
// The 24 inputs of a D3Q19 node from its density and non-equilibrium populations (unscaled):
// the 19 MRT moments of f - feq over rho (the conserved four are zero), tr S, S:S, tr(Sd^3),
// |Sd| and the Cs = 0.1 Smagorinsky increment, S = -3 Pi / (2 rho tau0).
// spp (optional) receives sqrt(2 Pi:Pi), the stress norm of the relaxation formula.
// `unscale` multiplies neq first (the inverse storage scale for scaled deviations).
__device__ __forceinline__ void features(float rho, const float* neq, float tau0, float* x, float* spp = nullptr,
                                         float unscale = 1.f) {
    // moments M neq through sums / differences of opposite pairs (rows of lbm_d3q19.h:98-167)
    const float* n = neq;
    const float S1 = n[1] + n[2], D1 = n[1] - n[2];
    const float S2 = n[3] + n[4], D2 = n[3] - n[4];
    const float S3 = n[5] + n[6], D3 = n[5] - n[6];
    const float S4 = n[7] + n[10], D4 = n[7] - n[10];
    const float S5 = n[8] + n[9], D5 = n[8] - n[9];
    const float S6 = n[11] + n[14], D6 = n[11] - n[14];
    const float S7 = n[12] + n[13], D7 = n[12] - n[13];
    const float S8 = n[15] + n[18], D8 = n[15] - n[18];
    const float S9 = n[16] + n[17], D9 = n[16] - n[17];
    const float Sa = S1 + S2 + S3;
    const float Sxy = S4 + S5, Sxz = S6 + S7, Syz = S8 + S9;
    const float Sd = Sxy + Sxz + Syz;
    const float X1 = D4 - D5, X2 = D6 - D7, Y1 = D4 + D5, Y2 = D8 - D9, Z1 = D6 + D7, Z2 = D8 + D9;
    const float ir = unscale / rho;
    // mass and momentum of f - feq vanish (the collision conserves them): exact zero inputs,
    // not rounding noise that an input normalisation would amplify
    x[0] = 0.f;
    x[3] = 0.f;
    x[5] = 0.f;
    x[7] = 0.f;
    x[1] = (-30.f * n[0] - 11.f * Sa + 8.f * Sd) * ir;
    x[2] = (12.f * n[0] - 4.f * Sa + Sd) * ir;
    x[4] = (-4.f * D1 + X1 + X2) * ir;
    x[6] = (-4.f * D2 + Y1 + Y2) * ir;
    x[8] = (-4.f * D3 + Z1 + Z2) * ir;
    x[9] = (2.f * S1 - S2 - S3 + Sxy + Sxz - 2.f * Syz) * ir;
    x[10] = (-4.f * S1 + 2.f * (S2 + S3) + Sxy + Sxz - 2.f * Syz) * ir;
    x[11] = (S2 - S3 + Sxy - Sxz) * ir;
    x[12] = (-2.f * S2 + 2.f * S3 + Sxy - Sxz) * ir;
    x[13] = (S4 - S5) * ir;
    x[14] = (S8 - S9) * ir;
    x[15] = (S6 - S7) * ir;
    x[16] = (X1 - X2) * ir;
    x[17] = (-Y1 + Y2) * ir;
    x[18] = (Z1 - Z2) * ir;
    // non-equilibrium stress xx yy zz xy xz yz
    const float p[6] = {unscale * (S1 + S4 + S5 + S6 + S7), unscale * (S2 + S4 + S5 + S8 + S9),
                        unscale * (S3 + S6 + S7 + S8 + S9), unscale * (S4 - S5), unscale * (S6 - S7),
                        unscale * (S8 - S9)};
    const float k = -1.5f / (rho * tau0);
    float s[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) s[i] = k * p[i];
    const float tr = s[0] + s[1] + s[2];
    const float a = s[0] - tr / 3.f, b = s[1] - tr / 3.f, c = s[2] - tr / 3.f, d = s[3], e = s[4], g = s[5];
    const float ss = s[0] * s[0] + s[1] * s[1] + s[2] * s[2] + 2.f * (d * d + e * e + g * g);
    const float det = a * (b * c - g * g) - d * (d * c - g * e) + e * (d * g - b * e);
    const float sd2 = a * a + b * b + c * c + 2.f * (d * d + e * e + g * g);
    const float pp = p[0] * p[0] + p[1] * p[1] + p[2] * p[2] + 2.f * (p[3] * p[3] + p[4] * p[4] + p[5] * p[5]);
    x[19] = tr;
    x[20] = ss;
    x[21] = 3.f * det;
    x[22] = sqrtf(2.f * sd2);
    const float s2 = sqrtf(2.f * pp);
    x[23] = 0.5f * (sqrtf(tau0 * tau0 + 18.f * kCUnit * s2) - tau0);
    if (spp) *spp = s2;
}

// The same features of a node from its deviations d (scaled units), in the closed
// forms of fused_collide: the relaxed moments and the stress of f - feq from the pair sums of d and the
// equilibrium's moments, no per-direction feq.  m9 = 2 Pxx - Pyy - Pzz, m11 = Pyy - Pzz, m13..15 the off-diagonal
// stress.  inv_rho: 1 / rho, correctly rounded, for the collision.
__device__ __forceinline__ void fused_features(const F1* d, const StepParams& p, float tau0, F1* x, F1& inv_rho) {
    using V = F1;
    auto S = [](float s) { return splat_as<V>(s); };
    const V S1 = d[1] + d[2], D1 = d[1] - d[2];
    const V S2 = d[3] + d[4], D2 = d[3] - d[4];
    const V S3 = d[5] + d[6], D3 = d[5] - d[6];
    const V S4 = d[7] + d[10], D4 = d[7] - d[10];
    const V S5 = d[8] + d[9], D5 = d[8] - d[9];
    const V S6 = d[11] + d[14], D6 = d[11] - d[14];
    const V S7 = d[12] + d[13], D7 = d[12] - d[13];
    const V S8 = d[15] + d[18], D8 = d[15] - d[18];
    const V S9 = d[16] + d[17], D9 = d[16] - d[17];
    const V S23 = S2 + S3, Sa = S1 + S23;
    const V Sxy = S4 + S5, Sxz = S6 + S7, Syz = S8 + S9;
    const V Sd = (Sxy + Sxz) + Syz;
    const V drho = (d[0] + Sa) + Sd;
    const V X1 = D4 - D5, X2 = D6 - D7, Y1 = D4 + D5, Y2 = D8 - D9, Z1 = D6 + D7, Z2 = D8 + D9;
    const V X12 = X1 + X2, Y12 = Y1 + Y2, Z12 = Z1 + Z2;
    const V zero = S(0.f), is = S(p.inv_scale);
    const V rho = vfma(drho, is, S(1.f));
    const V r = each(rho, [](float v) { return __frcp_rn(v); });
    inv_rho = r;
    const V k = is * r;  // unscaled over rho
    const V ux = (D1 + X12) * k, uy = (D2 + Y12) * k, uz = (D3 + Z12) * k;
    const V ux2 = ux * ux, uy2 = uy * uy, uz2 = uz * uz;
    const V usq = (ux2 + uy2) + uz2;
    const V G = S(p.scale) * rho, nG = zero - G, Gu = G * usq, hG = S(0.5f) * G;
    const V t = drho * S(1.f / 3.f);
    const V pxx = vfma(nG, ux2, (S1 + (Sxy + Sxz)) - t);
    const V pyy = vfma(nG, uy2, (S2 + (Sxy + Syz)) - t);
    const V pzz = vfma(nG, uz2, (S3 + (Sxz + Syz)) - t);
    const V pxy = vfma(nG, ux * uy, S4 - S5);
    const V pxz = vfma(nG, ux * uz, S6 - S7);
    const V pyz = vfma(nG, uy * uz, S8 - S9);
    // mass and momentum of f - feq vanish: exact zero inputs
    x[0] = zero;
    x[3] = zero;
    x[5] = zero;
    x[7] = zero;
    x[1] = (S(19.f) * ((Sd - d[0]) - Gu)) * k;
    x[2] = vfma(S(5.5f), Gu, vfma(S(9.f), d[0], vfma(S(-7.f), Sa, S(-2.f) * Sd))) * k;
    x[4] = vfma(S(-10.f / 3.f), D1, S(5.f / 3.f) * X12) * k;
    x[6] = vfma(S(-10.f / 3.f), D2, S(5.f / 3.f) * Y12) * k;
    x[8] = vfma(S(-10.f / 3.f), D3, S(5.f / 3.f) * Z12) * k;
    x[9] = vfma(S(2.f), pxx, zero - (pyy + pzz)) * k;
    x[10] = vfma(hG, vfma(S(3.f), ux2, zero - usq),
                 vfma(S(-4.f), S1, vfma(S(2.f), S23, (Sxy + Sxz) - S(2.f) * Syz))) * k;
    x[11] = (pyy - pzz) * k;
    x[12] = vfma(hG, uy2 - uz2, vfma(S(2.f), S3 - S2, Sxy - Sxz)) * k;
    x[13] = pxy * k;
    x[14] = pyz * k;
    x[15] = pxz * k;
    x[16] = (X1 - X2) * k;
    x[17] = (Y2 - Y1) * k;
    x[18] = (Z1 - Z2) * k;
    // strain S = -3 Pi / (2 rho tau0) and its invariants
    const V ks = S(-1.5f / tau0) * k;
    const V sxx = ks * pxx, syy = ks * pyy, szz = ks * pzz, sxy = ks * pxy, sxz = ks * pxz, syz = ks * pyz;
    const V tr = (sxx + syy) + szz, third = tr * S(1.f / 3.f);
    const V a = sxx - third, b = syy - third, c = szz - third;
    const V off = vfma(syz, syz, vfma(sxz, sxz, sxy * sxy)), off2 = S(2.f) * off;
    const V ss = vfma(szz, szz, vfma(syy, syy, vfma(sxx, sxx, off2)));
    const V sd2 = vfma(c, c, vfma(b, b, vfma(a, a, off2)));
    const V det = vfma(a, vfma(b, c, zero - syz * syz),
                       vfma(zero - sxy, vfma(sxy, c, zero - syz * sxz), sxz * vfma(sxy, syz, zero - b * sxz)));
    const V pp = vfma(pzz, pzz, vfma(pyy, pyy, pxx * pxx));
    const V po = vfma(pyz, pyz, vfma(pxz, pxz, pxy * pxy));
    x[19] = tr;
    x[20] = ss;
    x[21] = S(3.f) * det;
    x[22] = each(S(2.f) * sd2, [](float v) { return __fsqrt_rn(v); });
    const V s2 = each((is * is) * (S(2.f) * vfma(S(2.f), po, pp)), [](float v) { return __fsqrt_rn(v); });
    const V root = each(vfma(S(18.f * kCUnit), s2, S(tau0 * tau0)), [](float v) { return __fsqrt_rn(v); });
    x[23] = S(0.5f) * (root - S(tau0));
}

}  // namespace closure
}  // namespace zl
