// Learned LES closure on the device: the fused forward + backward tensor-core training kernel,
// the Adam update, the tensor-core forward pass, and the kernels that build training data from
// a fine level (box filter, subgrid-stress targets, features).  Full-box level I/O (set
// equilibrium, read macros from dense device arrays) lives here too.
//
// None of this has a counterpart in the reference; its relaxation formula is the reference's
// Smagorinsky increment (lbm_project/les_models/lbm_les_smagorinsky.cpp:22-94).
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "closure.cuh"
#include "closure_launch.cuh"
#include "persistent_grid.cuh"
#include "zllbm_b200.h"

namespace zl {
namespace closure {

// ---------------------------------------------------------------- training
// Shared memory of the training kernel (bytes): two tiles, the weights, FP32 vectors and sums
constexpr uint32_t kTrTiles = 2, kTrThreads = kTrTiles * kTile;
constexpr uint32_t kTrX = 0, kTrA1 = kTrX + kTrTiles * kBytesX, kTrDz2 = kTrA1 + kTrTiles * kBytesA1,
                   kTrDz1 = kTrDz2 + kTrTiles * kBytesDz, kTrW1 = kTrDz1 + kTrTiles * kBytesDz, kTrW2 = kTrW1 + kBytesW1,
                   kTrF = kTrW2 + kBytesW2, kTrSums = kTrF + 2048, kTrBar = kTrSums + kTrThreads / 32 * kHid * 4,
                   kTrSmem = kTrBar + 64;
static_assert(kTrSmem <= 227 * 1024, "one CTA per SM");
// TMEM columns: per tile Z1, then per tile Z2 (later dA1), then dW2 | db2 (80) and dW1 | db1 (32)
constexpr uint32_t kTmemCols = 512, kColZ1 = 0, kColZ2 = kTrTiles * 64, kColDw2 = 2 * kTrTiles * 64,
                   kColDw1 = kColDw2 + 80;

// One CTA of 256 threads takes two tiles of 128 samples at a time (thread = sample = TMEM lane of its
// tile).  Per tile:
//   MMA1  Z1 = X W1^T               MMA2  Z2 = A1 W2^T
//   MMA3  dA1 = dZ2 W2              MMA4  [dW2 | db2] += dZ2^T [A1 | 1]
//   MMA5  [dW1 | db1] += dZ1^T [X | 1]
// with the epilogues (bias, GELU, output, loss, dZ) on the CUDA cores between them.  The weight
// gradients accumulate in TMEM over the CTA's tiles, one after another, and are added to `grad` once at
// the end.
//
// Bound by the latency of a tile's chain (five MMA rounds, 128 tanh per thread between them): two tiles
// share each round's waits, each activation's tanh is kept in a register for the backward pass, and the
// sums of dw3 over a warp's samples are one recursive halving per 16 columns.  Eight steps of 37,888 samples
// and the read-back of gradients and weights: 900 us with one tile of 128 threads at a time, recomputed tanh
// and a butterfly per column, 280 now.  (Two CTAs of one tile per SM instead: 310 us, and other partial sums
// of the gradients, which BF16 operands carry on from step to step.)
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums of 16 values over a warp's lanes by recursive halving: 16 shuffles (a butterfly per value: 80).
// Lane l returns the sum of value (l >> 1).
__device__ __forceinline__ float warp_sum16(const float* in, int lane) {
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = in[i];
#pragma unroll
    for (int o = 16, n = 8; n > 0; o >>= 1, n >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float keep = up ? v[n + i] : v[i], give = up ? v[i] : v[n + i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

__global__ void __launch_bounds__(kTrThreads, 1) mlp_train_kernel(const float* __restrict__ net,
                                                                  const float* __restrict__ x,
                                                                  const float* __restrict__ target, long long n,
                                                                  float inv_n, float* __restrict__ grad,
                                                                  float* __restrict__ loss, int* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, slot = tid / kTile, row = tid & (kTile - 1);
    float* fs = reinterpret_cast<float*>(sm + kTrF);
    float *w3 = fs + 128, *b3 = fs + 192, *mean = fs + 200, *istd = fs + 224;
    float* red = fs + 256;  // db3, loss
    float* sums = reinterpret_cast<float*>(sm + kTrSums);  // dw3 of each warp's samples
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kTrBar);
    uint32_t* tbase = reinterpret_cast<uint32_t*>(sm + kTrBar + 8);
    uint8_t *xs = sm + kTrX + slot * kBytesX, *a1s = sm + kTrA1 + slot * kBytesA1, *dz2s = sm + kTrDz2 + slot * kBytesDz,
            *dz1s = sm + kTrDz1 + slot * kBytesDz;
    pdl_wait();

    stage_weights(net, sm + kTrW1, sm + kTrW2, w3, b3, mean, istd, 1.f);
    stage_ones(a1s);
    if (tid < 2) red[tid] = 0.f;
    {
        // the zero halves of the dZ tiles
        const float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int c = 64; c < 128; c += 8) {
            st_row_chunk(dz2s, row, c, kSboDz, v);
            st_row_chunk(dz1s, row, c, kSboDz, v);
        }
    }
    if (warp == 0) tc::tmem_alloc(tbase, kTmemCols);
    if (tid == 0) tc::mbar_init(bar, 1);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tbase;
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t z1 = tmem + lane_addr + kColZ1 + 64 * slot, z2 = tmem + lane_addr + kColZ2 + 64 * slot;
    const uint32_t sX = tc::smem_u32(sm + kTrX), sA1 = tc::smem_u32(sm + kTrA1), sDz2 = tc::smem_u32(sm + kTrDz2),
                   sDz1 = tc::smem_u32(sm + kTrDz1), sW1 = tc::smem_u32(sm + kTrW1), sW2 = tc::smem_u32(sm + kTrW2);
    uint32_t phase = 0;
    float loss_acc = 0.f, db3_acc = 0.f, dw3 = 0.f;  // dw3: of column tid, in the first 64 threads
    bool first = true, ok = true;
    const bool x16 = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;  // 96-byte rows of a 16-byte aligned array
    const long long tiles = (n + kTile - 1) / kTile;

    // the CTA's tiles are blockIdx.x + k gridDim.x; two at a time, in that order in the weight gradients
    for (long long tile0 = blockIdx.x; tile0 < tiles && ok; tile0 += (long long)kTrTiles * gridDim.x) {
        const int active = tile0 + gridDim.x < tiles ? 2 : 1;
        const long long g = (tile0 + (long long)slot * gridDim.x) * kTile + row;
        const bool valid = slot < active && g < n;
        {
            float v[32];
            if (valid && x16) {
                const float4* x4 = reinterpret_cast<const float4*>(x + g * kIn);
#pragma unroll
                for (int k = 0; k < kIn / 4; ++k) {
                    const float4 r = __ldg(x4 + k);
                    v[4 * k] = r.x;
                    v[4 * k + 1] = r.y;
                    v[4 * k + 2] = r.z;
                    v[4 * k + 3] = r.w;
                }
            } else {
#pragma unroll
                for (int k = 0; k < kIn; ++k) v[k] = valid ? x[g * kIn + k] : 0.f;
            }
#pragma unroll
            for (int k = 0; k < kIn; ++k) v[k] = valid ? (v[k] - mean[k]) * istd[k] : 0.f;
            v[24] = 1.f;
#pragma unroll
            for (int k = 25; k < 32; ++k) v[k] = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) st_row_chunk(xs, row, 8 * c, kSboX, v + 8 * c);
        }
        const float t = valid ? target[g] : 0.f;

        // MMA1: Z1 = [X | 1] [W1 | b1]^T
        tc::fence_proxy_async();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            for (int a = 0; a < active; ++a)
                for (int s = 0; s < 2; ++s)
                    tc::mma_bf16(tmem + kColZ1 + 64 * a, tc::desc_kmajor(sX + a * kBytesX, kSboX, s),
                                 tc::desc_kmajor(sW1, kSboW1, s), kIdescFwd, s > 0);
            tc::commit(bar);
        }
        if (!(ok = wait_mma(bar, phase, err))) break;
        float th1[kHid], th2[kHid];  // tanh of the two layers' GELUs, for the backward pass
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float v[16];
            tc::tmem_ld16(z1 + 16 * c, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = gelu(v[i], th1[16 * c + i]);
            st_row_chunk(a1s, row, 16 * c, kSboA1, v);
            st_row_chunk(a1s, row, 16 * c + 8, kSboA1, v + 8);
        }

        // MMA2: Z2 = [A1 | 1] [W2 | b2]^T
        tc::fence_proxy_async();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            for (int a = 0; a < active; ++a)
                for (int s = 0; s < 5; ++s)
                    tc::mma_bf16(tmem + kColZ2 + 64 * a, tc::desc_kmajor(sA1 + a * kBytesA1, kSboA1, s),
                                 tc::desc_kmajor(sW2, kSboW2, s), kIdescFwd, s > 0);
            tc::commit(bar);
        }
        if (!(ok = wait_mma(bar, phase, err))) break;
        float y = *b3;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float v[16];
            tc::tmem_ld16(z2 + 16 * c, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) y = fmaf(gelu(v[i], th2[16 * c + i]), w3[16 * c + i], y);
        }
        const float e = valid ? y - t : 0.f;
        loss_acc = fmaf(e, e, loss_acc);
        const float dy = 2.f * e * inv_n;
        db3_acc += dy;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float v[16], g3[16];
            tc::tmem_ld16(z2 + 16 * c, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int j = 16 * c + i;
                const float z = v[i], t2 = th2[j];
                g3[i] = valid ? dy * (0.5f * z * (1.f + t2)) : 0.f;
                v[i] = valid ? dy * w3[j] * gelu_grad(z, t2) : 0.f;
            }
            const float s = warp_sum16(g3, lane);
            if (!(lane & 1)) sums[warp * kHid + 16 * c + (lane >> 1)] = s;
            st_row_chunk(dz2s, row, 16 * c, kSboDz, v);
            st_row_chunk(dz2s, row, 16 * c + 8, kSboDz, v + 8);
        }

        // MMA3: dA1 = dZ2 W2 (into the Z2 columns), MMA4: [dW2 | db2] += dZ2^T [A1 | 1]
        tc::fence_proxy_async();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            for (int a = 0; a < active; ++a) {
                for (int s = 0; s < 4; ++s)
                    tc::mma_bf16(tmem + kColZ2 + 64 * a, tc::desc_kmajor(sDz2 + a * kBytesDz, kSboDz, s),
                                 tc::desc_mnmajor(sW2, kSboW2, s), kIdescDa1, s > 0);
                for (int s = 0; s < 8; ++s)
                    tc::mma_bf16(tmem + kColDw2, tc::desc_mnmajor(sDz2 + a * kBytesDz, kSboDz, s),
                                 tc::desc_mnmajor(sA1 + a * kBytesA1, kSboA1, s), kIdescDw2, !first || a > 0 || s > 0);
            }
            tc::commit(bar);
        }
        if (tid < kHid) {
            // the warps' dw3 sums in order (behind the barrier above; the next ones are written behind others)
            for (int w = 0; w < 4 * active; ++w) dw3 += sums[w * kHid + tid];
        }
        if (!(ok = wait_mma(bar, phase, err))) break;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float da[16], z[16];
            tc::tmem_ld16(z2 + 16 * c, da);
            tc::tmem_ld16(z1 + 16 * c, z);
#pragma unroll
            for (int i = 0; i < 16; ++i) da[i] *= gelu_grad(z[i], th1[16 * c + i]);
            st_row_chunk(dz1s, row, 16 * c, kSboDz, da);
            st_row_chunk(dz1s, row, 16 * c + 8, kSboDz, da + 8);
        }

        // MMA5: [dW1 | db1] += dZ1^T [X | 1]
        tc::fence_proxy_async();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            for (int a = 0; a < active; ++a)
                for (int s = 0; s < 8; ++s)
                    tc::mma_bf16(tmem + kColDw1, tc::desc_mnmajor(sDz1 + a * kBytesDz, kSboDz, s),
                                 tc::desc_mnmajor(sX + a * kBytesX, kSboX, s), kIdescDw1, !first || a > 0 || s > 0);
            tc::commit(bar);
        }
        if (!(ok = wait_mma(bar, phase, err))) break;
        first = false;
    }
    if (!ok) {
        // a wait gave up: give the tensor cores one more bounded wait before TMEM is released
        tc::mbar_wait(bar, phase, kWaitLimit);
    }

    // weight gradients: rows j = 0 .. 63 of the accumulators sit in TMEM lanes 0 .. 63
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (ok && !first && warp < 2) {
        const int j = tid;
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            float v[16];
            tc::tmem_ld16(tmem + lane_addr + kColDw2 + 16 * c, v);
            if (c < 4) {
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                    atomicAdd(reinterpret_cast<float4*>(grad + oW2 + j * kHid + 16 * c + i),
                              make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]));
            } else {
                atomicAdd(grad + oB2 + j, v[0]);
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            float v[16];
            tc::tmem_ld16(tmem + lane_addr + kColDw1 + 16 * c, v);
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
                const int col = 16 * c + i;
                if (col < kIn)
                    atomicAdd(reinterpret_cast<float4*>(grad + oW1 + j * kIn + col),
                              make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]));
                else if (col == kIn) atomicAdd(grad + oB1 + j, v[i]);
            }
        }
    }
    loss_acc = warp_sum(loss_acc);
    db3_acc = warp_sum(db3_acc);
    if (lane == 0) {
        atomicAdd(red, db3_acc);
        atomicAdd(red + 1, loss_acc);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (ok && tid < kHid) atomicAdd(grad + oW3 + tid, dw3);
    if (ok && tid == 0) {
        atomicAdd(grad + oB3, red[0]);
        atomicAdd(loss, red[1]);
    }
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, kTmemCols);
    }
}

// One Adam update from the gradients that the training kernel summed.  It moves them and the loss to the
// read-out arrays and leaves the sums cleared, so that every step, launched or replayed from a graph, finds
// them cleared and leaves them so, and no step clears them in a launch of its own.
__global__ void adam_kernel(float* __restrict__ w, float* __restrict__ g_sum, float* __restrict__ m,
                            float* __restrict__ v, int n, float lr, float c1, float c2, float* __restrict__ g,
                            float* __restrict__ loss_sum, float* __restrict__ loss) {
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        *loss = __ldcg(loss_sum);
        *loss_sum = 0.f;
    }
    if (i >= n) return;
    const float gi = __ldcg(g_sum + i);
    g_sum[i] = 0.f;
    g[i] = gi;
    const float mi = 0.9f * m[i] + 0.1f * gi;
    const float vi = 0.999f * v[i] + 0.001f * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
}

// ---------------------------------------------------------------- forward (inference)
// Shared memory of the inference kernels for N tiles per CTA (bytes); TMEM: 64 columns per tile, Z1 then Z2
template <int N> struct InferSmem {
    static constexpr uint32_t kA1 = 0, kW1 = kA1 + N * kBytesA1, kW2 = kW1 + kBytesW1, kF = kW2 + kBytesW2,
                              kBar = kF + 1024, kBytes = kBar + 64;
    static constexpr uint32_t kCols = kHid * N;
    static constexpr int kMaxCtaPerSm = 512 / (kHid * N);
};

// Set-up shared by the inference kernels: weights staged, TMEM allocated, barrier initialised.
template <int N>
__device__ __forceinline__ InferTile infer_setup(uint8_t* sm, const float* net, float*& mean, float*& istd) {
    using M = InferSmem<N>;
    const int warp = threadIdx.x >> 5;
    float* fs = reinterpret_cast<float*>(sm + M::kF);
    float *w3 = fs + 128, *b3 = fs + 192;
    mean = fs + 200;
    istd = fs + 224;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + M::kBar);
    uint32_t* tbase = reinterpret_cast<uint32_t*>(sm + M::kBar + 8);
    stage_weights(net, sm + M::kW1, sm + M::kW2, w3, b3, mean, istd, 0.5f);
    for (int t = threadIdx.x / kTile; t < N; t += blockDim.x / kTile) stage_ones(sm + M::kA1 + t * kBytesA1);
    if (warp == 0) tc::tmem_alloc(tbase, M::kCols);
    if (threadIdx.x == 0) tc::mbar_init(bar, 1);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    InferTile it;
    it.a1s = sm + M::kA1;
    it.sA1 = tc::smem_u32(sm + M::kA1);
    it.sW1 = tc::smem_u32(sm + M::kW1);
    it.sW2 = tc::smem_u32(sm + M::kW2);
    it.tmem = *tbase;
    it.lane_addr = (uint32_t)((warp & 3) * 32) << 16;  // warp w reaches TMEM lanes 32 (w mod 4) ..
    it.bar = bar;
    it.w3 = w3;
    it.b3 = *b3;
    return it;
}

template <int N> __device__ __forceinline__ void infer_teardown(const InferTile& it, bool ok, uint32_t phase) {
    if (!ok) tc::mbar_wait(it.bar, phase, kWaitLimit);  // give the tensor cores a last bounded wait
    tc::fence_before_sync();
    __syncthreads();
    if ((threadIdx.x >> 5) == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(it.tmem, InferSmem<N>::kCols);
    }
}

// Write this thread's normalised feature row [x_hat | 1 | 0] into a tile's X columns (in its A1 tile).
__device__ __forceinline__ void write_x_row(uint8_t* xs, const float* x, const float* mean, const float* istd,
                                            bool valid) {
    float v[32];
#pragma unroll
    for (int k = 0; k < kIn; ++k) v[k] = valid ? (x[k] - mean[k]) * istd[k] : 0.f;
    v[kIn] = 1.f;
#pragma unroll
    for (int k = kIn + 1; k < 32; ++k) v[k] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) st_row_chunk(xs, threadIdx.x, 8 * c, kSboA1, v + 8 * c);
}

__global__ void __launch_bounds__(128) mlp_forward_kernel(const float* __restrict__ net, const float* __restrict__ x,
                                                          long long n, float* __restrict__ out, int* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t sm[];
    float *mean, *istd;
    const InferTile it = infer_setup<1>(sm, net, mean, istd);
    uint32_t phase = 0;
    bool ok = true;
    const long long tiles = (n + kTile - 1) / kTile;
    for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const long long g = tile * kTile + threadIdx.x;
        const bool valid = g < n;
        float xv[kIn];
#pragma unroll
        for (int k = 0; k < kIn; ++k) xv[k] = valid ? x[g * kIn + k] : 0.f;
        write_x_row(it.a1s, xv, mean, istd, valid);
        float y;
        if (!(ok = infer_tiles<1>(it, phase, err, y))) break;
        if (valid) out[g] = y;
    }
    infer_teardown<1>(it, ok, phase);
}

// ---------------------------------------------------------------- full-box I/O, features, filter
// Node i of the box (x fastest; a box holds fewer than 2^31 cells): multiply-shift divisions by n0 and n1.
struct BoxDiv {
    FastDiv n0, n1;
};
__device__ __forceinline__ Coord box_coord(const LevelGeom& geo, const BoxDiv& dv, uint32_t i) {
    const uint32_t r = dv.n0.div(i), z = dv.n1.div(r);
    Coord c;
    c.x[0] = (int)(i - r * (uint32_t)geo.n[0]);
    c.x[1] = (int)(r - z * (uint32_t)geo.n[1]);
    c.x[2] = (int)z;
    return c;
}

using StreamSlots = NodeSlots<D3Q19>;

template <class S>
__global__ void set_equilibrium_kernel(S* __restrict__ f, LevelGeom geo, StepParams p, int even, BoxDiv dv,
                                       const float* __restrict__ rho, const float* __restrict__ u, long long nn) {
    using Tb = Tables<D3Q19>;
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= nn) return;
    const StreamSlots slot(geo, box_coord(geo, dv, (uint32_t)i), even);
    const float r = rho[i], ux = u[i * 3], uy = u[i * 3 + 1], uz = u[i * 3 + 2];
    const float usq15 = 1.5f * (ux * ux + uy * uy + uz * uz);
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const float cu = signed_dot<D3Q19>(q, ux, uy, uz);
        const float w = (float)Tb::w(q);
        // feq - w = w (rho - 1) + w rho (3 cu + 4.5 cu^2 - 1.5 u^2)
        const float d = w * fmaf(r, fmaf(cu, fmaf(4.5f, cu, 3.f), -usq15), r - 1.f);
        Storage<S>::store(f + slot.post_stream(q), d, p);
    }
}

template <class S>
__device__ __forceinline__ void load_node(const S* f, const StreamSlots& slot, float* d) {
#pragma unroll
    for (int q = 0; q < 19; ++q) d[q] = Storage<S>::load_raw(f + slot.post_stream(q));
}

constexpr int kMacroThreads = 256;

// A block's velocities through shared memory, so that the (x, y, z) records leave as whole lines.
__device__ __forceinline__ void store_velocities(float* __restrict__ u, long long base, long long nn, const float* v) {
    __shared__ float rec[3 * kMacroThreads];
    const int t = threadIdx.x;
    rec[3 * t] = v[0];
    rec[3 * t + 1] = v[1];
    rec[3 * t + 2] = v[2];
    __syncthreads();
    const long long first = 3 * base, last = 3 * (nn - base < kMacroThreads ? nn : base + kMacroThreads);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const long long j = first + t + k * kMacroThreads;
        if (j < last) u[j] = rec[t + k * kMacroThreads];
    }
}

// rho and u of every node (Q populations in, 16 bytes out).  256^3 with 64-bit divisions, slot arithmetic per
// population and velocities stored with stride three: FP32 520 us, FP16 947, FP64 599; now 312 (1.55 GB, 5.0
// TB/s), 329 and 402.
template <class S>
__global__ void __launch_bounds__(kMacroThreads) get_macros_kernel(const S* __restrict__ f, LevelGeom geo, StepParams p,
                                                                   int even, BoxDiv dv, float* __restrict__ rho,
                                                                   float* __restrict__ u, long long nn) {
    const long long base = blockIdx.x * (long long)kMacroThreads, i = base + threadIdx.x;
    float mac[4] = {0.f, 0.f, 0.f, 0.f};
    if (i < nn) {
        float d[19], neq[19];
        load_node(f, StreamSlots(geo, box_coord(geo, dv, (uint32_t)i), even), d);
        feq_neq_dev<D3Q19>(d, neq, p.scale, p.inv_scale, mac);
        rho[i] = mac[0];
    }
    store_velocities(u, base, nn, mac + 1);
}

// FP64 storage (absolute populations): feq in the reference's arithmetic order from the FP32
// fields, and rho / u by the reference's macro rule, rounded to FP32 on output.
__global__ void set_equilibrium_f64_kernel(double* __restrict__ f, LevelGeom geo, int even, BoxDiv dv,
                                           const float* __restrict__ rho, const float* __restrict__ u, long long nn) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= nn) return;
    const StreamSlots slot(geo, box_coord(geo, dv, (uint32_t)i), even);
    double feq[19];
    feq_exact<D3Q19>((double)rho[i], (double)u[i * 3], (double)u[i * 3 + 1], (double)u[i * 3 + 2], feq);
#pragma unroll
    for (int q = 0; q < 19; ++q) f[slot.post_stream(q)] = feq[q];
}

__global__ void __launch_bounds__(kMacroThreads) get_macros_f64_kernel(const double* __restrict__ f, LevelGeom geo,
                                                                       int even, BoxDiv dv, float* __restrict__ rho,
                                                                       float* __restrict__ u, long long nn) {
    const long long base = blockIdx.x * (long long)kMacroThreads, i = base + threadIdx.x;
    float w[3] = {0.f, 0.f, 0.f};
    if (i < nn) {
        const StreamSlots slot(geo, box_coord(geo, dv, (uint32_t)i), even);
        double v[19], r, ux, uy, uz;
#pragma unroll
        for (int q = 0; q < 19; ++q) v[q] = f[slot.post_stream(q)];
        macro_exact<D3Q19>(v, r, ux, uy, uz);
        rho[i] = (float)r;
        w[0] = (float)ux;
        w[1] = (float)uy;
        w[2] = (float)uz;
    }
    store_velocities(u, base, nn, w);
}

template <class S>
__global__ void features_kernel(const S* __restrict__ f, LevelGeom geo, StepParams p, int even, BoxDiv dv,
                                float* __restrict__ x, long long nn) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= nn) return;
    float d[19], neq[19], mac[4], v[kIn];
    load_node(f, StreamSlots(geo, box_coord(geo, dv, (uint32_t)i), even), d);
    feq_neq_dev<D3Q19>(d, neq, p.scale, p.inv_scale, mac);
    features(mac[0], neq, (float)p.tau, v, nullptr, p.inv_scale);
#pragma unroll
    for (int k = 0; k < kIn; ++k) x[i * kIn + k] = v[k];
}

// Adds one node's share of the filter: rho, u, u_a u_b and f - feq.
__device__ __forceinline__ void filter_add(const float* d, const StepParams& p, float* acc) {
    float neq[19], mac[4];
    feq_neq_dev<D3Q19>(d, neq, p.scale, p.inv_scale, mac);
    acc[0] += mac[0];
    acc[1] += mac[1];
    acc[2] += mac[2];
    acc[3] += mac[3];
    acc[4] += mac[1] * mac[1];
    acc[5] += mac[2] * mac[2];
    acc[6] += mac[3] * mac[3];
    acc[7] += mac[1] * mac[2];
    acc[8] += mac[1] * mac[3];
    acc[9] += mac[2] * mac[3];
#pragma unroll
    for (int q = 0; q < 19; ++q) acc[10 + q] += neq[q] * p.inv_scale;
}

// Block means over factor^3 nodes, any factor: one thread per block.
template <class S>
__global__ void filter_kernel(const S* __restrict__ f, LevelGeom geo, StepParams p, int even, int factor, int ncx,
                              int ncy, int ncz, float* __restrict__ out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long nc = (long long)ncx * ncy * ncz;
    if (i >= nc) return;
    const int X = (int)(i % ncx), Y = (int)((i / ncx) % ncy), Z = (int)(i / ((long long)ncx * ncy));
    float acc[29];
#pragma unroll
    for (int k = 0; k < 29; ++k) acc[k] = 0.f;
    for (int dz = 0; dz < factor; ++dz)
        for (int dy = 0; dy < factor; ++dy)
            for (int dx = 0; dx < factor; ++dx) {
                Coord c;
                c.x[0] = X * factor + dx;
                c.x[1] = Y * factor + dy;
                c.x[2] = Z * factor + dz;
                float d[19];
                load_node(f, StreamSlots(geo, c, even), d);
                filter_add(d, p, acc);
            }
    const float inv = 1.f / (float)(factor * factor * factor);
#pragma unroll
    for (int k = 0; k < 29; ++k) out[i * 29 + k] = acc[k] * inv;
}

// The same for factors that divide a warp: a warp takes 32 consecutive nodes of a row of the fine level
// (coalesced loads; one thread per block strode by the factor), a thread sums the factor^2 nodes of its
// column in the block, and a butterfly over the factor lanes of a block adds the columns.  The block's
// lanes share its 29 stores.  256^3 by 4, FP32 (1.4 GB): 585 us with one thread per block, 349 now.
constexpr int kFilterThreads = 128;
template <class S>
__global__ void __launch_bounds__(kFilterThreads) filter_warp_kernel(const S* __restrict__ f, LevelGeom geo, StepParams p,
                                                                     int even, int factor, int ncx, int ncy,
                                                                     unsigned segments, float* __restrict__ out) {
    const unsigned lane = threadIdx.x & 31u, seg = blockIdx.x * (kFilterThreads / 32) + (threadIdx.x >> 5);
    if (seg >= segments) return;  // whole warps
    const int x = (int)(seg * 32u + lane);
    const bool live = x < geo.n[0];  // the factor divides n0: a block's lanes are all live or all not
    float acc[29];
#pragma unroll
    for (int k = 0; k < 29; ++k) acc[k] = 0.f;
    if (live) {
        for (int dz = 0; dz < factor; ++dz)
            for (int dy = 0; dy < factor; ++dy) {
                Coord c;
                c.x[0] = x;
                c.x[1] = (int)blockIdx.y * factor + dy;
                c.x[2] = (int)blockIdx.z * factor + dz;
                float d[19];
                load_node(f, StreamSlots(geo, c, even), d);
                filter_add(d, p, acc);
            }
    }
    const float inv = 1.f / (float)(factor * factor * factor);
    for (int o = 1; o < factor; o <<= 1)
#pragma unroll
        for (int k = 0; k < 29; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    if (!live) return;
    const long long i = x / factor + (long long)ncx * (blockIdx.y + (long long)ncy * blockIdx.z);
    const int sub = (int)lane & (factor - 1);
#pragma unroll
    for (int k = 0; k < 29; ++k)
        if ((k & (factor - 1)) == sub) out[i * 29 + k] = acc[k] * inv;
}

// ---------------------------------------------------------------- training pairs
__device__ __forceinline__ long long wrap_index(int x, int y, int z, const int* n) {
    x = (x + n[0]) % n[0];
    y = (y + n[1]) % n[1];
    z = (z + n[2]) % n[2];
    return (long long)x + (long long)n[0] * (y + (long long)n[1] * z);
}

struct Grid3 {
    int n[3];
};

// Strain of the filtered field as the coarse lattice sees it, S = -3 factor Pi<f - feq> / (2 rho tau_f)
// (the fine non-equilibrium stress is -2/3 rho tau_f S_fine and S_coarse = factor S_fine), the exact
// subgrid stress, and the least-squares pieces of c over a node: num = tau^d : M, den = M : M,
// M = 2 |S| S.  Using the strain the collision itself estimates keeps the target consistent with
// the way the closure is applied.
__device__ __forceinline__ void filtered_strain(const float* cf, float tau_fine, int factor, float* s) {
    using Tb = Tables<D3Q19>;
    float p[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 1; q < 19; ++q) {
        const float n = cf[10 + q];
        const int cx = Tb::cx(q), cy = Tb::cy(q), cz = Tb::cz(q);
        if (cx) p[0] += n;
        if (cy) p[1] += n;
        if (cz) p[2] += n;
        if (cx * cy) p[3] += cx * cy > 0 ? n : -n;
        if (cx * cz) p[4] += cx * cz > 0 ? n : -n;
        if (cy * cz) p[5] += cy * cz > 0 ? n : -n;
    }
    const float k = -1.5f * (float)factor / (cf[0] * tau_fine);
#pragma unroll
    for (int i = 0; i < 6; ++i) s[i] = k * p[i];
}

__global__ void pairs_stage1_kernel(Grid3 g, const float* __restrict__ filt, float tau_fine, int factor,
                                    float* __restrict__ scratch) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long nn = (long long)g.n[0] * g.n[1] * g.n[2];
    if (i >= nn) return;
    const int pa[6] = {0, 1, 2, 0, 0, 1}, pb[6] = {0, 1, 2, 1, 2, 2};
    const float* c = filt + i * 29;
    float s[6], td[6];
    filtered_strain(c, tau_fine, factor, s);
    for (int k = 0; k < 6; ++k) td[k] = c[4 + k] - c[1 + pa[k]] * c[1 + pb[k]];
    const float tr = (td[0] + td[1] + td[2]) / 3.f;
    td[0] -= tr;
    td[1] -= tr;
    td[2] -= tr;
    const float ss = s[0] * s[0] + s[1] * s[1] + s[2] * s[2] + 2.f * (s[3] * s[3] + s[4] * s[4] + s[5] * s[5]);
    const float smag = sqrtf(2.f * ss);
    float num = 0.f, den = 0.f;
    for (int k = 0; k < 6; ++k) {
        const float m = 2.f * smag * s[k];
        const float w = k < 3 ? 1.f : 2.f;
        num += w * td[k] * m;
        den += w * m * m;
    }
    scratch[i * 3] = num;
    scratch[i * 3 + 1] = den;
    scratch[i * 3 + 2] = smag;
}

__global__ void pairs_stage2_kernel(Grid3 g, const float* __restrict__ filt, const float* __restrict__ scratch,
                                    float tau_fine, float tau_coarse, int factor, float* __restrict__ xo,
                                    float* __restrict__ yo) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long nn = (long long)g.n[0] * g.n[1] * g.n[2];
    if (i >= nn) return;
    const int x = (int)(i % g.n[0]), y = (int)((i / g.n[0]) % g.n[1]), z = (int)(i / ((long long)g.n[0] * g.n[1]));
    float num = 0.f, den = 0.f;
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx) {
                const long long j = wrap_index(x + dx, y + dy, z + dz, g.n);
                num += scratch[j * 3];
                den += scratch[j * 3 + 1];
            }
    num /= 27.f;
    den /= 27.f;
    const float c = den > 1e-30f ? -num / den : 0.f;  // no resolved strain: no constant to fit
    const float yv = fminf(fmaxf(c / kCUnit, 0.f), kYMax);
    const float tau_eff = tau_coarse + 3.f * kCUnit * yv * scratch[i * 3 + 2];
    const float r = (float)factor * tau_eff / tau_fine;
    const float* cf = filt + i * 29;
    float neq[19], v[kIn];
#pragma unroll
    for (int q = 0; q < 19; ++q) neq[q] = r * cf[10 + q];
    features(cf[0], neq, tau_coarse, v);
#pragma unroll
    for (int k = 0; k < kIn; ++k) xo[i * kIn + k] = v[k];
    yo[i] = yv;
}

// ---------------------------------------------------------------- fused collide-stream with the network
// The AA step of a full periodic box with the learned closure evaluated inside the collision: a
// persistent CTA of 256 threads takes 256 consecutive nodes at a time as two tiles of the two
// tensor-core layers, one node per thread; a node relaxes with tau = tau0 + 0.5 (sqrt(tau0^2 + 18 c
// sqrt(2 Pi:Pi)) - tau0), the Smagorinsky collision of fused_collide with C = 18 c, and streams; c is also
// stored per node (c_node) for the steps that reuse it.
//
// Bound by its instructions and the waits between its phases (issue slots 63 %, HBM at a fifth of its copy
// rate, tensor cores 7 %).  The features and the collision come from the pair sums of the populations in closed
// form, only the populations (SRT: and 1 / rho) are kept across the network (the collision forms everything else
// again, which is cheaper than registers), and the GELU leaves its factor 1/2 to the next layer's weights.  Two tiles per
// CTA share the weights and each barrier, so that three CTAs of 80 registers (24 warps) fit an SM.  Two
// nodes per thread as packed FP32 pairs execute a fifth fewer instructions and are slower (16 warps);
// four CTAs of 64 registers are slower too.
// us per step of one run, one tile and one node per thread with per-direction equilibria / now: SRT 33^3 69 / 12.9
// (the weights' staging), 64^3 89 / 31.8, 128^3 238 / 187, 256^3 1409 / 1400; MRT 128^3 256 / 191, 256^3
// 1544 / 1431.
// The grid is the number of CTAs that fit on the GPU (shared memory 55 KiB, TMEM 128 columns per CTA).
constexpr int kLsTiles = 2, kLsThreads = kLsTiles * kTile;

template <class S, int Coll, bool Odd>
__global__ void __launch_bounds__(kLsThreads, 3) learned_step_kernel(S* __restrict__ f, LevelGeom geo, StepParams p,
                                                                    const float* __restrict__ net, float fallback_c,
                                                                    float* __restrict__ c_node, int* __restrict__ err,
                                                                    BoxDiv dv) {
    using Tb = Tables<D3Q19>;
    using St = Storage<S>;
    extern __shared__ __align__(1024) uint8_t sm[];
    float *mean, *istd;
    const InferTile it = infer_setup<kLsTiles>(sm, net, mean, istd);
    const uint32_t tid = threadIdx.x;
    const uint32_t nn = (uint32_t)geo.n[0] * (uint32_t)geo.n[1] * (uint32_t)geo.n[2];  // fewer than 2^31
    const long long st = geo.stride;
    uint32_t phase = 0;
    bool ok = true;

    for (uint32_t base = blockIdx.x * kLsThreads; base < nn; base += gridDim.x * kLsThreads) {
        const uint32_t i = base + tid;
        const bool valid = i < nn;
        F1 pre[19], inv_rho;
        {
            const NodeCells<D3Q19> cell(geo, box_coord(geo, dv, valid ? i : 0u));
#pragma unroll
            for (int q = 0; q < 19; ++q) {
                const int k = Odd && q != 0 ? 1 : 0, plane = k ? Tb::opp(q) : q;
                pre[q] = {valid ? St::load_raw(f + plane * st + cell(-k * Tb::cx(q), -k * Tb::cy(q), -k * Tb::cz(q))) : 0.f};
            }
        }
        {
            F1 x[kIn];
            fused_features(pre, p, (float)p.tau, x, inv_rho);
            float v[32];
#pragma unroll
            for (int j = 0; j < kIn; j += 4) {
                const float4 m = *reinterpret_cast<const float4*>(mean + j), s = *reinterpret_cast<const float4*>(istd + j);
                v[j] = (x[j].v - m.x) * s.x;
                v[j + 1] = (x[j + 1].v - m.y) * s.y;
                v[j + 2] = (x[j + 2].v - m.z) * s.z;
                v[j + 3] = (x[j + 3].v - m.w) * s.w;
            }
            v[kIn] = 1.f;
#pragma unroll
            for (int j = kIn + 1; j < 32; ++j) v[j] = 0.f;
            uint8_t* tile = it.a1s + (tid / kTile) * kBytesA1;
#pragma unroll
            for (int c = 0; c < 4; ++c) st_row_chunk(tile, tid & (kTile - 1), 8 * c, kSboA1, v + 8 * c);
        }
        float y;
        if (!(ok = infer_tiles<kLsTiles>(it, phase, err, y))) break;
        if (!valid) continue;
        const float cn = isfinite(y) ? kCUnit * fminf(fmaxf(y, 0.f), kYMax) : fallback_c;
        F1 post[19];
        // (MRT forms 1 / rho again: held across the network it costs 10 steps and the read-out at 160^3, runs in
        // turn, 3383 us against 3297; SRT the other way round, 3.17 ms against 3.21)
        fused_collide<Coll == kMrt, true, false>(pre, post, p, F1{18.f * cn}, (const F1*)nullptr, (F1*)nullptr,
                                                 Coll == kMrt ? (const F1*)nullptr : &inv_rho);
        const NodeCells<D3Q19> cell(geo, box_coord(geo, dv, i));
        if (c_node) c_node[cell(0, 0, 0)] = cn;
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            const int k = Odd && q != 0 ? 1 : 0, plane = k ? q : Tb::opp(q);
            St::store_raw(f + plane * st + cell(k * Tb::cx(q), k * Tb::cy(q), k * Tb::cz(q)), post[q].v);
        }
    }
    infer_teardown<kLsTiles>(it, ok, phase);
}

template <class S>
static cudaError_t learned_step_s(int coll, bool odd, void* f, const LevelGeom& geo, const StepParams& p,
                                  const float* net, float fallback_c, float* c_node, int* err, cudaStream_t s) {
    static PersistentGrid grids[4];
    auto launch = [&](auto kernel, int slot) -> cudaError_t {
        using M = InferSmem<kLsTiles>;
        int grid = 0;
        // (TMEM: 512 columns per SM, so that no CTA waits for some)
        const cudaError_t e = grids[slot].get((const void*)kernel, kLsThreads, (int)M::kBytes, M::kMaxCtaPerSm, &grid);
        if (e != cudaSuccess) return e;
        kernel<<<grid, kLsThreads, M::kBytes, s>>>(
            static_cast<S*>(f), geo, p, net, fallback_c, c_node, err,
            BoxDiv{FastDiv::make((uint32_t)geo.n[0]), FastDiv::make((uint32_t)geo.n[1])});
        return cudaGetLastError();
    };
    if (coll == kMrt)
        return odd ? launch(learned_step_kernel<S, kMrt, true>, 0) : launch(learned_step_kernel<S, kMrt, false>, 1);
    return odd ? launch(learned_step_kernel<S, kSrt, true>, 2) : launch(learned_step_kernel<S, kSrt, false>, 3);
}

// ---------------------------------------------------------------- launchers used by the API
template <class S>
static cudaError_t dispatch_box(int op, void* f, const LevelGeom& geo, const StepParams& p, int even, const float* a,
                                float* b, float* c, int factor, const int* nc, cudaStream_t s) {
    const long long nn = (long long)geo.n[0] * geo.n[1] * geo.n[2];
    const unsigned blocks = (unsigned)((nn + 255) / 256);
    const BoxDiv dv{FastDiv::make((uint32_t)geo.n[0]), FastDiv::make((uint32_t)geo.n[1])};
    switch (op) {
        case kBoxSetEq:
            set_equilibrium_kernel<S><<<blocks, 256, 0, s>>>((S*)f, geo, p, even, dv, a, b, nn);
            break;
        case kBoxGetMacros:
            get_macros_kernel<S><<<blocks, kMacroThreads, 0, s>>>((const S*)f, geo, p, even, dv, b, c, nn);
            break;
        case kBoxFeatures:
            features_kernel<S><<<blocks, 256, 0, s>>>((const S*)f, geo, p, even, dv, b, nn);
            break;
        case kBoxFilter: {
            const long long ncn = (long long)nc[0] * nc[1] * nc[2];
            if (factor <= 32 && !(factor & (factor - 1)) && nc[1] <= 65535 && nc[2] <= 65535) {
                const unsigned segments = (unsigned)((geo.n[0] + 31) / 32), per = kFilterThreads / 32;
                filter_warp_kernel<S><<<dim3((segments + per - 1) / per, nc[1], nc[2]), kFilterThreads, 0, s>>>(
                    (const S*)f, geo, p, even, factor, nc[0], nc[1], segments, b);
            } else {
                filter_kernel<S><<<(unsigned)((ncn + 127) / 128), 128, 0, s>>>((const S*)f, geo, p, even, factor, nc[0],
                                                                                nc[1], nc[2], b);
            }
            break;
        }
        default:
            return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace closure

cudaError_t closure_learned_step(int storage, int coll, bool odd, void* f, const LevelGeom& geo, const StepParams& p,
                                 const float* net, float fallback_c, float* c_node, int* err, cudaStream_t s) {
    using namespace closure;
    switch (storage) {
        case ZL_STORAGE_F32: return learned_step_s<float>(coll, odd, f, geo, p, net, fallback_c, c_node, err, s);
        case ZL_STORAGE_F16: return learned_step_s<__half>(coll, odd, f, geo, p, net, fallback_c, c_node, err, s);
        case ZL_STORAGE_BF16:
            return learned_step_s<__nv_bfloat16>(coll, odd, f, geo, p, net, fallback_c, c_node, err, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t closure_box_op(int op, int storage, void* f, const LevelGeom& geo, const StepParams& p, int even,
                           const float* a, float* b, float* c, int factor, const int* nc, cudaStream_t s) {
    using namespace closure;
    switch (storage) {
        case ZL_STORAGE_F32: return dispatch_box<float>(op, f, geo, p, even, a, b, c, factor, nc, s);
        case ZL_STORAGE_F16: return dispatch_box<__half>(op, f, geo, p, even, a, b, c, factor, nc, s);
        case ZL_STORAGE_BF16: return dispatch_box<__nv_bfloat16>(op, f, geo, p, even, a, b, c, factor, nc, s);
        case ZL_STORAGE_F64: {
            const long long nn = (long long)geo.n[0] * geo.n[1] * geo.n[2];
            const unsigned blocks = (unsigned)((nn + 255) / 256);
            const BoxDiv dv{FastDiv::make((uint32_t)geo.n[0]), FastDiv::make((uint32_t)geo.n[1])};
            if (op == kBoxSetEq)
                set_equilibrium_f64_kernel<<<blocks, 256, 0, s>>>((double*)f, geo, even, dv, a, b, nn);
            else if (op == kBoxGetMacros)
                get_macros_f64_kernel<<<blocks, kMacroThreads, 0, s>>>((const double*)f, geo, even, dv, b, c, nn);
            else
                return cudaErrorInvalidValue;
            return cudaGetLastError();
        }
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace zl

// ---------------------------------------------------------------- C ABI (context-free part)
using namespace zl;
using namespace zl::closure;

struct zl_trainer {
    int device = 0;
    cudaStream_t stream = nullptr;      // stream the trainer issues on
    cudaStream_t own_stream = nullptr;  // the trainer's own stream
    float* w = nullptr;     // kFlat: weights (trainable part first) + normalisation
    float* g_sum = nullptr;     // a running step's gradients and squared errors, cleared between steps
    float* loss_sum = nullptr;
    bool sums_dirty = false;    // a step was not launched whole: the next one clears the sums first
    float* g = nullptr;     // kTrainable gradients of the last step
    float* m = nullptr;     // Adam moments
    float* v = nullptr;
    float* loss = nullptr;  // sum of squared errors of the last step
    int* err = nullptr;
    long long t = 0;        // Adam step count
    long long last_n = 0;
};

static_assert(sizeof(zl_mlp) == sizeof(float) * kFlat, "zl_mlp layout");

static int train_attr_once(int device) {
    static std::mutex mu;
    static bool done[64] = {false};
    std::lock_guard<std::mutex> lock(mu);
    if (device < 0 || device >= 64) return ZL_EINVAL;
    if (!done[device]) {
        if (cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrSmem) !=
                cudaSuccess ||
            cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)InferSmem<1>::kBytes) != cudaSuccess)
            return ZL_EDEVICE;
        done[device] = true;
    }
    return ZL_OK;
}

extern "C" {

int zl_trainer_create(const zl_mlp* init, int device, zl_trainer** out) {
    if (!init || !out) return ZL_EINVAL;
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return ZL_EDEVICE;
    int rc = train_attr_once(device);
    if (rc) return rc;
    zl_trainer* tr = new zl_trainer();
    tr->device = device;
    bool ok = cudaStreamCreateWithFlags(&tr->own_stream, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMalloc(&tr->w, sizeof(float) * kFlat) == cudaSuccess &&
              cudaMalloc(&tr->g, sizeof(float) * kTrainable) == cudaSuccess &&
              cudaMalloc(&tr->g_sum, sizeof(float) * kTrainable) == cudaSuccess &&
              cudaMalloc(&tr->loss_sum, sizeof(float)) == cudaSuccess &&
              cudaMalloc(&tr->m, sizeof(float) * kTrainable) == cudaSuccess &&
              cudaMalloc(&tr->v, sizeof(float) * kTrainable) == cudaSuccess &&
              cudaMalloc(&tr->loss, sizeof(float)) == cudaSuccess && cudaMalloc(&tr->err, sizeof(int)) == cudaSuccess;
    ok = ok && cudaMemcpy(tr->w, init, sizeof(float) * kFlat, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemset(tr->g, 0, sizeof(float) * kTrainable) == cudaSuccess &&
         cudaMemset(tr->g_sum, 0, sizeof(float) * kTrainable) == cudaSuccess &&
         cudaMemset(tr->loss_sum, 0, sizeof(float)) == cudaSuccess &&
         cudaMemset(tr->m, 0, sizeof(float) * kTrainable) == cudaSuccess &&
         cudaMemset(tr->v, 0, sizeof(float) * kTrainable) == cudaSuccess &&
         cudaMemset(tr->loss, 0, sizeof(float)) == cudaSuccess && cudaMemset(tr->err, 0, sizeof(int)) == cudaSuccess;
    tr->stream = tr->own_stream;
    if (!ok) {
        zl_trainer_destroy(tr);
        return ZL_EDEVICE;
    }
    *out = tr;
    return ZL_OK;
}

int zl_trainer_set_stream(zl_trainer* tr, void* stream) {
    if (!tr) return ZL_EINVAL;
    if (cudaSetDevice(tr->device) != cudaSuccess || cudaStreamSynchronize(tr->stream) != cudaSuccess)
        return ZL_EDEVICE;
    tr->stream = stream ? static_cast<cudaStream_t>(stream) : tr->own_stream;
    return ZL_OK;
}

int zl_trainer_step(zl_trainer* tr, const float* x_device, const float* y_device, int64_t n, float lr) {
    if (!tr || !x_device || !y_device || n <= 0) return ZL_EINVAL;
    if (cudaSetDevice(tr->device) != cudaSuccess) return ZL_EDEVICE;
    cudaStream_t s = tr->stream;
    if (tr->sums_dirty) {
        if (cudaMemsetAsync(tr->g_sum, 0, sizeof(float) * kTrainable, s) != cudaSuccess ||
            cudaMemsetAsync(tr->loss_sum, 0, sizeof(float), s) != cudaSuccess)
            return ZL_EDEVICE;
        // a captured clear runs only if its graph does
        cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &capturing) != cudaSuccess) return ZL_EDEVICE;
        tr->sums_dirty = capturing != cudaStreamCaptureStatusNone;
    }
    const long long tiles = (n + kTile - 1) / kTile;
    const unsigned grid = (unsigned)(tiles < 148 ? tiles : 148);
    if (launch_dependent(mlp_train_kernel, dim3(grid), dim3(kTrThreads), kTrSmem, s, (const float*)tr->w, x_device, y_device,
                         (long long)n, 1.f / (float)n, tr->g_sum, tr->loss_sum, tr->err) != cudaSuccess)
        return ZL_EDEVICE;
    ++tr->t;
    const float c1 = 1.f - powf(0.9f, (float)tr->t), c2 = 1.f - powf(0.999f, (float)tr->t);
    if (launch_dependent(adam_kernel, dim3((kTrainable + 127) / 128), dim3(128), 0, s, tr->w, tr->g_sum, tr->m, tr->v,
                         kTrainable, lr, c1, c2, tr->g, tr->loss_sum, tr->loss) != cudaSuccess) {
        tr->sums_dirty = true;
        return ZL_EDEVICE;
    }
    tr->last_n = n;
    return cudaGetLastError() == cudaSuccess ? ZL_OK : ZL_EDEVICE;
}

static int trainer_check(zl_trainer* tr) {
    if (cudaSetDevice(tr->device) != cudaSuccess || cudaStreamSynchronize(tr->stream) != cudaSuccess)
        return ZL_EDEVICE;
    int e = 0;
    if (cudaMemcpy(&e, tr->err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return ZL_EDEVICE;
    return e ? ZL_ETIMEOUT : ZL_OK;
}

int zl_trainer_loss(zl_trainer* tr, double* loss) {
    if (!tr || !loss) return ZL_EINVAL;
    int rc = trainer_check(tr);
    if (rc) return rc;
    float v = 0.f;
    if (cudaMemcpy(&v, tr->loss, sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess) return ZL_EDEVICE;
    *loss = tr->last_n > 0 ? (double)v / (double)tr->last_n : 0.;
    return ZL_OK;
}

int zl_trainer_gradients(zl_trainer* tr, zl_mlp* grad) {
    if (!tr || !grad) return ZL_EINVAL;
    int rc = trainer_check(tr);
    if (rc) return rc;
    std::memset(grad, 0, sizeof(zl_mlp));
    return cudaMemcpy(grad, tr->g, sizeof(float) * kTrainable, cudaMemcpyDeviceToHost) == cudaSuccess ? ZL_OK
                                                                                                      : ZL_EDEVICE;
}

int zl_trainer_weights(zl_trainer* tr, zl_mlp* out) {
    if (!tr || !out) return ZL_EINVAL;
    int rc = trainer_check(tr);
    if (rc) return rc;
    return cudaMemcpy(out, tr->w, sizeof(zl_mlp), cudaMemcpyDeviceToHost) == cudaSuccess ? ZL_OK : ZL_EDEVICE;
}

void zl_trainer_destroy(zl_trainer* tr) {
    if (!tr) return;
    cudaSetDevice(tr->device);
    if (tr->stream) cudaStreamSynchronize(tr->stream);
    if (tr->own_stream && tr->own_stream != tr->stream) cudaStreamSynchronize(tr->own_stream);
    cudaFree(tr->w);
    cudaFree(tr->g);
    cudaFree(tr->g_sum);
    cudaFree(tr->loss_sum);
    cudaFree(tr->m);
    cudaFree(tr->v);
    cudaFree(tr->loss);
    cudaFree(tr->err);
    if (tr->own_stream) cudaStreamDestroy(tr->own_stream);
    delete tr;
}

int zl_mlp_forward(const zl_mlp* net, const float* x_device, int64_t n, float* y_device, void* stream) {
    if (!net || !x_device || !y_device || n < 0) return ZL_EINVAL;
    if (n == 0) return ZL_OK;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return ZL_EDEVICE;
    int rc = train_attr_once(device);
    if (rc) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float* w = nullptr;
    int* err = nullptr;
    if (cudaMalloc(&w, sizeof(zl_mlp)) != cudaSuccess || cudaMalloc(&err, sizeof(int)) != cudaSuccess) {
        cudaFree(w);
        return ZL_EDEVICE;
    }
    int e = 0;
    bool ok = cudaMemcpyAsync(w, net, sizeof(zl_mlp), cudaMemcpyHostToDevice, s) == cudaSuccess &&
              cudaMemsetAsync(err, 0, sizeof(int), s) == cudaSuccess;
    if (ok) {
        const long long tiles = (n + kTile - 1) / kTile;
        const long long cap = 148 * 4;  // four CTAs per SM: 4 x 64 TMEM columns and 4 x 37 KiB
        const unsigned grid = (unsigned)(tiles < cap ? tiles : cap);
        mlp_forward_kernel<<<grid, 128, InferSmem<1>::kBytes, s>>>(w, x_device, n, y_device, err);
        ok = cudaGetLastError() == cudaSuccess &&
             cudaMemcpyAsync(&e, err, sizeof(int), cudaMemcpyDeviceToHost, s) == cudaSuccess &&
             cudaStreamSynchronize(s) == cudaSuccess;
    }
    cudaFree(w);
    cudaFree(err);
    if (!ok) return ZL_EDEVICE;
    return e ? ZL_ETIMEOUT : ZL_OK;
}

int zl_closure_pairs(const int32_t nc[3], const float* filtered_device, double tau_fine, double tau_coarse,
                     int factor, float* x_device, float* y_device, float* scratch_device, void* stream) {
    if (!nc || !filtered_device || !x_device || !y_device || !scratch_device || factor < 1 || !(tau_fine > 0.5) ||
        !(tau_coarse > 0.5))
        return ZL_EINVAL;
    Grid3 g;
    for (int a = 0; a < 3; ++a) {
        if (nc[a] < 3) return ZL_EINVAL;
        g.n[a] = nc[a];
    }
    const long long nn = (long long)nc[0] * nc[1] * nc[2];
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const unsigned blocks = (unsigned)((nn + 255) / 256);
    pairs_stage1_kernel<<<blocks, 256, 0, s>>>(g, filtered_device, (float)tau_fine, factor, scratch_device);
    pairs_stage2_kernel<<<blocks, 256, 0, s>>>(g, filtered_device, scratch_device, (float)tau_fine, (float)tau_coarse,
                                               factor, x_device, y_device);
    return cudaGetLastError() == cudaSuccess ? ZL_OK : ZL_EDEVICE;
}

}  // extern "C"
