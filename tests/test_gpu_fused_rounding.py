"""The velocity inside the fused D3Q19 collisions: 1 / rho correctly rounded where a collision has always divided
so (MRT with Smagorinsky, with a force, and the learned step's), for one node and for pairs."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "closure.cuh"
#include "pair_value.cuh"
using namespace zl;

// thread t: populations of a node with rho in about [0.8, 1.2]; counts the nodes whose ux is not the rounded
// jx / rho; Learned: with the reciprocal that the learned step's features leave
template <bool Mrt, bool Les, bool Forced, bool Learned>
__global__ void check(StepParams p, int n, unsigned* off) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    uint32_t s = 2654435761u * (uint32_t)(t + 1);
    F1 d[19], out[19], mac[4], F[3] = {{0.f}, {0.f}, {0.f}};
    F2 d2[19], out2[19], mac2[4], Fp[3] = {splat(0.f), splat(0.f), splat(0.f)};
    for (int q = 0; q < 19; ++q) {
        s = s * 1664525u + 1013904223u;
        d[q].v = ((s >> 8) * (1.f / 16777216.f) - 0.5f) * 0.08f;
        d2[q] = splat(d[q].v);
    }
    if constexpr (Learned) {
        F1 x[closure::kIn], r;
        closure::fused_features(d, p, (float)p.tau, x, r);
        const F2 r2 = splat(r.v);
        fused_collide<Mrt, Les, Forced>(d, out, p, F1{0.18f}, F, mac, &r);
        fused_collide<Mrt, Les, Forced>(d2, out2, p, splat(0.18f), Fp, mac2, &r2);
    } else {
        fused_collide<Mrt, Les, Forced>(d, out, p, F1{0.18f}, F, mac);
        fused_collide<Mrt, Les, Forced>(d2, out2, p, splat(0.18f), Fp, mac2);
    }
    const F1 X1 = (d[7] - d[10]) - (d[8] - d[9]), X2 = (d[11] - d[14]) - (d[12] - d[13]);
    const F1 jx = (d[1] - d[2]) + (X1 + X2);
    const float want = __fmul_rn(jx.v, __frcp_rn(mac[0].v));
    if (mac[1].v != want) atomicAdd(off, 1u);
    if (mac2[1].v.x != mac[1].v || mac2[1].v.y != mac[1].v) atomicAdd(off + 1, 1u);
    for (int q = 0; q < 19; ++q)
        if (out2[q].v.x != out[q].v || out2[q].v.y != out[q].v) atomicAdd(off + 1, 1u);
}

int main() {
    const int n = 1 << 16;
    StepParams p = {};
    p.tau = 0.506;
    p.omega32 = 1.f / 0.506f;
    p.scale = p.inv_scale = 1.f;
    p.dt = 1.;
    unsigned *off, h[8];
    if (cudaMalloc(&off, sizeof(h)) != cudaSuccess || cudaMemset(off, 0, sizeof(h)) != cudaSuccess) return 1;
    check<true, true, false, false><<<n / 256, 256>>>(p, n, off);
    check<false, true, false, true><<<n / 256, 256>>>(p, n, off + 2);
    check<false, true, true, false><<<n / 256, 256>>>(p, n, off + 4);
    check<false, false, false, false><<<n / 256, 256>>>(p, n, off + 6);
    if (cudaMemcpy(h, off, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    for (unsigned v : h) std::printf("%u ", v);
}
"""


def test_rounded_reciprocal(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, exe = tmp_path / "rounding.cu", tmp_path / "rounding"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(ROOT, "zllbm_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    off = [int(v) for v in out.split()]
    assert off[:6] == [0] * 6 and off[7] == 0
    assert off[6] > 0  # the fast reciprocal, which the others must not be, shows in the same count


def test_the_learned_step_hands_its_reciprocal_on():
    src = open(os.path.join(ROOT, "zllbm_b200", "csrc", "closure.cu")).read()
    body = src[src.index("learned_step_kernel(S*"):src.index("static cudaError_t learned_step_s")]
    assert "fused_features(pre, p, (float)p.tau, x, inv_rho)" in body and "Coll == kMrt ? (const F1*)nullptr : &inv_rho)" in body
