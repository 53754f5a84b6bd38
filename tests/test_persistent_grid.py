"""The launch shape of the persistent learned step is settled per device: a process with contexts on two
devices opts in to the kernel's shared memory on each of them, once, from any number of threads, and an
attempt that failed is made again.  Built against a CUDA runtime that this program plays."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "persistent_grid.cuh"

static thread_local int device = 0;
static std::atomic<int> opt_ins[3];
static std::atomic<int> bytes_asked{0};
static bool refuse = false;

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int v) {
    if (refuse) return cudaErrorInvalidValue;
    bytes_asked = v;
    ++opt_ins[device];
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int d) {
    switch (a) {
        case cudaDevAttrMultiProcessorCount: *v = 100 + d; break;
        case cudaDevAttrMaxRegistersPerMultiprocessor: *v = 65536; break;
        case cudaDevAttrMaxSharedMemoryPerMultiprocessor: *v = 233472; break;
        case cudaDevAttrReservedSharedMemoryPerBlock: *v = 1024; break;
        default: return cudaErrorInvalidValue;
    }
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* fa, const void*) {
    fa->numRegs = 80;
    fa->sharedSizeBytes = 0;
    return cudaSuccess;
}
}

static int kernel;

int main() {
    zl::PersistentGrid g;
    int grid = 0, bad = 0;
    auto ask = [&](int d) { device = d; return g.get(&kernel, 256, 56384, 4, &grid); };
    refuse = true;
    bad += ask(0) == cudaSuccess;
    refuse = false;
    for (int round = 0; round < 3; ++round)
        for (int d = 0; d < 2; ++d)
            bad += ask(d) != cudaSuccess || grid != 3 * (100 + d);  // 80 registers x 256 threads: 3 CTAs per SM
    std::vector<std::thread> pool;
    std::atomic<int> wrong{0};
    for (int t = 0; t < 8; ++t)
        pool.emplace_back([&] {
            device = 2;
            int mine = 0;
            if (g.get(&kernel, 256, 56384, 4, &mine) != cudaSuccess || mine != 306) ++wrong;
        });
    for (auto& t : pool) t.join();
    std::printf("%d %d %d %d %d %d\n", bad, wrong.load(), opt_ins[0].load(), opt_ins[1].load(), opt_ins[2].load(),
                bytes_asked.load());
}
"""


def test_opt_in_per_device(tmp_path):
    cuda = os.path.join(os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")), "include")
    if not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "grid.cpp", tmp_path / "grid"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-x", "c++", "-I", os.path.join(ROOT, "zllbm_b200", "csrc"),
                    "-I", cuda, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True)
    assert out.stdout.split() == ["0", "0", "1", "1", "1", "56384"]


def test_the_learned_step_asks_it():
    """Every launch of the learned step takes its shape there: the source holds no launch shape of its own."""
    src = open(os.path.join(ROOT, "zllbm_b200", "csrc", "closure.cu")).read()
    body = src[src.index("static cudaError_t learned_step_s"):src.index("static cudaError_t dispatch_box")]
    assert "static PersistentGrid" in body and "static int" not in body and "cudaFuncSetAttribute" not in body
