"""Which FP32 D3Q19 levels take the kernel with two nodes per thread (launch.cuh), on the host: by default from
a size, never against an explicit one-node shape, with Smagorinsky as without; by a pair shape wherever the
kernel applies."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "launch.cuh"
int main() {
    int bad = 0;
    auto level = [](int n0, int n1, int n2, int block) {
        zl::LevelGeom g = {};
        const int n[3] = {n0, n1, n2};
        for (int a = 0; a < 3; ++a) g.n[a] = g.a[a] = n[a], g.periodic[a] = 1;
        g.stride = ((long long)n0 * n1 * n2 + 63) / 64 * 64;
        g.full = 1;
        g.block[0] = block;
        g.block[1] = 1;
        return g;
    };
    zl::StepParams les = {}, plain = {};
    les.les = 1;
    auto expect = [&](bool a, bool b) { bad += a != b; };
    for (int n : {128, 256}) {
        for (const auto* p : {&les, &plain}) {
            expect(zl::pair_default(3, false, *p, 4, level(n, n, n, 0)), true);
            for (int block : {32, 64, 128, 256}) expect(zl::pair_default(3, false, *p, 4, level(n, n, n, block)), false);
            expect(zl::pair_default(3, false, *p, 4, level(n - 1, n, n, 0)), false);
            expect(zl::pair_default(3, false, *p, 4, level(32, 32, 32, 0)), false);
            expect(zl::pair_default(3, false, *p, 2, level(n, n, n, 0)), false);
            expect(zl::pair_default(3, false, *p, 8, level(n, n, n, 0)), false);
        }
        for (int block : {-64, 0, 64}) expect(zl::pair_les_eligible(3, les, 4, level(n, n, n, block)), true);
    }
    // rows that leave lanes idle: 33 of 64 and 45 of 64 never, 23 of 32 and 75 of 96 with Smagorinsky only, and 23
    // of 32 on smaller levels with MRT only
    for (bool mrt : {false, true}) {
        expect(zl::pair_default(3, mrt, les, 4, level(46, 150, 150, 0)), mrt);
        expect(zl::pair_default(3, mrt, les, 4, level(46, 200, 200, 0)), true);
        expect(zl::pair_default(3, mrt, les, 4, level(96, 96, 96, 0)), true);
        expect(zl::pair_default(3, mrt, les, 4, level(66, 200, 200, 0)), false);
    }
    for (int n : {66, 90}) expect(zl::pair_default(3, false, les, 4, level(n, 200, 200, 0)), false);
    for (int n : {46, 150}) expect(zl::pair_default(3, false, les, 4, level(n, 200, 200, 0)), true);
    for (int n : {46, 66, 90, 150}) expect(zl::pair_default(3, false, plain, 4, level(n, 200, 200, 0)), false);
    expect(zl::pair_les_eligible(3, plain, 4, level(128, 128, 128, -64)), false);
    expect(zl::pair_les_eligible(3, les, 4, level(129, 128, 128, -64)), false);
    expect(zl::pair_les_eligible(3, les, 2, level(128, 128, 128, -64)), false);
    zl::LevelGeom g = level(128, 128, 128, -64);
    g.periodic[1] = 0;
    expect(zl::pair_les_eligible(3, les, 4, g), false);
    g = level(128, 128, 128, -64);
    g.full = 0;
    expect(zl::pair_les_eligible(3, les, 4, g), false);
    les.forced = 1;
    expect(zl::pair_les_eligible(3, les, 4, level(128, 128, 128, -64)), false);
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


def test_pair_rule(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "rule.cu", tmp_path / "rule"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(ROOT, "zllbm_b200", "csrc"), "-I", os.path.join(ROOT, "include"), str(src), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.split() == ["0"]
