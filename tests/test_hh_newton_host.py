"""CPU test of the Hodgkin-Huxley BDF step's linear solve (eb_device.cuh, compiled for
the host): the elimination that leaves out an arrow matrix's structural zeros gives
the general Gauss-Jordan inverse's result bit for bit, or hands the matrix to it --
on ordinary matrices and on ones with zero, tiny, huge, infinite and NaN entries."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
struct float4 { float x, y, z, w; };
struct float2 { float x, y; };
template <class T> static inline T __ldg(const T *p) { return *p; }
static inline float __int_as_float(int i) { float f; memcpy(&f, &i, 4); return f; }
#include "eb_device.cuh"
int main() {
    std::mt19937 g(5);
    std::uniform_real_distribution<float> U(-1, 1);
    const float odd[] = {0.0f, -0.0f, 1e-45f, 1e-38f, 1e38f, -3e38f, INFINITY, -INFINITY, NAN, 1.0f};
    long handed = 0, differ = 0;
    for (int n = 0; n < 300000; ++n) {
        eb::Arrow4 A;
        float r[4], a[4], b[4];
        auto draw = [&](float scale) { return n % 3 && g() % 40 == 0 ? odd[g() % 10] : scale * U(g); };
        for (int j = 0; j < 4; ++j) {
            A.d[j] = draw(0.5f) - 1;
            A.row[j] = draw(300.0f);
            A.col[j] = draw(0.1f);
            r[j] = draw(1.0f);
        }
        const bool ok = eb::arrow_solve(A, r, a);
        if (!ok) { ++handed; continue; }
        if (!eb::arrow_solve_general(A, r, b)) { ++differ; continue; }
        for (int j = 0; j < 4; ++j) differ += a[j] != b[j];
    }
    printf("%ld %ld\n", handed, differ);
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="needs g++")
def test_arrow_elimination_equals_general_inverse(tmp_path):
    src = tmp_path / "arrow.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "arrow")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-w", "-I" + os.path.join(ROOT, "edlut_b200", "csrc"),
                    str(src), "-o", exe], check=True)
    handed, differ = map(int, subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split())
    assert differ == 0
    assert 0 < handed < 150000  # the odd matrices, not the ordinary ones
