"""Register DFTs of the fused plans added for further line lengths (10 = 2 x 5,
12 = 3 x 4 and 18 = 2 x 9 by the prime-factor split, 16 = 4 x 4), compiled by
nvcc into a host program and compared with a direct DFT, both signs, FP32 and
FP64; and the padded line layout: positions distinct and inside the stride."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pwdft.jl_b200", "csrc")

PROG = r'''
#include <cmath>
#include <cstdio>
#include <random>
#include <set>
#include "pw_fft_fused.cuh"
template <typename T, int R> double worst(T s) {
    std::mt19937 g(97 * R + (s > 0));
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    double w = 0.0;
    for (int trial = 0; trial < 300; ++trial) {
        Cx<T> v[R];
        double xr[R], xi[R];
        for (int n = 0; n < R; ++n) {
            v[n] = cmake((T)U(g), (T)U(g));
            xr[n] = v[n].x;
            xi[n] = v[n].y;
        }
        pwf::Dft<T, R>::run(v, s, nullptr, 0);
        for (int k = 0; k < R; ++k) {
            double ar = 0.0, ai = 0.0;
            for (int n = 0; n < R; ++n) {
                const double a = (double)s * 2.0 * M_PI * (double)((n * k) % R) / R;
                ar += xr[n] * std::cos(a) - xi[n] * std::sin(a);
                ai += xr[n] * std::sin(a) + xi[n] * std::cos(a);
            }
            w = std::fmax(w, std::fmax(std::fabs(ar - v[k].x), std::fabs(ai - v[k].y)));
        }
    }
    return w;
}
template <int N> bool layout() {
    std::set<int> p;
    for (int x = 0; x < N; ++x) p.insert(pwf::fp_pos<N>(x));
    const int r0 = pwf::FPlan<N>::r(0), r1 = pwf::FPlan<N>::nst == 2 ? pwf::FPlan<N>::r(1) : 1;
    return (int)p.size() == N && *p.rbegin() < pwf::fp_xs<N>() && r0 * r1 == N;
}
int main() {
    bool ok = true;
#define CHK(R)                                                                                  \
    for (int s = -1; s <= 1; s += 2)                                                             \
        if (!(worst<float, R>((float)s) < 4e-7 * R) || !(worst<double, R>((double)s) < 1e-14 * R)) { \
            std::printf("radix %d sign %d\n", R, s);                                             \
            ok = false;                                                                          \
        }
    CHK(10) CHK(12) CHK(16) CHK(18)
#define LAY(N)                          \
    if (!layout<N>()) {                 \
        std::printf("layout %d\n", N); \
        ok = false;                     \
    }
    LAY(20) LAY(24) LAY(25) LAY(27) LAY(30) LAY(32) LAY(36) LAY(40) LAY(45) LAY(48) LAY(50) LAY(54) LAY(60) LAY(64)
    LAY(72) LAY(75) LAY(80) LAY(81) LAY(90) LAY(96) LAY(100) LAY(108) LAY(120) LAY(125) LAY(128)
    std::printf(ok ? "ok\n" : "bad\n");
    return ok ? 0 : 1;
}
'''


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_new_radices_and_layouts(tmp_path):
    src = tmp_path / "radices.cu"
    src.write_text(PROG)
    exe = tmp_path / "radices"
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
