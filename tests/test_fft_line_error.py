"""Rounding errors of the FP64 line FFTs, on the CPU: the roots that the composite
radices hold as constants are correctly rounded."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pwdft.jl_b200", "csrc")
INC = os.path.join(ROOT, "include")

ROOTS = r'''
#include <cmath>
#include <cstdio>
#include "pw_fft_fused.cuh"
static bool ok = true;
static void check(int m, int R, double got, long double want) {
    // half an ulp, and the rounding of the long double angle and function
    const long double ulp = std::ldexp(1.0L, std::ilogb(got == 0.0 ? 1e-300 : got) - 52);
    if (std::fabs((long double)got - want) > 0.5L * ulp + 4e-19L) {
        std::printf("%d / %d: off by %.2Lf ulp\n", m, R, std::fabs(got - want) / ulp);
        ok = false;
    }
}
template <int R> void all() {
    pwf::sfor<0, 2 * R>([](auto mc) {
        constexpr int m = decltype(mc)::value;
        const long double a = 2.0L * 3.14159265358979323846264338327950288L * (m % R) / R;
        check(m, R, pwf::Root<m, R>::c, std::cos(a));
        check(m, R, pwf::Root<m, R>::s, -std::sin(a));
    });
}
int main() {
    all<9>(), all<16>(), all<24>(), all<25>(), all<27>();
    std::printf(ok ? "ok\n" : "bad\n");
    return ok ? 0 : 1;
}
'''


def build_and_run(tmp_path, name, prog):
    src = tmp_path / (name + ".cu")
    src.write_text(prog)
    exe = tmp_path / name
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-I", CSRC, "-I", INC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_roots_are_rounded_once(tmp_path):
    build_and_run(tmp_path, "roots", ROOTS)
