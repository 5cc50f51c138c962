"""Rounding errors of the line FFTs, on the CPU: the roots that the composite
radices hold as constants and the table's twiddles are correctly rounded, and the
lines of every length that the any-length plane passes take (their radices, twiddle
table and roots, compiled for the host) are as close to extended precision as the
run-time plans that these lengths ran on before, with tables of unreduced angles: at
most 0.97 times their error (FP32 1.05: other roots are rounded to 24 bits in 9 = 3 x
3 than in 3, 3) over 400 lines of normal values; the seed moves the ratio by less
than 0.01.  Powers formed in registers give up to 1.24."""
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


LINES = r'''
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "pw_fft_any.cuh"
#include "pw_fft_tmpl.cuh"
#include "pw_twiddle.h"
template <typename T> using V = std::vector<Cx<T>>;
// the run-time plan's stages (radices 8, 4, 2, 3, 5 in this order, natural table)
template <typename T, int N, int S> void run_time(V<T> &x, const V<T> &tw, int sign) {
    if constexpr (S < pwt::plan_len(N)) {
        constexpr int R = pwt::plan_radix(N, S), NS = pwt::plan_ns(N, S), NBF = N / R, TWS = N / (NS * R);
        V<T> y(N);
        for (int j = 0; j < NBF; ++j) {
            Cx<T> v[R];
            for (int r = 0; r < R; ++r) {
                v[r] = x[j + r * NBF];
                Cx<T> w = tw[r * (j % NS) * TWS];
                if (sign > 0) w.y = -w.y;
                if (r && NS > 1) v[r] = cmul(v[r], w);
            }
            SmallDft<T, R>::run(v, (T)sign);
            for (int r = 0; r < R; ++r) y[(j / NS) * NS * R + j % NS + r * NS] = v[r];
        }
        x = y;
        run_time<T, N, S + 1>(x, tw, sign);
    }
}
template <typename T, int N> void fused(V<T> &x, const V<T> &tw, int sign) {
    constexpr int NST = pwf::FPlan<N>::nst, R0 = pwf::FPlan<N>::r(0), R1 = NST == 2 ? pwf::FPlan<N>::r(1) : 1;
    V<T> y(N), table(pwk::any::TWN);
    for (int i = R0; NST == 2 && i < N; ++i) table[i] = tw[pwk::any::tw_entry(i, R0)];
    for (int j = 0; j < R1; ++j) {
        Cx<T> v[R0];
        for (int r = 0; r < R0; ++r) v[r] = x[j + r * R1];
        pwf::Dft<T, R0>::run(v, (T)sign, nullptr, 0);
        for (int r = 0; r < R0; ++r) y[j * R0 + r] = v[r];
    }
    x = y;
    if constexpr (NST == 2) {
        for (int j = 0; j < R0; ++j) {
            Cx<T> v[R1];
            for (int r = 0; r < R1; ++r) v[r] = x[j + r * R0];
            pwf::apply_tw<T, N, 1, R1>(v, pwk::any::Tw<T>{table.data()}, j, sign);
            pwf::Dft<T, R1>::run(v, (T)sign, nullptr, 0);
            for (int r = 0; r < R1; ++r) y[j + r * R0] = v[r];
        }
        x = y;
    }
}
template <typename T, int N> bool line() {
    V<T> tw(N), tw0(N);
    std::vector<long double> c(N), s(N);
    for (int m = 0; m < N; ++m) {
        double re, im;
        pwk::twiddle(m, N, re, im);
        tw[m] = cmake((T)re, (T)im);
        const double a = -2.0 * M_PI * (double)m / (double)N;     // angle not reduced
        tw0[m] = cmake((T)std::cos(a), (T)std::sin(a));
        const long double b = 2.0L * 3.14159265358979323846264338327950288L * m / N;
        c[m] = std::cos(b);
        s[m] = std::sin(b);
        // half an ulp of 1 at most, and what the long double functions leave
        if (std::fabs(re - c[m]) > 5.6e-17L || std::fabs(im + s[m]) > 5.6e-17L) {
            std::printf("twiddle %d / %d\n", m, N);
            return false;
        }
    }
    std::mt19937_64 g(N);
    std::normal_distribution<double> U;
    double e[2] = {0.0, 0.0};
    for (int t = 0; t < 400; ++t) {
        const int sign = t & 1 ? 1 : -1;
        V<T> x(N);
        for (auto &q : x) q = cmake((T)U(g), (T)U(g));
        V<T> y[2] = {x, x};
        run_time<T, N, 0>(y[0], tw0, sign);
        fused<T, N>(y[1], tw, sign);
        for (int k = 0; k < N; ++k) {
            long double a = 0.0L, b = 0.0L;
            for (int m = 0; m < N; ++m) {
                const int q = m * k % N;
                a += x[m].x * c[q] - sign * x[m].y * s[q];
                b += sign * x[m].x * s[q] + x[m].y * c[q];
            }
            for (int u = 0; u < 2; ++u) {
                const long double p = y[u][k].x - a, r = y[u][k].y - b;
                e[u] += (double)(p * p + r * r);
            }
        }
    }
    const bool ok = std::sqrt(e[1]) <= (sizeof(T) == 4 ? 1.05 : 0.97) * std::sqrt(e[0]);
    if (!ok) std::printf("%s, %d points: %.3f times the run-time plan's error\n", sizeof(T) == 4 ? "FP32" : "FP64", N, std::sqrt(e[1] / e[0]));
    return ok;
}
int main() {
    bool ok = true;
#define LINE(N) ok &= line<double, N>(), ok &= line<float, N>();
    PW_ANY_SIZES(LINE)
    std::printf(ok ? "ok\n" : "bad\n");
    return ok ? 0 : 1;
}
'''


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_roots_are_rounded_once(tmp_path):
    build_and_run(tmp_path, "roots", ROOTS)


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_lines_are_as_exact_as_the_run_time_plans(tmp_path):
    build_and_run(tmp_path, "lines", LINES)
