"""The column exchange of the cluster tridiagonalisation (pw_tri.h), on the CPU:
the ranks' step counts compiled into a host program that runs the protocol
(arm, publish, wait, read; two buffers) with every rank in turn held back as long as
the others can go on without it, and in random order.  A store into a buffer
whose earlier step has not been read yet, a step that never completes, or a
writer that has already left fails.  The same program with every rank receiving
to the end (the form that needs luck in timing) has to be caught.  And the choice
of the kernel for the columns before the cluster's, on devices with few SMs."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pwdft.jl_b200", "csrc")

PROG = r'''
#include <cstdio>
#include <random>
#include <vector>
#include "pw_tri.h"
using namespace pwk::eig;
static bool to_end = false;   // plant: every rank receives in every step
static int recv_steps(int n, int r) { return to_end ? n - 1 : tri_steps(n, r); }
struct Rank {
    int j = 0, at = 0;              // step, and what comes next in it: publish, wait, read
    std::vector<unsigned> got;      // bytes of each step
};
struct Run {
    int n;
    bool bad = false;
    std::vector<Rank> r;
    explicit Run(int n_) : n(n_), r(TRC) {
        for (auto &q : r) q.got.assign(n + 1, 0u);
    }
    bool done(int a) const { return r[a].j >= recv_steps(n, a); }
    // one move of rank a; false if it cannot go on
    bool move(int a) {
        Rank &q = r[a];
        if (done(a)) return false;
        if (q.at == 0) {
            unsigned cols = 0;
            for (int i = 1 + a; i < n; i += TRC) cols += i > q.j;
            if (cols)
                for (int d = 0; d < TRC; ++d)
                    if (q.j < recv_steps(n, d)) {
                        // the buffer's last use, step j - 2, must have been read
                        if (r[d].j < q.j - 1) bad = true;
                        r[d].got[q.j] += 32u * cols;
                    }
            q.at = 1;
        } else if (q.at == 1) {
            if (q.got[q.j] > tri_bytes(n, q.j)) bad = true;
            if (q.got[q.j] < tri_bytes(n, q.j)) return false;
            q.at = 2;
        } else {
            q.at = 0;
            ++q.j;
        }
        return true;
    }
    bool finish(int held, std::mt19937 *g) {
        for (;;) {
            bool any = false;
            if (g) {
                for (int t = 0; t < 200; ++t) any |= move((int)((*g)() % TRC));
                if (!any)
                    for (int a = 0; a < TRC; ++a) any |= move(a);
            } else {
                for (int a = 0; a < TRC; ++a)
                    while (a != held && move(a)) any = true;
                if (!any) any = move(held);
            }
            if (!any) break;
        }
        for (int a = 0; a < TRC; ++a) bad |= !done(a);
        return !bad;
    }
};
int main() {
    bool ok = true;
    for (int n = 1; n <= 256; ++n) {
        for (int held = 0; held < TRC; ++held) ok &= Run(n).finish(held, nullptr);
        for (int s = 0; s < 3; ++s) {
            std::mt19937 g(1000 * n + s);
            ok &= Run(n).finish(0, &g);
        }
        for (int j = 0; j < n - 1; ++j)
            ok &= j < tri_steps(n, tri_last_rank(n)) && j < tri_steps(n, tri_writer(j));
        if (!ok) {
            std::printf("n = %d\n", n);
            return 1;
        }
    }
    // the register kernel of the grid is taken only where all its CTAs are resident:
    // a whole B200 (148 SMs; 4 and 1 CTAs an SM up to and past n = 512, at the
    // least), an eighth of one, and no device at all
    for (int n = 1; n <= 2000; ++n)
        for (int sms : {148, 18, 0})
            for (int per : {4, 1})
                for (int clusters : {9, 0}) {
                    const TriRoute t = tri_route(n, sms * per, clusters);
                    ok &= t.cluster == (clusters > 0) && t.jend == (clusters ? n > 256 ? n - 256 : 0 : n - 1);
                    ok &= !t.registers || (n <= 1024 && tri_r_ctas(n) <= sms * per);
                    ok &= tri_r_ctas(n) * tri_r_warps(n) >= n - 1;
                    if (sms == 148) ok &= t.registers == (n <= 1024);
                }
    if (!ok) {
        std::printf("route\n");
        return 1;
    }
    to_end = true;
    for (int n : {12, 17, 160, 256}) {
        bool caught = false;
        for (int held = 0; held < TRC; ++held) caught |= !Run(n).finish(held, nullptr);
        if (!caught) {
            std::printf("not caught at n = %d\n", n);
            return 1;
        }
    }
    std::printf("ok\n");
    return 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_late_ranks_and_the_route(tmp_path):
    src = tmp_path / "tri.cpp"
    src.write_text(PROG)
    exe = tmp_path / "tri"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
