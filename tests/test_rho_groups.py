"""Band groups of the density pass (pw_rho.h), on the CPU: as many as there are bands
where those fit on the GPU at once, whatever the number of CTAs an SM holds; never
an empty group, and no more than 16."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pwdft.jl_b200", "csrc")

PROG = r'''
#include <cstdio>
#include "pw_rho.h"
int main() {
    for (int N3 = 12; N3 <= 250; ++N3)
        for (int cnt = 1; cnt <= 70; ++cnt)
            for (int per = 0; per <= 8; ++per) {
                const int G = pwk::rho_groups(N3, cnt, per);
                bool ok = G >= 1 && G <= cnt && G <= 16;
                if (cnt <= 8 && N3 * cnt <= 148 * per) ok &= G == cnt;
                // 9 to 16 bands: a CTA's second band costs more than 0.1 a group saves
                if (cnt <= 16 && N3 * cnt <= 148 * per) ok &= (cnt + G - 1) / G == 1;
                if (!ok) {
                    std::printf("N3 %d, %d bands, %d a SM: %d groups\n", N3, cnt, per, G);
                    return 1;
                }
            }
    return 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_groups(tmp_path):
    src = tmp_path / "rho.cpp"
    src.write_text(PROG)
    exe = tmp_path / "rho"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
