"""The error norm of the wide solver reads the tolerances four species at a time, so the last step
reads one past the 59 species: the parameter arrays hold 60, the last species' again."""
import os
import subprocess

from conftest import PKG

SOURCE = r'''
#include <cmath>
#include "radm2_device.cuh"
#include "radm2_internal.h"
using namespace radm2;
int main()
{
    constexpr int n = sizeof(SolveParams::AbsTol) / sizeof(double), want = (NVAR + 3) / 4 * 4;
    static_assert(sizeof(SolveParams::RelTol) == sizeof(SolveParams::AbsTol), "");
    if (n < want) return 1;
    double at[NVAR], rt[NVAR], rpar[20] = {0};
    for (int i = 0; i < NVAR; i++) at[i] = 1.0 + i, rt[i] = 1e-3 / (1 + i);
    for (int scalar = 0; scalar < 2; scalar++) {
        int ipar[20] = {1, scalar, 0, 2}, autonomous;
        SolveParams p;
        if (parse_params(0.0, 600.0, at, rt, rpar, ipar, 1, &p, &autonomous) != 1) return 2;
        for (int i = 0; i < n; i++) {
            const int k = scalar ? 0 : i < NVAR ? i : NVAR - 1;
            if (p.AbsTol[i] != at[k] || p.RelTol[i] != rt[k]) return 3;
        }
    }
    return 0;
}
'''


def test_tolerances_cover_the_norm_s_last_step(tmp_path):
    src, exe = tmp_path / "pad.cpp", tmp_path / "pad"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(PKG, "csrc"), "-I", "/usr/local/cuda/include", str(src), "-o", str(exe), "-L", PKG,
                    "-lradm2_b200", "-Wl,-rpath," + PKG], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
