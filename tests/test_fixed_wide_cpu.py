"""CPU test of the fixed-point results' conversion at both ends of FP64's range
(fx_to_normal and fx_rest of csrc/s2d_fixed.cuh, which also compiles as C++): the same as
ldexp of the rounded integer, gradual underflow included."""

import os
import subprocess

SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include "s2d_fixed.cuh"
using namespace s2d;
int main() {
    int bad = 0, low = 0;
    unsigned long long seed = 1;
    auto wide = [](long long x, int eb) {
        const long long b = fx_to_normal(x, fx_normal_base(eb));
        double v;
        memcpy(&v, &b, 8);
        return fx_normal_base(eb) == eb ? v : v * fx_rest(eb);
    };
    for (int i = 0; i < 400000; ++i) {
        seed = seed * 6364136223846793005ULL + 1442695040888963407ULL;
        long long x = (long long)(seed >> (1 + (seed >> 20) % 62));
        if (seed & 1) x = -x;
        for (int eb : {(int)(seed >> 33) % 4000 - 1500, (int)(seed >> 33) % 64, 2047 + (int)(seed >> 33) % 64}) {
            const double want = ldexp((double)x, eb - 1086);
            low += want != 0.0 && fabs(want) < 0x1p-1022;
            if (wide(x, eb) != want) ++bad;
        }
    }
    bad += wide(0, 40) != 0.0 || !std::isnan(wide(5, fx_exponent_base(0x7FF, 4, 3)));
    printf("%d bad, %d subnormal\n", bad, low);
    return bad != 0 || low < 1000;
}
"""


def test_conversion_at_both_ends_of_the_range(tmp_path):
    from spectral2d_gb300.build import CSRC
    src, exe = tmp_path / "wide.cpp", tmp_path / "wide"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    p = subprocess.run([os.fspath(exe)], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout
