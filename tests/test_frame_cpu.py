"""CPU test of the framed images' index arithmetic (csrc/s2d_frame.cuh, which
also compiles as C++)."""

import os
import subprocess

SRC = r"""
#include <cstdio>
#include "s2d_frame.cuh"
using namespace s2d;
int main() {
    int bad = 0;
    for (int n = 8; n <= 4096; ++n) {
        const int pitch = net_pitch(n);
        if (pitch % 2 || pitch < n + 2 || pitch > n + 3) ++bad;
        for (int f = 0; f < pitch; ++f) {
            const int s = net_frame_source(f, n);
            if (s < 0 || s >= n) ++bad;                      // inside the image, the padding too
            if (f < n + 2 && s != (f - 1 + n) % n) ++bad;    // circular
        }
    }
    printf("%d bad\n", bad);
    return bad != 0;
}
"""


def test_every_framed_position_has_its_source_inside_the_image(tmp_path):
    from spectral2d_gb300.build import CSRC
    src, exe = tmp_path / "frame.cpp", tmp_path / "frame"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    p = subprocess.run([os.fspath(exe)], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout
