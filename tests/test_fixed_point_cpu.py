"""CPU test of the FP64 transforms' fixed-point arithmetic (csrc/s2d_fixed.cuh,
which also compiles as C++): products, conversions and shift counts against
128-bit integers and long double, over random values and the edges of the
limbs (low words of 0, 2^31 - 1, 2^31, 2^32 - 1)."""

import os
import subprocess

SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include "s2d_fixed.cuh"
using namespace s2d;
typedef __int128 i128;
static unsigned long long seed = 1;
static unsigned long long rnd() {
    seed += 0x9E3779B97F4A7C15ULL;
    unsigned long long x = seed;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
    return x ^ (x >> 31);
}
static long long value(int bits) {   // |x| < 2^bits, every second low word at an edge
    long long x = (long long)(rnd() >> (64 - bits));
    const unsigned edge[4] = {0u, 0x7FFFFFFFu, 0x80000000u, 0xFFFFFFFFu};
    if (rnd() & 1) x = (x & ~0xFFFFFFFFLL) | edge[rnd() & 3];
    return rnd() & 1 ? -x : x;
}
static int bad = 0;
static void check(bool ok, const char* what) {
    if (!ok && bad++ < 10) printf("%s\n", what);
}
template <bool INV>
static void products() {
    for (int i = 0; i < 400000; ++i) {
        const double a = (rnd() >> 11) * 6.283185307179586 / 9007199254740992.0;
        long long c = llrintl(ldexpl(cosl(a), 62)), d = llrintl(ldexpl(sinl(a), 62));
        if (i % 3 == 0) d = (d & ~0xFFFFFFFFLL) | 0x80000000LL;
        if (i % 3 == 1) c = (c & ~0xFFFFFFFFLL) | 0x80000000LL;
        const fx2 z{value(61), value(61)};
        for (int r = 0; r <= 2; ++r) {
            const fx2 o = fx_cmul<INV>(z, fx_limbs(c, d), r);
            const i128 s = INV ? -1 : 1;
            const i128 re = (i128)z.x * c - s * ((i128)z.y * d), im = (i128)z.y * c + s * ((i128)z.x * d);
            const i128 one = (i128)1 << (62 + r);
            // low x low of two products (2), the moved unit of d (1), rounding (1/2)
            const i128 ex = (i128)o.x * one - re, ey = (i128)o.y * one - im;
            check(ex < 4 * one && -ex < 4 * one && ey < 4 * one && -ey < 4 * one, "fx_cmul");
        }
        const long long p = value(61), q = value(61);
        const i128 e = ((i128)fx_mul64(p, q) << 64) - (i128)p * q;
        check(e < ((i128)1 << 64) && -e < ((i128)1 << 64), "fx_mul64");
        const i128 h = ((i128)fx_mulc(z.x, kFxSin3H, kFxSin3L) << 62) - (i128)z.x * kFxSin3;
        check(h < ((i128)2 << 62) && -h < ((i128)2 << 62), "fx_mulc");
    }
}
int main() {
    products<false>();
    products<true>();
    for (int i = 0; i < 400000; ++i) {
        // FP64 -> fixed -> FP64: exact to the grid, then to FP64's rounding
        double v = ldexp((double)((rnd() >> 11) | (1ULL << 52)), -52 - (int)(rnd() % 60));
        if (rnd() & 1) v = -v;
        long long b;
        memcpy(&b, &v, 8);
        for (int n0 = 3; n0 <= 4; ++n0) {
            const long long x = fx_from((int)(b >> 32), (unsigned)b, 1023, n0);
            check(fabsl((long double)x - ldexpl(v, 62 - n0)) <= 0.5L, "fx_from");
            const long long y = value(1 + (int)(rnd() % 62));
            const long long t = fx_to(y, 1023 + 63);   // value = y
            double w;
            memcpy(&w, &t, 8);
            check(fabsl((long double)w - (long double)y) <= fabsl((long double)y) * 0x1p-53L, "fx_to");
        }
    }
    double z;
    long long t = fx_to(1, 40);
    memcpy(&z, &t, 8);
    check(z == 0.0, "below the normal range");
    t = fx_to(1LL << 60, 2050);
    memcpy(&z, &t, 8);
    check(std::isinf(z), "above the range");
    t = fx_to(5, fx_exponent_base(0x7FF, 3, 0));
    memcpy(&z, &t, 8);
    check(std::isnan(z), "an infinity or NaN in the input");
    // at most two bits more per radix-4 or radix-3 pass, for every sum
    for (float per : {fx_per(3), fx_per(4), 0.2357f})
        for (unsigned sum = 1; sum < 1u << 30; sum += sum / 4 + 1)
            for (int ns = per < 0.3f ? 4 : 3; ns <= 6144; ns *= 2)
                for (int R = 2; R <= 4; ++R) {
                    const int d = fx_shift_total(ns * R, per, sum, kFxByLimit) - fx_shift_total(ns, per, sum, kFxByLimit);
                    check(d >= 0 && d <= 2, "fx_shift_total");
                }
    printf("%d bad\n", bad);
    return bad != 0;
}
"""


def test_fixed_point_arithmetic(tmp_path):
    from spectral2d_gb300.build import CSRC
    src, exe = tmp_path / "fixed.cpp", tmp_path / "fixed"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    p = subprocess.run([os.fspath(exe)], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout
