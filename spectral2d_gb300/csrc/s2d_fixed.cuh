// s2d_fixed.cuh -- FP64 transforms in 64-bit block fixed point on the integer
// pipes.
//
// GB300 issues 2 FP64 operations per cycle and SM, but 60 to 90 32-bit
// integer operations and 23 32 x 32 -> 64 multiply-adds.  A transform of FP64
// values is therefore done on 64-bit integers that share one exponent: a
// twiddled radix-4 butterfly (3 complex products, 16 additions) takes 2.0
// cycles of an SM that way against 11.2 as 22 FP64 instructions (measured in
// registers, 32 warps per SM).
//
// A transform's elements become x = value * 2^s0 with the largest component
// in [2^59, 2^60), so the grid of values is finer than FP64's at the largest
// component by 2^7; every pass works on x and the last pass rounds to FP64.
// Values grow by at most the radix R per pass, and never beyond the sum of
// all input magnitudes; x is shifted right by just the bits that the smaller
// of these two bounds asks for (fx_shift_total), so a spectrum of a few large modes
// is not shifted at all and a white one by log2 M bits in all, against
// sqrt(M) growth of the rounding noise.  With S = sum |x| / max |x| the error
// relative to the 2-norm of the output is at most about
// 0.6 sqrt(M S) / sqrt(1 + S^2 / M) 2^-60, 1.5e-16 at worst (S = sqrt(M),
// M = 3072); with the final rounding to FP64, 4e-17 to 8e-17 were measured for
// white, steep and single-mode spectra: an FP64 transform of that length has
// 1e-16 to 2.5e-16.
//
// The bounds come from integer reductions (a maximum, a sum), whose result
// does not depend on the order, and all else is integer arithmetic: the same
// input gives the same bits in every kernel and launch shape.
#pragma once

#include <stdint.h>

#ifndef __CUDACC__
#define S2D_HD inline
#else
#define S2D_HD __device__ __forceinline__
#endif

namespace s2d {

// c + i d in units of 2^-62 as signed 32-bit limbs: c = ch 2^32 + cl.
struct __attribute__((aligned(16))) FxTw {
    int ch, cl, dh, dl;
};
struct __attribute__((aligned(16))) fx2 {
    long long x, y;
};

// A twiddle from its parts in units of 2^-62.  A low limb of -2^31 is moved by
// one unit (2^-62), so that -d has limbs too.
inline FxTw fx_limbs(long long c, long long d) {
    if ((d & 0xFFFFFFFFLL) == 0x80000000LL) ++d;
    FxTw w;
    w.cl = (int)(unsigned)(c & 0xFFFFFFFFLL);
    w.ch = (int)((c - w.cl) / 4294967296LL);
    w.dl = (int)(unsigned)(d & 0xFFFFFFFFLL);
    w.dh = (int)((d - w.dl) / 4294967296LL);
    return w;
}

// |z| <= 2^62.085 = 3 sqrt(2) 2^60 before and after every pass.
constexpr int kFxOne = 62;              // twiddle fraction bits
// sin(2 pi / 3) = sqrt(3) / 2 in units of 2^-62, as limbs
constexpr long long kFxSin3 = 3993837246235628775LL;
constexpr int kFxSin3L = (int)(unsigned)(kFxSin3 & 0xFFFFFFFFLL);
constexpr int kFxSin3H = (int)((kFxSin3 + 0x80000000LL) >> 32);

S2D_HD long long fx_madw(int a, int b, long long c) {
#ifdef __CUDA_ARCH__
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
#else
    return (long long)((unsigned long long)((long long)a * b) + (unsigned long long)c);
#endif
}

// x >> n, n >= 0 (0 for n > 63)
S2D_HD unsigned long long fx_shr(unsigned long long x, int n) {
#ifdef __CUDA_ARCH__
    unsigned long long r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(n));
    return r;
#else
    return n > 63 ? 0ULL : x >> n;
#endif
}

S2D_HD int fx_lo(long long x) { return (int)(unsigned)x; }
// the high limb once the low one is taken as signed: (x + 2^31) >> 32
S2D_HD int fx_hi(long long x) { return (int)(x >> 32) + (int)((unsigned)x >> 31); }

// Rounded x >> r, 0 <= r < 31.
S2D_HD long long fx_round(long long x, int r) {
    const long long y = x + (int)((1u << r) >> 1);
#ifdef __CUDA_ARCH__
    const unsigned lo = __funnelshift_r((unsigned)y, (unsigned)(y >> 32), r);
    return (long long)(((unsigned long long)(unsigned)((int)(y >> 32) >> r) << 32) | lo);
#else
    return y >> r;
#endif
}

// (H 2^32 + M) >> (32 - s) for 0 <= s < 32, where H was started from M's high
// word (fx_sext): two funnel shifts.
S2D_HD long long fx_join(long long H, long long M, int s) {
#ifdef __CUDA_ARCH__
    const int hl = (int)H, hh = (int)(H >> 32);
    const unsigned lo = __funnelshift_l((unsigned)M, (unsigned)hl, s);
    const unsigned hi = __funnelshift_l((unsigned)hl, (unsigned)hh, s);
    return (long long)(((unsigned long long)hi << 32) | lo);
#else
    return (long long)(((unsigned long long)H << s) | (s ? (unsigned)M >> (32 - s) : 0u));
#endif
}
// The high word of the mixed terms, the start of the high x high sum.
S2D_HD long long fx_sext(long long M) { return (long long)(int)(M >> 32); }

// z w (INV: z conj(w)) >> r, rounded, 0 <= r <= 2; |z| <= 2^62.085.  The two
// limbs of each factor give four partial products of which low x low is
// dropped (at most 2, 0.5 rms, of the last place, with no bias since the limbs
// are signed): 12 multiply-adds.  M, the mixed terms, fits 2^62.6; its high
// word starts the high x high sum.
// The one negated factor is d: its low limb is never -2^31 (fx_limbs), which
// has no negative, while the data's may be.
template <bool INV>
S2D_HD fx2 fx_cmul(fx2 z, FxTw w, int r) {
    const int ah = fx_hi(z.x), al = fx_lo(z.x), bh = fx_hi(z.y), bl = fx_lo(z.y);
    const long long half = 1LL << (29 + r);
    // re = a c + b d1, im = b c + a d2; d1 = -d (forward) or d (INV), d2 = -d1
    const int nh = -w.dh, nl = -w.dl;
    const int d1h = INV ? w.dh : nh, d1l = INV ? w.dl : nl, d2h = INV ? nh : w.dh, d2l = INV ? nl : w.dl;
    fx2 o;
    long long M = fx_madw(bl, d1h, fx_madw(bh, d1l, fx_madw(al, w.ch, fx_madw(ah, w.cl, half))));
    o.x = fx_join(fx_madw(bh, d1h, fx_madw(ah, w.ch, fx_sext(M))), M, 2 - r);
    M = fx_madw(bl, w.ch, fx_madw(bh, w.cl, fx_madw(al, d2h, fx_madw(ah, d2l, half))));
    o.y = fx_join(fx_madw(bh, w.ch, fx_madw(ah, d2h, fx_sext(M))), M, 2 - r);
    return o;
}

// x (h 2^32 + l) >> 62, rounded.
S2D_HD long long fx_mulc(long long x, int h, int l) {
    const int xh = fx_hi(x), xl = fx_lo(x);
    const long long M = fx_madw(xl, h, fx_madw(xh, l, 1LL << 29));
    return fx_join(fx_madw(xh, h, fx_sext(M)), M, 2);
}

// a b >> 64, rounded; |a|, |b| <= 2^62.
S2D_HD long long fx_mul64(long long a, long long b) {
    const int ah = fx_hi(a), al = fx_lo(a), bh = fx_hi(b), bl = fx_lo(b);
    const long long M = fx_madw(al, bh, fx_madw(ah, bl, 1LL << 31));
    return fx_madw(ah, bh, fx_sext(M));
}

S2D_HD fx2 fx_add(fx2 a, fx2 b) { return fx2{a.x + b.x, a.y + b.y}; }
S2D_HD fx2 fx_sub(fx2 a, fx2 b) { return fx2{a.x - b.x, a.y - b.y}; }
// a + S i b with S = -1 (forward) or +1 (INV)
template <bool INV>
S2D_HD fx2 fx_addi(fx2 a, fx2 b) { return INV ? fx2{a.x - b.y, a.y + b.x} : fx2{a.x + b.y, a.y - b.x}; }
template <bool INV>
S2D_HD fx2 fx_subi(fx2 a, fx2 b) { return fx_addi<!INV>(a, b); }

template <bool INV>
S2D_HD void fx_bf2(fx2* v) {
    const fx2 a = v[0], b = v[1];
    v[0] = fx_add(a, b);
    v[1] = fx_sub(a, b);
}
template <bool INV>
S2D_HD void fx_bf4(fx2* v) {
    const fx2 t0 = fx_add(v[0], v[2]), t1 = fx_sub(v[0], v[2]), t2 = fx_add(v[1], v[3]), t3 = fx_sub(v[1], v[3]);
    v[0] = fx_add(t0, t2);
    v[2] = fx_sub(t0, t2);
    v[1] = fx_addi<INV>(t1, t3);
    v[3] = fx_subi<INV>(t1, t3);
}
template <bool INV>
S2D_HD void fx_bf3(fx2* v) {
    const fx2 a = v[0], t1 = fx_add(v[1], v[2]), t2 = fx_sub(v[1], v[2]);
    const fx2 m = fx2{a.x - ((t1.x + 1) >> 1), a.y - ((t1.y + 1) >> 1)};
    const fx2 s = fx2{fx_mulc(t2.x, kFxSin3H, kFxSin3L), fx_mulc(t2.y, kFxSin3H, kFxSin3L)};
    v[0] = fx_add(a, t1);
    v[1] = fx_addi<INV>(m, s);
    v[2] = fx_subi<INV>(m, s);
}
// outputs 0 and 2 only
template <bool INV>
S2D_HD void fx_bf3_02(fx2* v) {
    const fx2 a = v[0], t1 = fx_add(v[1], v[2]), t2 = fx_sub(v[1], v[2]);
    const fx2 m = fx2{a.x - ((t1.x + 1) >> 1), a.y - ((t1.y + 1) >> 1)};
    const fx2 s = fx2{fx_mulc(t2.x, kFxSin3H, kFxSin3L), fx_mulc(t2.y, kFxSin3H, kFxSin3L)};
    v[0] = fx_add(a, t1);
    v[2] = fx_subi<INV>(m, s);
}
// (a, 0, c)
template <bool INV>
S2D_HD void fx_bf3_bzero(fx2* v) {
    const fx2 a = v[0], c = v[2];
    const fx2 m = fx2{a.x - ((c.x + 1) >> 1), a.y - ((c.y + 1) >> 1)};
    const fx2 s = fx2{fx_mulc(c.x, kFxSin3H, kFxSin3L), fx_mulc(c.y, kFxSin3H, kFxSin3L)};
    v[0] = fx_add(a, c);
    v[1] = fx_subi<INV>(m, s);
    v[2] = fx_addi<INV>(m, s);
}

// The high word's exponent-and-mantissa part: the maximum over a transform
// gives its exponent, 0x7ff0.... and above for an infinity or NaN.
S2D_HD int fx_magnitude(int hi) { return hi & 0x7FFFFFFF; }

// FP64 (words hi, lo) -> x with components of exponent emax in
// [2^(62 - n0), 2^(63 - n0)).
S2D_HD long long fx_from(int hi, unsigned lo, int emax, int n0) {
    int e = (hi >> 20) & 0x7FF;
    unsigned mh = (hi & 0xFFFFF) | 0x100000;
    if (emax < 64) {   // uniform over a transform: zeros and subnormals have no hidden bit
        mh = e ? mh : mh & 0xFFFFF;
        e = e ? e : 1;
    }   // (else they are shifted out)
    const unsigned long long m = ((unsigned long long)mh << 42) | ((unsigned long long)lo << 10);
    const long long t = (long long)((fx_shr(m, emax - e + n0 - 1) + 1) >> 1);
    const long long s = (long long)(hi >> 31);
    return (t ^ s) - s;
}

// Exponent base of a transform's results: emax its input's largest exponent,
// t the bits shifted out on the way.  2^16 and above: the input had an
// infinity or NaN.
S2D_HD int fx_exponent_base(int emax, int n0, int t) { return emax >= 0x7FF ? 1 << 16 : emax + n0 + 1 + t; }

// x -> FP64 bits, x 2^(eb - 1086) rounded to nearest, for 64 <= eb <= 2046: zero
// or in the normal range.  The conversion instruction runs at 2 per cycle and SM
// like all FP64, but beside the integer work, and the exponent is added to its
// result's high word: 5 instructions, where normalising and rounding with
// integer operations took 32.
S2D_HD long long fx_to_normal(long long x, int eb) {
    const double v = (double)x;
#ifdef __CUDA_ARCH__
    const int h = __double2hiint(v), l = __double2loint(v);
#else
    long long vb;
    __builtin_memcpy(&vb, &v, 8);
    const int h = (int)(vb >> 32), l = (int)vb;
#endif
    const int g = h ? h + (int)((unsigned)(eb - 1086) << 20) : 0;
    return (long long)(((unsigned long long)(unsigned)g << 32) | (unsigned)l);
}
// An eb of fx_exponent_base brought into that range, and the power of two that
// the results then lack: a product that overflows to infinity or underflows
// gradually with one rounding, as FP64 arithmetic does; NaN for an input with an
// infinity or NaN.  (With less than 2^-1022 every result is zero.)
S2D_HD int fx_normal_base(int eb) { return eb < 64 ? 64 : (eb > 2046 ? 2046 : eb); }
S2D_HD double fx_rest(int eb) {
    const int d = eb - fx_normal_base(eb), r = d < -1022 ? -1022 : (d > 1023 ? 1023 : d);
    const long long b = eb >= 1 << 16 ? 0x7FF8000000000000LL : (long long)(r + 1023) << 52;
#ifdef __CUDA_ARCH__
    return __longlong_as_double(b);
#else
    double v;
    __builtin_memcpy(&v, &b, 8);
    return v;
#endif
}

// One result by itself, flushed to zero below the normal range.
S2D_HD long long fx_to(long long x, int eb) {
    const int n = fx_normal_base(eb);
    const long long t = fx_to_normal(x, n);
    if (n == eb) return t;
    const int e = (int)((unsigned long long)t >> 52 & 0x7FF) + eb - n;
    if (eb >= 1 << 16) return 0x7FF8000000000000LL;
    if (e < 1 || x == 0) return 0;
    const long long sign = t & (long long)0x8000000000000000ULL;
    return e > 2046 ? sign | 0x7FF0000000000000LL : (t & (long long)0x800FFFFFFFFFFFFFULL) | (long long)e << 52;
}

// Magnitude bound of an element for the sum: |x| + |y| >= |z| of the high
// words, in units of 2^44, rounded up.
S2D_HD unsigned fx_weight(fx2 z) {
    const int a = (int)(z.x >> 32), b = (int)(z.y >> 32);
    return ((unsigned)((a < 0 ? -a : a) + (b < 0 ? -b : b) + 2) >> 12) + 1;
}

// Bits shifted out before a pass that brings the product of the radices to
// ns, for the limit |z| <= L = 3 sqrt(2) 2^60: one input element is at most
// per L, their sum at most sum 2^44, and by_limit = 2^44 / L (twice that for
// half the limit).
constexpr float kFxByLimit = 1.0f / (262144.0f * 1.06066f);
S2D_HD int fx_shift_total(int ns, float per, unsigned sum, float by_limit) {
    const float by_radix = (float)ns * per, by_sum = (float)sum * by_limit;
    const float f = by_radix < by_sum ? by_radix : by_sum;
#ifdef __CUDA_ARCH__
    const int b = __float_as_int(f);
#else
    int b;
    __builtin_memcpy(&b, &f, 4);
#endif
    const int e = ((b + 0x7FFFFF) >> 23) - 127;   // ceil(log2 f)
    return e > 0 ? e : 0;
}
// per of a transform whose largest component is in [2^(62 - n0), 2^(63 - n0))
// and whose element magnitudes are up to sqrt(2) times that (a hair less, so
// that 3 elements of n0 = 3 are not over the limit)
S2D_HD float fx_per(int n0) { return (n0 == 3 ? 1.0f / 3.0f : 1.0f / 6.0f) * 0.99999f; }

}  // namespace s2d
