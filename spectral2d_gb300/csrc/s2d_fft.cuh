// s2d_fft.cuh -- block-level mixed-radix Stockham FFT in shared memory.
//
// One transform of length M is owned by Tg = M/E consecutive threads, E = 12 or
// (small grids) 4 elements each; a CTA runs several transforms of the same
// length side by side.  Each pass with
// radix R is the self-sorting Stockham step (Govindaraju et al., SC'08):
// butterfly j (0 <= j < M/R) reads x[j + r*M/R], multiplies by the twiddle
// w^(r*(j mod Ns)*M/(Ns*R)) with w = exp(-2 pi i/M), does a radix-R DFT and
// writes x[(j/Ns)*Ns*R + j mod Ns + r*Ns], Ns being the product of the
// earlier radices.  The pass is done in place: every thread first loads all of
// its elements into registers, the CTA synchronises, then every thread writes
// its results.
//
// FP64 values are transformed in 64-bit block fixed point on the integer
// pipes (fx_run below; the arithmetic is in s2d_fixed.cuh): the first pass
// converts, the last converts back, the passes in between work on integers.
//
// FP32 runs the passes on floats: twiddles come from a table (a load, not a
// sincos), twiddled radix-4/2 passes use the FMA form (TwEnt).  Its cost is
// the shared-memory traffic and the barriers of the in-place passes.
#pragma once

#include "s2d_internal.h"

namespace s2d {

template <typename T>
struct Vec;
template <>
struct Vec<double> {
    using t = double2;
};
template <>
struct Vec<float> {
    using t = float2;
};

template <typename VT, typename T>
__device__ __forceinline__ VT mk(T x, T y) {
    VT r;
    r.x = x;
    r.y = y;
    return r;
}

// a * w (forward) or a * conj(w) (inverse)
template <bool INV, typename VT>
__device__ __forceinline__ VT twmul(VT a, VT w) {
    VT r;
    if (!INV) {
        r.x = a.x * w.x - a.y * w.y;
        r.y = a.x * w.y + a.y * w.x;
    } else {
        r.x = a.x * w.x + a.y * w.y;
        r.y = a.y * w.x - a.x * w.y;
    }
    return r;
}

template <bool INV, typename VT>
__device__ __forceinline__ void bf2(VT* v) {
    VT a = v[0], b = v[1];
    v[0].x = a.x + b.x;
    v[0].y = a.y + b.y;
    v[1].x = a.x - b.x;
    v[1].y = a.y - b.y;
}

// Radix-3 DFT: y1 = a - (b+c)/2 -/+ i sin(2pi/3) (b-c) (forward/inverse).
template <bool INV, typename VT>
__device__ __forceinline__ void bf3(VT* v) {
    using T = decltype(v[0].x);
    const T s = (T)0.86602540378443864676;
    const T h = (T)0.5;
    VT a = v[0], b = v[1], c = v[2];
    T t1x = b.x + c.x, t1y = b.y + c.y;
    T t2x = b.x - c.x, t2y = b.y - c.y;
    T mx = a.x - h * t1x, my = a.y - h * t1y;
    v[0].x = a.x + t1x;
    v[0].y = a.y + t1y;
    if (!INV) {
        v[1].x = mx + s * t2y;
        v[1].y = my - s * t2x;
        v[2].x = mx - s * t2y;
        v[2].y = my + s * t2x;
    } else {
        v[1].x = mx - s * t2y;
        v[1].y = my + s * t2x;
        v[2].x = mx + s * t2y;
        v[2].y = my - s * t2x;
    }
}

template <bool INV, typename VT>
__device__ __forceinline__ void bf4(VT* v) {
    VT a = v[0], b = v[1], c = v[2], d = v[3];
    auto t0x = a.x + c.x, t0y = a.y + c.y;
    auto t1x = a.x - c.x, t1y = a.y - c.y;
    auto t2x = b.x + d.x, t2y = b.y + d.y;
    auto t3x = b.x - d.x, t3y = b.y - d.y;
    v[0].x = t0x + t2x;
    v[0].y = t0y + t2y;
    v[2].x = t0x - t2x;
    v[2].y = t0y - t2y;
    if (!INV) {  // y1 = t1 - i t3, y3 = t1 + i t3
        v[1].x = t1x + t3y;
        v[1].y = t1y - t3x;
        v[3].x = t1x - t3y;
        v[3].y = t1y + t3x;
    } else {
        v[1].x = t1x - t3y;
        v[1].y = t1y + t3x;
        v[3].x = t1x + t3y;
        v[3].y = t1y - t3x;
    }
}

template <int R, bool INV, typename VT>
__device__ __forceinline__ void butterfly(VT* v) {
    if constexpr (R == 2) bf2<INV>(v);
    else if constexpr (R == 3) bf3<INV>(v);
    else bf4<INV>(v);
}

// j mod Ns by a multiply-high: q = floor(j mg / 2^32) with mg = ceil(2^32 /
// Ns) (Dims::mg, set on the host) is floor(j / Ns) exactly while
// j (mg Ns - 2^32) < 2^32, i.e. for every j < 2^32 / Ns (here j < M <= 6144).
// No integer division on the device: about 20 instructions per butterfly, on
// the integer pipes that the FP64 transforms are bound by.
struct ModNs {
    int Ns;
    unsigned mg;
    __device__ __forceinline__ ModNs(int ns, unsigned m) : Ns(ns), mg(m) {}
    __device__ __forceinline__ int operator()(int j) const {
        return Ns == 1 ? 0 : j - (int)__umulhi((unsigned)j, mg) * Ns;
    }
};

// floor(n / d) by the same multiply-high with m = ceil(2^32 / d), built once
// per thread (one division) and used per element: exact while
// n (m d - 2^32) < 2^32, which holds for the index splits of the column
// gathers and stores (n < 2^17, d < 2^14).  Small plans take G > 1
// transforms per CTA, and a division per element there was a third of the
// instructions of their latency-bound column kernels.
struct DivBy {
    int d;
    unsigned m;
    __device__ __forceinline__ explicit DivBy(int dd) : d(dd), m(dd > 1 ? 0xFFFFFFFFu / (unsigned)dd + 1u : 0u) {}
    __device__ __forceinline__ int operator()(int n) const { return d == 1 ? n : (int)__umulhi((unsigned)n, m); }
};

// Butterflies of radix R per thread with E elements per thread (T = M / E
// threads), and whether butterfly j exists (the last round may be partial
// when R does not divide E).
template <int E, int R>
constexpr int kFxNB = (E + R - 1) / R;
template <int E, int R>
__device__ __forceinline__ bool fx_on(int j, int M) {
    return E % R == 0 || j < M / R;
}

// One in-place Stockham pass of radix R over the transform in buf.
template <int E, int R, bool INV, typename VT>
__device__ __forceinline__ void fft_pass(VT* buf, int M, int Ns, unsigned mg, int tstep, int lane, int Tg,
                                         const VT* __restrict__ tw) {
    constexpr int NB = kFxNB<E, R>;
    VT v[NB][R];
    const int stride = M / R;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * Tg;
        if (!fx_on<E, R>(j, M)) continue;
#pragma unroll
        for (int r = 0; r < R; ++r) v[b][r] = buf[j + r * stride];
    }
    __syncthreads();
    const ModNs mod(Ns, mg);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * Tg;
        if (!fx_on<E, R>(j, M)) continue;
        const int k = mod(j);
        if (Ns > 1) {
            const int ts = k * tstep;
#pragma unroll
            for (int r = 1; r < R; ++r) v[b][r] = twmul<INV>(v[b][r], __ldg(&tw[r * ts]));
        }
        butterfly<R, INV>(v[b]);
        const int base = (j - k) * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r) buf[base + r * Ns] = v[b][r];
    }
    __syncthreads();
}

// Radix-3 DFT of (a, 0, c): 8 instead of 12 floating-point instructions.
template <bool INV, typename VT>
__device__ __forceinline__ void bf3_bzero(VT* v) {
    using T = decltype(v[0].x);
    const T s = (T)0.86602540378443864676;
    const T h = (T)0.5;
    const VT a = v[0], c = v[2];
    const T mx = a.x - h * c.x, my = a.y - h * c.y;
    v[0].x = a.x + c.x;
    v[0].y = a.y + c.y;
    if (!INV) {  // y1 = m + i s c, y2 = m - i s c
        v[1].x = mx - s * c.y;
        v[1].y = my + s * c.x;
        v[2].x = mx + s * c.y;
        v[2].y = my - s * c.x;
    } else {
        v[1].x = mx + s * c.y;
        v[1].y = my - s * c.x;
        v[2].x = mx - s * c.y;
        v[2].y = my + s * c.x;
    }
}

// First pass of an inverse transform whose input is zero in the middle third
// except at index M/3 -- every inverse transform here: the spectra are
// truncated to |k| <= K = M/3, so index n is non-zero only for n <= K or
// n >= M - K.  Butterfly j reads (x[j], x[j + M/3], x[j + 2M/3]); its middle
// input is zero for j > 0.
template <int E, bool INV, typename VT>
__device__ __forceinline__ void fft_pass3_midzero(VT* buf, int M, int lane, int Tg) {
    constexpr int NB = kFxNB<E, 3>;
    VT v[NB][3];
    const int stride = M / 3;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * Tg;
        if (!fx_on<E, 3>(j, M)) continue;
        v[b][0] = buf[j];
        v[b][1] = buf[j + stride];
        v[b][2] = buf[j + 2 * stride];
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * Tg;
        if (!fx_on<E, 3>(j, M)) continue;
        if (j == 0) bf3<INV>(v[b]);
        else bf3_bzero<INV>(v[b]);
        buf[j * 3] = v[b][0];
        buf[j * 3 + 1] = v[b][1];
        buf[j * 3 + 2] = v[b][2];
    }
    __syncthreads();
}

__device__ __forceinline__ float ffma(float a, float b, float c) { return fmaf(a, b, c); }

__device__ __forceinline__ float neg_if(float v, int cond) {
    return __int_as_float(__float_as_int(v) ^ ((cond != 0) << 31));
}

// x * i^q by register moves and sign flips only (integer operations).
template <typename VT>
__device__ __forceinline__ VT rot_iq(VT x, int q) {
    VT r;
    r.x = (q & 1) ? x.y : x.x;
    r.y = (q & 1) ? x.x : x.y;
    r.x = neg_if(r.x, (q + 1) & 2);
    r.y = neg_if(r.y, q & 2);
    return r;
}

// (x * i^q) * (1 + i t): two FMAs; the inverse uses conj(w) = i^-q c (1 - i t).
template <bool INV, typename VT, typename T>
__device__ __forceinline__ VT tw_fma(VT x, T t, int q) {
    const VT y = rot_iq(x, INV ? ((4 - q) & 3) : q);
    const T tt = INV ? -t : t;
    VT r;
    r.x = ffma(-tt, y.y, y.x);
    r.y = ffma(tt, y.x, y.y);
    return r;
}

// Radix-4 butterfly with FMA-form twiddles: 22 instructions instead of 12 (3
// complex products) + 16.
template <bool INV, typename VT>
__device__ __forceinline__ void bf4_fma(VT* v, const TwEnt<float>& e) {
    const VT a = v[0];
    const VT B = tw_fma<INV>(v[1], e.t1, e.q & 3);
    const VT Cc = tw_fma<INV>(v[2], e.t2, (e.q >> 2) & 3);
    const VT D = tw_fma<INV>(v[3], e.t3, (e.q >> 4) & 3);
    // t0,1 = a +- c2 C ; E,F = B +- (c3/c1) D ; y = t +- c1 E, t -+ i c1 F
    const float t0x = ffma(e.c2, Cc.x, a.x), t0y = ffma(e.c2, Cc.y, a.y);
    const float t1x = ffma(-e.c2, Cc.x, a.x), t1y = ffma(-e.c2, Cc.y, a.y);
    const float Ex = ffma(e.r31, D.x, B.x), Ey = ffma(e.r31, D.y, B.y);
    const float Fx = ffma(-e.r31, D.x, B.x), Fy = ffma(-e.r31, D.y, B.y);
    v[0].x = ffma(e.c1, Ex, t0x);
    v[0].y = ffma(e.c1, Ey, t0y);
    v[2].x = ffma(-e.c1, Ex, t0x);
    v[2].y = ffma(-e.c1, Ey, t0y);
    if (!INV) {  // y1 = t1 - i c1 F, y3 = t1 + i c1 F
        v[1].x = ffma(e.c1, Fy, t1x);
        v[1].y = ffma(-e.c1, Fx, t1y);
        v[3].x = ffma(-e.c1, Fy, t1x);
        v[3].y = ffma(e.c1, Fx, t1y);
    } else {
        v[1].x = ffma(-e.c1, Fy, t1x);
        v[1].y = ffma(e.c1, Fx, t1y);
        v[3].x = ffma(e.c1, Fy, t1x);
        v[3].y = ffma(-e.c1, Fx, t1y);
    }
}

// Radix-4 Stockham pass with FMA-form twiddles (Ns > 1).
template <int E, bool INV, typename VT>
__device__ __forceinline__ void fft_pass4_fma(VT* buf, int M, int Ns, unsigned mg, int lane, int Tg,
                                              const TwEnt<float>* __restrict__ tab) {
    constexpr int NB = kFxNB<E, 4>;
    VT v[NB][4];
    const int stride = M / 4;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * Tg;
#pragma unroll
        for (int r = 0; r < 4; ++r) v[b][r] = buf[j + r * stride];
    }
    __syncthreads();
    const ModNs mod(Ns, mg);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * Tg;
        const int k = mod(j);
        const TwEnt<float> e = tab[k];
        bf4_fma<INV>(v[b], e);
        const int base = (j - k) * 4 + k;
#pragma unroll
        for (int r = 0; r < 4; ++r) buf[base + r * Ns] = v[b][r];
    }
    __syncthreads();
}

// Radix-2 Stockham pass with an FMA-form twiddle (Ns > 1): y = a +- c1 B.
template <int E, bool INV, typename VT>
__device__ __forceinline__ void fft_pass2_fma(VT* buf, int M, int Ns, unsigned mg, int lane, int Tg,
                                              const TwEnt<float>* __restrict__ tab) {
    constexpr int NB = kFxNB<E, 2>;
    VT v[NB][2];
    const int stride = M / 2;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * Tg;
        v[b][0] = buf[j];
        v[b][1] = buf[j + stride];
    }
    __syncthreads();
    const ModNs mod(Ns, mg);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * Tg;
        const int k = mod(j);
        const float t1 = tab[k].t1, c1 = tab[k].c1;
        const int q = tab[k].q;
        const VT a = v[b][0];
        const VT B = tw_fma<INV>(v[b][1], t1, q & 3);
        const int base = (j - k) * 2 + k;
        VT y0, y1;
        y0.x = ffma(c1, B.x, a.x);
        y0.y = ffma(c1, B.y, a.y);
        y1.x = ffma(-c1, B.x, a.x);
        y1.y = ffma(-c1, B.y, a.y);
        buf[base] = y0;
        buf[base + Ns] = y1;
    }
    __syncthreads();
}

// ---- FP64 in block fixed point --------------------------------------------
// Passes over a transform of M elements in shared memory by T = M / E threads
// (E = 12 or 4 elements per thread); the forward transforms of direct plans
// (Dims::direct) run the radices in reverse order.

// Words of the CTA's transforms, eight each, set by their first users: the
// largest high word of the input, the sum of its magnitudes, the same of a
// second transform of the row, and a constant (re, im) that is kept out of the
// transform.  S2D_FX_GROUPS transforms per CTA at most: kFxGroups in the single
// runs' launches, 256 in the batch's.  (8 KB in all of them left the 2048^2
// kernels less L1 beside their three CTAs' shared memory: K3 631 -> 660 us per
// step.)
#ifndef S2D_FX_GROUPS
#define S2D_FX_GROUPS kFxGroups
#endif
__device__ __forceinline__ int* fx_words() {
    __shared__ __align__(16) int w[8 * S2D_FX_GROUPS];
    return w;
}
// Whether element 0 of an inverse transform of M elements, of magnitude m0, is
// so large beside the rest, of magnitude mr (both fx_magnitude), that the
// common exponent takes more bits from the rest than FP64 would.  It is then
// kept out of the fixed point and added in FP64: it enters every result alike,
// as in an FP64 transform, whose butterflies never twiddle it, so that its real
// part (the mean of u) takes no bits from the other results' imaginary parts
// (v).  With it always in, the tendency of ky = 0 of a perturbation 1e-6 of a
// flow that depends on y alone had errors of 3e-11 (64^2), in FP64 3e-15.
// The line: one large element alone leaves an error of about 0.6 sqrt(M) 2^-60
// of it, 2.9e-17 for M = 3072; the rest, smaller by up to 8 (16 for M <= 1024),
// keeps 2e-16 of its norm, an FP64 transform's.  Kept out where two numbers
// differ by a factor of two already, some rows of ordinary turbulence are, which
// then read their spectra again (96^2: 63.5 -> 65.5 us per step).
__device__ __forceinline__ bool fx_constant_out(int m0, int mr, int M) {
    return (m0 >> 20) > (mr >> 20) + (M <= 1024 ? 3 : 2);
}
// Maximum or sum over a transform into a zeroed word.  whole: the transform
// owns whole warps (32 divides T).
__device__ __forceinline__ void fx_reduce_max(int* word, int v, int lane, bool whole) {
    if (whole) {
        v = __reduce_max_sync(0xffffffffu, v);
        if ((lane & 31) == 0) atomicMax(word, v);
    } else {
        atomicMax(word, v);
    }
}
__device__ __forceinline__ void fx_reduce_add(int* word, unsigned v, int lane, bool whole) {
    if (whole) {
        v = __reduce_add_sync(0xffffffffu, v);
        if ((lane & 31) == 0) atomicAdd((unsigned*)word, v);
    } else {
        atomicAdd((unsigned*)word, v);
    }
}
__device__ __forceinline__ int fx_magnitude(double2 z) {
    return max(fx_magnitude(__double2hiint(z.x)), fx_magnitude(__double2hiint(z.y)));
}
__device__ __forceinline__ fx2 fx_from(double2 z, int emax, int n0) {
    return fx2{fx_from(__double2hiint(z.x), (unsigned)__double2loint(z.x), emax, n0),
               fx_from(__double2hiint(z.y), (unsigned)__double2loint(z.y), emax, n0)};
}
// n: fx_normal_base of the results' exponent base eb.  Where they differ, which
// is rare, the kernels multiply their results by fx_rest(eb) afterwards or in a
// copy of the last pass (beside each conversion every row pays for it: 2048^2
// 1770 us per step, 1787 with a branch there, 1833 with the product).
__device__ __forceinline__ double2 fx_to(fx2 z, int n) {
    return make_double2(__longlong_as_double(fx_to_normal(z.x, n)), __longlong_as_double(fx_to_normal(z.y, n)));
}
__device__ __forceinline__ fx2 fx_ld(const longlong2* buf, int i) {
    const longlong2 z = buf[i];
    return fx2{z.x, z.y};
}
__device__ __forceinline__ void fx_st(longlong2* buf, int i, fx2 z) { buf[i] = make_longlong2(z.x, z.y); }

// The exchange after a forward transform's first pass: radix-4 butterflies
// store elements 4 j + r, a stride of four (4-way bank conflicts in eight
// lanes), so that exchange goes through a permuted index that is
// conflict-free for these stores and for the next pass's loads.  The
// permutation stays within aligned blocks of 32 elements, so where T and M / 4
// are multiples of 32 it is applied to the thread's lane.
__device__ __forceinline__ bool swz_on(const Dims& d, int T) {
    return (T & 31) == 0 && ((d.M / 4) & 31) == 0 && d.npass > 2 && d.radix[d.npass - 2] == 4;
}
__device__ __forceinline__ int swz(int i) { return i ^ ((i >> 3) & 3) ^ ((i >> 2) & 4); }
// base of the four elements 4 j .. 4 j + 3 (element r at base ^ r)
__device__ __forceinline__ int swz4(int j, bool on) { return on ? swz(4 * j) : 4 * j; }

// The twiddled inputs of a butterfly, r bits shifted out on the way: by the R - 1
// factors w, or by those of position k of the table, read ahead of the first
// product or one by one.  Ahead, the direct kernels need fewer registers (80 at
// three CTAs per SM: 2048^2 K1 417 -> 392, K2 874 -> 833, K3 629 -> 610 us per
// step); fx_run only waits for them at once (512^2 conservative 291 -> 295).
__device__ __forceinline__ FxTw fx_tw(const FxTw* __restrict__ tab) {
    const int4 w = __ldg(reinterpret_cast<const int4*>(tab));
    return FxTw{w.x, w.y, w.z, w.w};
}
template <int R, bool INV>
__device__ __forceinline__ void fx_twiddle_by(fx2* v, const FxTw* w, int rsh) {
    if (rsh) {
        v[0].x = fx_round(v[0].x, rsh);
        v[0].y = fx_round(v[0].y, rsh);
    }
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = fx_cmul<INV>(v[r], w[r - 1], rsh);
}
template <int R, bool INV, bool AHEAD>
__device__ __forceinline__ void fx_twiddle(fx2* v, const FxTw* __restrict__ tab, int Ns, int k, int rsh) {
    if constexpr (AHEAD) {
        FxTw w[R - 1];
#pragma unroll
        for (int r = 1; r < R; ++r) w[r - 1] = fx_tw(tab + (r - 1) * Ns + k);
        fx_twiddle_by<R, INV>(v, w, rsh);
    } else {
        if (rsh) {
            v[0].x = fx_round(v[0].x, rsh);
            v[0].y = fx_round(v[0].y, rsh);
        }
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = fx_cmul<INV>(v[r], fx_tw(tab + (r - 1) * Ns + k), rsh);
    }
}
template <int R, bool INV>
__device__ __forceinline__ void fx_butterfly(fx2* v) {
    if constexpr (R == 2) fx_bf2<INV>(v);
    else if constexpr (R == 3) fx_bf3<INV>(v);
    else fx_bf4<INV>(v);
}

// One pass after the first, in place (all loads, barrier, all stores,
// barrier).  LAST: results rounded to FP64, eb their exponent base (fx_to), *c a
// constant to add (or null).
// lsw: the permutation of the lane for the loads (swz), or the lane.
template <int E, int R, bool INV, bool LAST = false, bool AHEAD = false>
__device__ __forceinline__ void fx_pass(longlong2* buf, int M, int Ns, unsigned mg, int lane, int T,
                                        const FxTw* __restrict__ tab, int rsh, int lsw, int eb = 0,
                                        const double2* c = nullptr) {
    constexpr int NB = kFxNB<E, R>;
    fx2 v[NB][R];
    const int stride = M / R;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        if (fx_on<E, R>(lane + b * T, M)) {
#pragma unroll
            for (int r = 0; r < R; ++r) v[b][r] = fx_ld(buf, lsw + b * T + r * stride);
        }
    }
    __syncthreads();
    const ModNs mod(Ns, mg);
    const int n = LAST ? fx_normal_base(eb) : 0;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * T;
        if (!fx_on<E, R>(j, M)) continue;
        const int k = mod(j);
        fx_twiddle<R, INV, AHEAD>(v[b], tab, Ns, k, rsh);
        fx_butterfly<R, INV>(v[b]);
        const int base = (j - k) * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if constexpr (LAST) {
                const double2 z = fx_to(v[b][r], n);
                buf[base + r * Ns] = make_longlong2(__double_as_longlong(z.x), __double_as_longlong(z.y));
            } else {
                fx_st(buf, base + r * Ns, v[b][r]);
            }
        }
    }
    if (LAST && (n != eb || c)) {   // this thread's results again (Ns = M / R: element j + r Ns)
        const double f = fx_rest(eb);
        const double2 a = c ? *c : make_double2(0.0, 0.0);
#pragma unroll 1
        for (int i = lane; i < stride; i += T)
#pragma unroll 1
            for (int e = i; e < M; e += stride) {
                double2* z = reinterpret_cast<double2*>(buf) + e;
                *z = make_double2(fma(z->x, f, a.x), fma(z->y, f, a.y));
            }
    }
    __syncthreads();
}

// Passes 1 .. npass - 2 of a direct plan (INV) or of its mirror image (forward);
// Ns and the bits shifted out so far are carried.
template <int E, bool INV>
__device__ __forceinline__ void fx_middle(longlong2* buf, const Dims& d, int lane, int T,
                                          const FxTw* __restrict__ tab, float per, unsigned sum, float by_limit,
                                          int& Ns, int& t) {
    for (int p = 1; p < d.npass - 1; ++p) {
        const int R = INV ? d.radix[p] : d.radix[d.npass - 1 - p];
        const unsigned mg = INV ? d.mg[p] : d.mgf[p];
        const FxTw* tp = tab + (INV ? d.twoff[p] : d.twofff[p]);
        const int tn = max(t, fx_shift_total(Ns * R, per, sum, by_limit));
        const int lsw = !INV && p == 1 && swz_on(d, T) ? swz(lane) : lane;
        if (R == 4) fx_pass<E, 4, INV, false, true>(buf, d.M, Ns, mg, lane, T, tp, tn - t, lsw);
        else if (R == 2) fx_pass<E, 2, INV, false, true>(buf, d.M, Ns, mg, lane, T, tp, tn - t, lane);
        else fx_pass<E, 3, INV, false, true>(buf, d.M, Ns, mg, lane, T, tp, tn - t, lane);
        t = tn;
        Ns *= R;
    }
}

// ---- the general FP64 transform, FP64 in and out (fft_run) -----------------
// First pass: the E elements of the thread from FP64, their common exponent
// emax, the sum of magnitudes, a radix-R DFT without twiddles.  PRUNE: radix 3
// with the middle input zero but for j = 0 (see fft_pass3_midzero).  out (INV):
// element 0 was kept out (fx_constant_out) and is in words + 4.
template <int E, int R, bool INV, bool PRUNE>
__device__ __forceinline__ int fx_first(longlong2* buf, int M, int lane, int Tg, int n0, int* words, bool& out) {
    constexpr int NB = kFxNB<E, R>;
    double2 z[NB][R];
    const int stride = M / R;
    int mx = 0;
    const int m0 = INV ? fx_magnitude(reinterpret_cast<const double2*>(buf)[0]) : 0;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * Tg;
        if (!fx_on<E, R>(j, M)) continue;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (PRUNE && r == 1 && (b > 0 || j > 0)) continue;
            z[b][r] = reinterpret_cast<const double2*>(buf)[j + r * stride];
            if (!INV || r || b || lane) mx = max(mx, fx_magnitude(z[b][r]));
        }
    }
    const bool whole = (Tg & 31) == 0;
    fx_reduce_max(&words[0], mx, lane, whole);
    __syncthreads();
    out = INV && fx_constant_out(m0, words[0], M);
    const int emax = (out ? words[0] : max(m0, words[0])) >> 20;
    if (out && lane == 0) {
        *reinterpret_cast<double2*>(words + 4) = z[0][0];
        z[0][0] = make_double2(0.0, 0.0);
    }
    unsigned sum = 0;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * Tg;
        if (!fx_on<E, R>(j, M)) continue;
        fx2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (PRUNE && r == 1 && (b > 0 || j > 0)) continue;
            v[r] = fx_from(z[b][r], emax, n0);
            sum += fx_weight(v[r]);
        }
        if constexpr (PRUNE) {
            if (b > 0 || j > 0) fx_bf3_bzero<INV>(v);
            else fx_bf3<INV>(v);
        } else {
            fx_butterfly<R, INV>(v);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) fx_st(buf, j * R + r, v[r]);
    }
    fx_reduce_add(&words[1], sum, lane, whole);
    __syncthreads();
    return emax;
}

// The FP64 transform (see fft_run).  An infinity or NaN reaches every result.
template <bool INV, int E, bool APART>
__device__ __forceinline__ void fx_run(longlong2* buf, const Dims& d, int lane, const FxTw* __restrict__ tab) {
    int* words = fx_words() + 8 * ((int)threadIdx.x / d.Tg);
    if (lane == 0) words[0] = words[1] = 0;
    __syncthreads();
    const int R0 = d.radix[0];
    const int n0 = R0 == 4 ? 4 : 3;
    int emax;
    bool out;
    if (INV && R0 == 3 && 3 * d.K == d.M) emax = fx_first<E, 3, INV, INV>(buf, d.M, lane, d.Tg, n0, words, out);
    else if (R0 == 3) emax = fx_first<E, 3, INV, false>(buf, d.M, lane, d.Tg, n0, words, out);
    else if (R0 == 4) emax = fx_first<E, 4, INV, false>(buf, d.M, lane, d.Tg, n0, words, out);
    else emax = fx_first<E, 2, INV, false>(buf, d.M, lane, d.Tg, n0, words, out);
    const unsigned sum = (unsigned)words[1];
    if (INV && APART && lane == 0) {
        words[3] = out;
        if (!out) *reinterpret_cast<double2*>(words + 4) = make_double2(0.0, 0.0);
    }
    const float per = fx_per(n0);
    int Ns = R0, t = 0;
    for (int p = 1; p < d.npass; ++p) {
        const int R = d.radix[p];
        const unsigned mg = d.mg[p];
        const FxTw* tp = tab + d.twoff[p];
        const int tn = max(t, fx_shift_total(Ns * R, per, sum, kFxByLimit));
        const int rsh = tn - t;
        t = tn;
        if (p + 1 < d.npass) {
            if (R == 4) fx_pass<E, 4, INV>(buf, d.M, Ns, mg, lane, d.Tg, tp, rsh, lane);
            else if (R == 2) fx_pass<E, 2, INV>(buf, d.M, Ns, mg, lane, d.Tg, tp, rsh, lane);
            else fx_pass<E, 3, INV>(buf, d.M, Ns, mg, lane, d.Tg, tp, rsh, lane);
        } else {
            const int eb = fx_exponent_base(emax, n0, t);
            const double2* c = INV && !APART && out ? reinterpret_cast<const double2*>(words + 4) : nullptr;
            if (R == 4) fx_pass<E, 4, INV, true>(buf, d.M, Ns, mg, lane, d.Tg, tp, rsh, lane, eb, c);
            else if (R == 2) fx_pass<E, 2, INV, true>(buf, d.M, Ns, mg, lane, d.Tg, tp, rsh, lane, eb, c);
            else fx_pass<E, 3, INV, true>(buf, d.M, Ns, mg, lane, d.Tg, tp, rsh, lane, eb, c);
        }
        Ns *= R;
    }
}

// The constant that an FP64 inverse transform with APART left out of its
// results (zero and false if none), from its end to the next one's start; g:
// the transform's group of the CTA.
struct FxMean {
    double2 m;
    bool out;
};
__device__ __forceinline__ FxMean fx_mean(int g) {
    const int* words = fx_words() + 8 * g;
    return FxMean{*reinterpret_cast<const double2*>(words + 4), words[3] != 0};
}

// FP32: passes [p0, p1) of the plan over the transform in buf.
__device__ __forceinline__ const TwEnt<float>* f32_tab(const Dims& d, const float2* tw) {
    return reinterpret_cast<const TwEnt<float>*>(reinterpret_cast<const char*>(tw) + d.tab_bytes);
}
template <int E, bool INV>
__device__ __forceinline__ void f32_passes(float2* buf, const Dims& d, int lane, const float2* __restrict__ tw, int p0,
                                           int p1) {
    const TwEnt<float>* tab = f32_tab(d, tw);
    int Ns = p0 == 0 ? 1 : d.radix[0];   // p0 is 0 or 1
    for (int p = p0; p < p1; ++p) {
        const int R = d.radix[p];
        const int off = d.twoff[p];
        const unsigned mg = d.mg[p];
        if (INV && p == 0 && R == 3 && 3 * d.K == d.M) {
            fft_pass3_midzero<E, INV>(buf, d.M, lane, d.Tg);
        } else if (R == 4) {
            if (off >= 0) fft_pass4_fma<E, INV>(buf, d.M, Ns, mg, lane, d.Tg, tab + off);
            else fft_pass<E, 4, INV>(buf, d.M, Ns, mg, d.tstep[p], lane, d.Tg, tw);
        } else if (R == 2) {
            if (off >= 0) fft_pass2_fma<E, INV>(buf, d.M, Ns, mg, lane, d.Tg, tab + off);
            else fft_pass<E, 2, INV>(buf, d.M, Ns, mg, d.tstep[p], lane, d.Tg, tw);
        } else {
            fft_pass<E, 3, INV>(buf, d.M, Ns, mg, d.tstep[p], lane, d.Tg, tw);
        }
        Ns *= R;
    }
}

// Full transform: unnormalised, sign -1 (forward) or +1 (INV).  Every thread
// of the CTA must call it (it synchronises the CTA); starts with a barrier so
// that callers may fill buf just before.  tw points at the handle's twiddles
// (Dims::twoff, tab_bytes).  Inverse transforms of truncated spectra (input
// zero for K < n < M - K, K = M/3: the inverse transforms of this library)
// take the pruned first radix-3 pass.  E elements per thread (d.Tg = M / E).
// APART: an inverse transform may leave its element 0 to the caller (fx_mean).
template <bool INV, int E = kElemsPerThread, bool APART = false, typename VT>
__device__ __forceinline__ void fft_run(VT* buf, const Dims& d, int lane, const VT* __restrict__ tw) {
    using T = decltype(buf[0].x);
    if constexpr (sizeof(T) == 8) {
        fx_run<INV, E, APART>(reinterpret_cast<longlong2*>(buf), d, lane, reinterpret_cast<const FxTw*>(tw));
    } else {
        __syncthreads();
        f32_passes<E, INV>(buf, d, lane, tw, 0, d.npass);
    }
}

}  // namespace s2d
