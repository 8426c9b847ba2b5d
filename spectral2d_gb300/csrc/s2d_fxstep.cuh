// s2d_fxstep.cuh -- the three right-hand-side kernels' transforms in FP64
// (64-bit block fixed point, s2d_fixed.cuh), for direct plans
// (Dims::direct): E = 12 or 4 elements per thread, T = Dims::Tg = M / E
// threads per transform.  The first pass of a transform reads its input from
// global memory and the last one writes its results there, so a transform of
// p passes exchanges its elements p - 1 times through shared memory.
#pragma once

#include <type_traits>

#include "s2d_step.cuh"

namespace s2d {

// K1: inverse y-transform of one column (see yinv_body).
template <int E>
__device__ __forceinline__ void fx_yinv_body(const Dims& d, const double2* __restrict__ S,
                                             const double* __restrict__ rk2, const FieldSet& fs,
                                             const FxTw* __restrict__ tw, int G, int blk, double2* bufs) {
    constexpr int NB = kFxNB<E, 3>;
    const int M = d.M, K = d.K, T = d.Tg;
    const int g = threadIdx.x / T;
    const int lane = threadIdx.x - g * T;
    const int ncg = (d.KX + G - 1) / G;
    const int f = blk / ncg;
    const int kx = (blk - f * ncg) * G + g;
    const bool active = kx < d.KX && g < G;
    int op;
    void* outp;
    const double* tab;
    switch (f) {   // select without dynamic indexing of the parameter struct
        case 0: op = fs.op[0]; outp = fs.out[0]; tab = fs.tab[0]; break;
        case 1: op = fs.op[1]; outp = fs.out[1]; tab = fs.tab[1]; break;
        case 2: op = fs.op[2]; outp = fs.out[2]; tab = fs.tab[2]; break;
        default: op = fs.op[3]; outp = fs.out[3]; tab = fs.tab[3]; break;
    }
    if (op == OP_TU || op == OP_TV) rk2 = tab;   // the factor table takes the 1/k^2 table's place
    longlong2* buf = reinterpret_cast<longlong2*>(bufs + (size_t)g * M);
    int* words = fx_words() + 8 * g;
    if (lane == 0) words[0] = words[1] = 0;
    const double2* col = S + (size_t)(active ? kx : 0) * d.ldS;
    const double* rcol = rk2 + (size_t)(active ? kx : 0) * d.ldS;

    // radix 3 on (x[j], x[j + K], x[j + 2K]): row j (ky = j), 0 (ky = K for
    // j = 0), and row j + K + 1 (ky = j - K)
    double2 x0[NB], x2[NB], xm = make_double2(0.0, 0.0);
    int mx = 0;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * T;
        x0[b] = x2[b] = make_double2(0.0, 0.0);
        if (active && fx_on<E, 3>(j, M)) {
            x0[b] = __ldcg(&col[j]);
            x2[b] = __ldcg(&col[j + K + 1]);
        }
    }
    if (active && lane == 0) xm = __ldcg(&col[K]);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * T;
        if (active && fx_on<E, 3>(j, M)) {
            x0[b] = apply_op(op, x0[b], kx, j, rcol[j]);
            x2[b] = apply_op(op, x2[b], kx, j - K, rcol[j + K + 1]);
            mx = max(mx, max(fx_magnitude(x0[b]), fx_magnitude(x2[b])));
        }
    }
    if (active && lane == 0) {
        xm = apply_op(op, xm, kx, K, rcol[K]);
        mx = max(mx, fx_magnitude(xm));
    }
    const bool whole = (T & 31) == 0;
    __syncthreads();
    fx_reduce_max(&words[0], mx, lane, whole);
    __syncthreads();
    const int emax = words[0] >> 20;
    unsigned sum = 0;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * T;
        if (!fx_on<E, 3>(j, M)) continue;
        fx2 v[3];
        v[0] = fx_from(x0[b], emax, 3);
        v[2] = fx_from(x2[b], emax, 3);
        sum += fx_weight(v[0]) + fx_weight(v[2]);
        if (b == 0 && lane == 0) {
            v[1] = fx_from(xm, emax, 3);
            sum += fx_weight(v[1]);
            fx_bf3<true>(v);
        } else {
            fx_bf3_bzero<true>(v);
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) fx_st(buf, 3 * j + r, v[r]);
    }
    fx_reduce_add(&words[1], sum, lane, whole);
    __syncthreads();
    sum = (unsigned)words[1];
    const float per = fx_per(3);
    int Ns = 3, t = 0;
    fx_middle<E, true>(buf, d, lane, T, tw, per, sum, kFxByLimit, Ns, t);

    // last pass, radix 4 (Ns = M / 4): results y = j + r M / 4 to the rows
    const int tn = max(t, fx_shift_total(M, per, sum, kFxByLimit));
    const int eb = fx_exponent_base(emax, 3, tn), n = fx_normal_base(eb);
    const FxTw* tp = tw + d.twoff[d.npass - 1];
    double2* out = reinterpret_cast<double2*>(outp) + kx;
    // (results that need more work: to the buffer, whose elements this thread has
    // read; one store either way, so that others pay for no branch)
    const bool park = n != eb;
    double2* to = park ? reinterpret_cast<double2*>(buf) : out;
    const int ld = park ? 1 : d.ldI;
#pragma unroll
    for (int b = 0; b < kFxNB<E, 4>; ++b) {
        const int j = lane + b * T;
        fx2 v[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) v[r] = fx_ld(buf, j + r * (M / 4));
        fx_twiddle<4, true, true>(v, tp, M / 4, j, tn - t);
        fx_bf4<true>(v);
        if (active) {
#pragma unroll
            for (int r = 0; r < 4; ++r) to[(size_t)(j + r * (M / 4)) * ld] = fx_to(v[r], n);
        }
    }
    if (active && park) {   // (T divides M / 4: the rows lane + i T are this thread's)
        const double f = fx_rest(eb);
#pragma unroll 1
        for (int y = lane; y < M; y += T) out[(size_t)y * d.ldI] = make_double2(to[y].x * f, to[y].y * f);
    }
}

// K2, Basdevant form, of one row (see xpass_bas_body), everything between the
// half spectra read and written in fixed point: u + i v, its inverse
// transform, the products u v and v^2 - u^2 = (v - u)(v + u), the forward
// transform (mirrored radices: the inverse's last radix-4 butterfly leaves in
// a thread just the elements that the forward's first one takes) and the
// split.  A thread's radix-3 butterflies come in pairs (q, K - q), whose
// inputs z(k), z(M - k) of the first pass and outputs P(k), P(M - k) of the
// last one belong to the same two entries of the half spectra, so that the
// Hermitian extension and the split stay in registers.  q = 0 pairs 0 with
// K / 2 and takes z(K), P(K) besides.
// Where the row's means (kx = 0) would take bits from the rest
// (fx_constant_out) they are left out of the transforms, and the products'
// parts that are linear in the rest are added in FP64 (linear_part_bas): at
// the end, in a copy of the last pass, so that other rows pay for no more than
// one branch (2048^2 K2: 824 us per step; in one copy 880, with the results
// parked in the buffer 836, by one store through a chosen pointer 830 and 4689
// against 4501 at 4096^2).  The copy also takes results whose exponents leave
// the normal range (fx_rest).
// scale: factor of the results (1 when u and v are prescaled).
template <int E>
__device__ __forceinline__ void fx_xpass_body(const Dims& d, double2* Iu, double2* Iv, const FxTw* __restrict__ tw,
                                              int G, double scale, int blk, double2* bufs) {
    constexpr int NP = E == 12 ? 2 : 1;   // pairs per thread: K / 2 over T = 3 K / E
    constexpr int NB = kFxNB<E, 4>;
    const int M = d.M, K = d.K, T = d.Tg;
    const int g = threadIdx.x / T;
    const int lane = threadIdx.x - g * T;
    const int y = blk * G + g;
    const bool active = y < d.rows && g < G;
    longlong2* buf = reinterpret_cast<longlong2*>(bufs + (size_t)g * M);
    int* words = fx_words() + 8 * g;
    if (lane == 0) *reinterpret_cast<int4*>(words) = make_int4(0, 0, 0, 0);
    double2* urow = Iu + (size_t)(active ? y : 0) * d.ldI;
    double2* vrow = Iv + (size_t)(active ? y : 0) * d.ldI;
    double2* means = reinterpret_cast<double2*>(words + 4);
    const bool whole = (T & 31) == 0;

    // ---- inverse, first pass
    double2 ua[NP], va[NP], ub[NP], vb[NP], um = make_double2(0.0, 0.0), vm = um;
    int mx = 0;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int q = lane + p * T;
        ua[p] = va[p] = ub[p] = vb[p] = make_double2(0.0, 0.0);
        if (active && (E == 12 || q < K / 2)) {
            const int q2 = q ? K - q : K / 2;
            ua[p] = __ldcg(&urow[q]);
            va[p] = __ldcg(&vrow[q]);
            ub[p] = __ldcg(&urow[q2]);
            vb[p] = __ldcg(&vrow[q2]);
        }
    }
    if (active && lane == 0) {
        um = __ldcg(&urow[K]);
        vm = __ldcg(&vrow[K]);
        ua[0].y = va[0].y = 0.0;   // kx = 0 contributes its real parts only
    }
    if (lane == 0) *means = make_double2(ua[0].x, va[0].x);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        mx = max(mx, max(fx_magnitude(ub[p]), fx_magnitude(vb[p])));
        if (p || lane) mx = max(mx, max(fx_magnitude(ua[p]), fx_magnitude(va[p])));
    }
    mx = max(mx, max(fx_magnitude(um), fx_magnitude(vm)));
    __syncthreads();
    fx_reduce_max(&words[0], mx, lane, whole);
    __syncthreads();
    const int m0 = fx_magnitude(*means), mr = words[0];
    const bool out = fx_constant_out(m0, mr, M);   // (the means are looked at apart)
    const int emax = (out ? mr : max(m0, mr)) >> 20;
    if (out && lane == 0) ua[0].x = va[0].x = 0.0;
    unsigned sum = 0;
    // components below 2^59 (n0 = 4), so that those of u + i v are below 2^60
    auto zp = [](fx2 a, fx2 b) { return fx2{a.x - b.y, a.y + b.x}; };    // z(k)
    auto zm = [](fx2 a, fx2 b) { return fx2{a.x + b.y, b.x - a.y}; };    // z(M - k)
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int q = lane + p * T;
        if (E != 12 && q >= K / 2) continue;
        const int q2 = q ? K - q : K / 2;
        const fx2 a = fx_from(ua[p], emax, 4), b = fx_from(va[p], emax, 4);
        const fx2 a2 = fx_from(ub[p], emax, 4), b2 = fx_from(vb[p], emax, 4);
        fx2 v[3], w[3];
        v[0] = zp(a, b);
        w[0] = zp(a2, b2);
        if (p == 0 && lane == 0) {
            const fx2 am = fx_from(um, emax, 4), bm = fx_from(vm, emax, 4);
            v[1] = zp(am, bm);
            v[2] = zm(am, bm);
            w[2] = zm(a2, b2);
            sum += fx_weight(v[1]);
        } else {
            v[2] = zm(a2, b2);
            w[2] = zm(a, b);
        }
        sum += fx_weight(v[0]) + fx_weight(v[2]) + fx_weight(w[0]) + fx_weight(w[2]);
        if (p == 0 && lane == 0) fx_bf3<true>(v);
        else fx_bf3_bzero<true>(v);
        fx_bf3_bzero<true>(w);
#pragma unroll
        for (int r = 0; r < 3; ++r) fx_st(buf, 3 * q + r, v[r]);
#pragma unroll
        for (int r = 0; r < 3; ++r) fx_st(buf, 3 * q2 + r, w[r]);
    }
    fx_reduce_add(&words[1], sum, lane, whole);
    __syncthreads();
    sum = (unsigned)words[1];
    int Ns = 3, t = 0;
    fx_middle<E, true>(buf, d, lane, T, tw, fx_per(3), sum, kFxByLimit, Ns, t);

    // ---- inverse, last pass: z = u + i v at n = j + r M / 4
    fx2 z[NB][4];
    const int tn = max(t, fx_shift_total(M, fx_per(3), sum, kFxByLimit));
    int m2 = 0;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * T;
#pragma unroll
        for (int r = 0; r < 4; ++r) z[b][r] = fx_ld(buf, j + r * (M / 4));
        fx_twiddle<4, true, true>(z[b], tw + d.twoff[d.npass - 1], M / 4, j, tn - t);
        fx_bf4<true>(z[b]);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            m2 = max(m2, max(abs((int)(z[b][r].x >> 32)), abs((int)(z[b][r].y >> 32))));
        }
    }
    fx_reduce_max(&words[2], m2, lane, whole);
    __syncthreads();
    // the row's largest component to [2^60, 2^61): |z| <= 2^61.5, |z^2| >> 64
    // <= 2^59, four of them <= 2^61 of the forward's limit 2^61.085 (half the
    // usual one: the split adds two results)
    const int sh = __clz(words[2]) - 3;
    // value = x 2^(eb - 1086)
    const int ebz = fx_exponent_base(emax, 4, tn);
    const bool sw = swz_on(d, T);
    int ebp = ebz >= 1 << 16 ? 1 << 16 : 2 * (ebz - sh) - 1022;
    sum = 0;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * T;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            long long u = z[b][r].x, v = z[b][r].y;
            if (sh >= 0) {
                u <<= sh;
                v <<= sh;
            } else {
                u >>= -sh;
                v >>= -sh;
            }
            z[b][r] = fx2{fx_mul64(u, v), fx_mul64(v - u, v + u)};
            sum += fx_weight(z[b][r]);
        }
        // ---- forward, first pass (radix 4)
        fx_bf4<false>(z[b]);
#pragma unroll
        for (int r = 0; r < 4; ++r) fx_st(buf, swz4(j, sw) ^ r, z[b][r]);
    }
    fx_reduce_add(&words[3], sum, lane, whole);
    __syncthreads();
    sum = (unsigned)words[3];
    const float per = 0.2357f;   // 2^59 / 2^61.085
    Ns = 4;
    t = 0;
    fx_middle<E, false>(buf, d, lane, T, tw, per, sum, 2.0f * kFxByLimit, Ns, t);

    // ---- forward, last pass (radix 3, Ns = K): P(j), P(j + 2K); the split
    const int tf = max(t, fx_shift_total(M, per, sum, 2.0f * kFxByLimit));
    if (ebp < 1 << 16) ebp += tf;
    const int n = fx_normal_base(ebp);
    const FxTw* tp = tw + d.twofff[d.npass - 1];
    auto put = [&](auto add, int k, fx2 p, fx2 c) {   // c = P(M - k)
        double2 a = fx_to(fx2{p.x + c.x, p.y - c.y}, n), b = fx_to(fx2{p.y + c.y, c.x - p.x}, n);
        if (scale != 1.0) {
            a = make_double2(a.x * scale, a.y * scale);
            b = make_double2(b.x * scale, b.y * scale);
        }
        if constexpr (add.value) {
            double2 U = make_double2(0.0, 0.0), V = U;
            if (out) {   // (this thread alone reads and writes entry k)
                U = __ldcg(&urow[k]);
                V = __ldcg(&vrow[k]);
                linear_part_bas(U, V, *means, 2.0 * M * scale, k == 0);
            }
            const double f = fx_rest(ebp);
            a = make_double2(fma(a.x, f, U.x), fma(a.y, f, U.y));
            b = make_double2(fma(b.x, f, V.x), fma(b.y, f, V.y));
        }
        urow[k] = a;
        vrow[k] = b;
    };
    // the first butterflies' twiddles, read before the branch so as not to wait
    // for them behind the last barrier
    const FxTw t0[2] = {fx_tw(tp + lane), fx_tw(tp + K + lane)};
    const int l2 = lane ? K - lane : K / 2;
    const FxTw t1[2] = {fx_tw(tp + l2), fx_tw(tp + K + l2)};
    auto split = [&](auto add) {
#pragma unroll(add.value ? 1 : NP)
        for (int p = 0; p < NP; ++p) {   // (unrolled, the rare form would spill)
            const int q = lane + p * T;
            if (E != 12 && q >= K / 2) continue;
            const int q2 = q ? K - q : K / 2;
            fx2 v[3], w[3];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                v[r] = fx_ld(buf, q + r * K);
                w[r] = fx_ld(buf, q2 + r * K);
            }
            if (p == 0) {
                fx_twiddle_by<3, false>(v, t0, tf - t);
                fx_twiddle_by<3, false>(w, t1, tf - t);
            } else {
                fx_twiddle<3, false, true>(v, tp, K, q, tf - t);
                fx_twiddle<3, false, true>(w, tp, K, q2, tf - t);
            }
            if (p == 0 && lane == 0) fx_bf3<false>(v);
            else fx_bf3_02<false>(v);
            fx_bf3_02<false>(w);
            if (active) {
                const bool first = p == 0 && lane == 0;
                if (first) put(add, K, v[1], v[2]);
                put(add, q, v[0], first ? v[0] : w[2]);
                put(add, q2, w[0], first ? w[2] : v[2]);
            }
        }
    };
    if (out || n != ebp) split(std::true_type{});
    else split(std::false_type{});
}

// K3's transform: column kx of one product, read from the half-spectral rows
// (mirrored radices, so that the retained rows are outputs 0 and 2 of the
// last radix-3 butterflies).  sink(jc) is where retained row jc goes, or null;
// SYNC: a barrier between the last pass's loads and the stores (in buf).
template <int E, bool SYNC, typename Sink>
__device__ __forceinline__ void fx_yfwd_column(const Dims& d, const double2* __restrict__ I, bool active, int kx,
                                               const FxTw* __restrict__ tw, int g, int lane, longlong2* buf,
                                               Sink sink) {
    constexpr int NB = kFxNB<E, 4>, N3 = kFxNB<E, 3>;
    const int M = d.M, K = d.K, T = d.Tg;
    int* words = fx_words() + 8 * g;
    if (lane == 0) words[0] = words[1] = 0;
    double2 x[NB][4];
    int mx = 0;
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            x[b][r] = make_double2(0.0, 0.0);
            if (active) x[b][r] = __ldcg(&I[(size_t)(lane + b * T + r * (M / 4)) * d.ldI + kx]);
        }
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int r = 0; r < 4; ++r) mx = max(mx, fx_magnitude(x[b][r]));
    const bool whole = (T & 31) == 0;
    __syncthreads();
    fx_reduce_max(&words[0], mx, lane, whole);
    __syncthreads();
    const int emax = words[0] >> 20;
    const bool sw = swz_on(d, T);
    unsigned sum = 0;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        fx2 v[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            v[r] = fx_from(x[b][r], emax, 4);
            sum += fx_weight(v[r]);
        }
        fx_bf4<false>(v);
#pragma unroll
        for (int r = 0; r < 4; ++r) fx_st(buf, swz4(lane + b * T, sw) ^ r, v[r]);
    }
    fx_reduce_add(&words[1], sum, lane, whole);
    __syncthreads();
    sum = (unsigned)words[1];
    const float per = fx_per(4);
    int Ns = 4, t = 0;
    fx_middle<E, false>(buf, d, lane, T, tw, per, sum, kFxByLimit, Ns, t);
    const int tn = max(t, fx_shift_total(M, per, sum, kFxByLimit));
    const int eb = fx_exponent_base(emax, 4, tn), n = fx_normal_base(eb);
    const FxTw* tp = tw + d.twofff[d.npass - 1];
    fx2 v[N3][3];
    auto put = [&](int jc, fx2 z) {
        if (double2* o = sink(jc)) *o = fx_to(z, n);
    };
#pragma unroll
    for (int b = 0; b < N3; ++b) {
        const int j = lane + b * T;
        if (!fx_on<E, 3>(j, M)) continue;
#pragma unroll
        for (int r = 0; r < 3; ++r) v[b][r] = fx_ld(buf, j + r * K);
    }
    if (SYNC) __syncthreads();
#pragma unroll
    for (int b = 0; b < N3; ++b) {
        const int j = lane + b * T;
        if (!fx_on<E, 3>(j, M)) continue;
        fx_twiddle<3, false, true>(v[b], tp, K, j, tn - t);
        if (b == 0 && lane == 0) {
            fx_bf3<false>(v[b]);
            put(K, v[b][1]);
        } else {
            fx_bf3_02<false>(v[b]);
        }
        put(j, v[b][0]);
        put(j + K + 1, v[b][2]);
    }
    if (n != eb) {
        const double f = fx_rest(eb);
        auto again = [&](int jc) {
            if (double2* o = sink(jc)) *o = make_double2(o->x * f, o->y * f);
        };
        if (lane == 0) again(K);
#pragma unroll 1
        for (int j = lane; j < K; j += T) {
            again(j);
            again(j + K + 1);
        }
    }
}

// The split K3's column transform (see yfwd_col_body).
template <int E>
__device__ __forceinline__ void fx_yfwd_col_body(const Dims& d, const double2* __restrict__ Iu,
                                                 const double2* __restrict__ Iv, double2* OutU, double2* OutV,
                                                 const FxTw* __restrict__ tw, int G, int blk, double2* bufs) {
    const int g = threadIdx.x / d.Tg;
    const int lane = threadIdx.x - g * d.Tg;
    const int ncg = (d.KX + G - 1) / G;
    const int f = blk / ncg;
    const int kx = (blk - f * ncg) * G + g;
    const bool active = kx < d.KX && g < G;
    double2* out = (f ? OutV : OutU) + (size_t)(active ? kx : 0) * d.ldS;
    fx_yfwd_column<E, false>(d, f ? Iv : Iu, active, kx, tw, g, lane,
                             reinterpret_cast<longlong2*>(bufs + (size_t)g * d.M),
                             [&](int jc) { return active ? out + jc : nullptr; });
}

// K3 in one kernel (see yfwd_body): 2G transforms, blockDim / T at a time,
// their retained rows left in shared memory, then the epilogue.
template <int E>
__device__ __forceinline__ bool fx_yfwd_body(const Dims& d, const double2* __restrict__ Iu,
                                             const double2* __restrict__ Iv, double2* S0, double2* S1, double2* Sdw,
                                             const double2* __restrict__ src, int stage, double dt, const Phys& ph,
                                             const FxTw* __restrict__ tw, int G, int blk, double2* bufs) {
    const int t = threadIdx.x / d.Tg;
    const int lane = threadIdx.x - t * d.Tg;
    const int kx0 = blk * G;
    const int gtot = min(G, d.KX - kx0);
    const int nconc = blockDim.x / d.Tg;
    for (int t0 = 0; t0 < 2 * G; t0 += nconc) {
        const int i = t0 + t, f = i >= G, gg = i - f * G;   // buffer i: field f, column gg
        double2* buf = bufs + (size_t)i * d.M;
        fx_yfwd_column<E, true>(d, f ? Iv : Iu, gg < gtot, kx0 + gg, tw, t, lane, reinterpret_cast<longlong2*>(buf),
                                [&](int jc) { return buf + jc; });
        __syncthreads();
    }
    bool bad = false;
    const DivBy byKY(d.KY);
    for (int idx = threadIdx.x; idx < gtot * d.KY; idx += blockDim.x) {
        const int gg = gtot == 1 ? 0 : byKY(idx);
        const int jc = idx - gg * d.KY;
        bad |= stage_point<double>(d, bufs[(size_t)gg * d.M + jc], bufs[(size_t)(G + gg) * d.M + jc], kx0 + gg, jc, S0,
                                   S1, Sdw, src, stage, dt, ph);
    }
    return bad;
}

}  // namespace s2d
