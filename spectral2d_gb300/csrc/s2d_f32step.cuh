// s2d_f32step.cuh -- the three right-hand-side kernels' transforms in FP32 for
// direct plans (Dims::direct): E = 12 or 4 elements per thread, T = Dims::Tg =
// M / E threads per transform, the first pass reading its input from global
// memory and the last one handing its results on, so that a transform of p
// passes exchanges its elements p - 1 times through shared memory.  Every
// element goes through the same operations as in the general kernels
// (s2d_step.cuh), so the results have the same bits.
#pragma once

#include "s2d_step.cuh"

namespace s2d {

// The last pass's butterflies: z[b][r] = element lane + b T + r M / 4.
template <int E, bool INV>
__device__ __forceinline__ void f32_last4(const float2* buf, const Dims& d, int lane, const float2* __restrict__ tw,
                                          float2 (*z)[4]) {
    const TwEnt<float>* tab = f32_tab(d, tw) + d.twoff[d.npass - 1];
#pragma unroll
    for (int b = 0; b < kFxNB<E, 4>; ++b) {
        const int j = lane + b * d.Tg;
#pragma unroll
        for (int r = 0; r < 4; ++r) z[b][r] = buf[j + r * (d.M / 4)];
        const TwEnt<float> e = tab[j];
        bf4_fma<INV>(z[b], e);
    }
}

// K1: inverse y-transform of one column (see yinv_body).
template <int E>
__device__ __forceinline__ void f32_yinv_body(const Dims& d, const float2* __restrict__ S,
                                              const double* __restrict__ rk2, const FieldSet& fs,
                                              const float2* __restrict__ tw, int G, int blk, float2* bufs) {
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
    const float* tabf;
    switch (f) {   // select without dynamic indexing of the parameter struct
        case 0: op = fs.op[0]; outp = fs.out[0]; tab = fs.tab[0]; tabf = fs.tabf[0]; break;
        case 1: op = fs.op[1]; outp = fs.out[1]; tab = fs.tab[1]; tabf = fs.tabf[1]; break;
        case 2: op = fs.op[2]; outp = fs.out[2]; tab = fs.tab[2]; tabf = fs.tabf[2]; break;
        default: op = fs.op[3]; outp = fs.out[3]; tab = fs.tab[3]; tabf = fs.tabf[3]; break;
    }
    const bool tfac = op == OP_TU || op == OP_TV;
    if (tfac) rk2 = tab;   // the factor table takes the 1/k^2 table's place
    const bool f32tab = tfac && tabf != nullptr;   // the factors pre-rounded: the same values
    float2* buf = bufs + (size_t)g * M;
    const size_t c0 = (size_t)(active ? kx : 0) * d.ldS;
    const float2* col = S + c0;
    const double* rcol = rk2 + c0;
    const float* fcol = f32tab ? tabf + c0 : nullptr;
    auto value = [&](int jc, int ky, float2 w) {
        if (f32tab) {   // i f w, as scale_by forms it from the FP64 factor
            const float fv = fcol[jc];
            return make_float2(-fv * w.y, fv * w.x);
        }
        return apply_op(op, w, kx, ky, rcol[jc]);
    };
    // radix 3 on (x[j], x[j + K], x[j + 2K]): row j (ky = j), 0 (ky = K for
    // j = 0), and row j + K + 1 (ky = j - K)
    const float2 zero = make_float2(0.f, 0.f);
    float2 x0[NB], x2[NB], xm = zero;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * T;
        x0[b] = x2[b] = zero;
        if (active && fx_on<E, 3>(j, M)) {
            x0[b] = __ldcg(&col[j]);
            x2[b] = __ldcg(&col[j + K + 1]);
        }
    }
    if (active && lane == 0) xm = value(K, K, __ldcg(&col[K]));
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * T;
        if (!fx_on<E, 3>(j, M)) continue;
        float2 v[3] = {zero, xm, zero};
        if (active) {
            v[0] = value(j, j, x0[b]);
            v[2] = value(j + K + 1, j - K, x2[b]);
        }
        if (b == 0 && lane == 0) bf3<true>(v);
        else bf3_bzero<true>(v);
#pragma unroll
        for (int r = 0; r < 3; ++r) buf[3 * j + r] = v[r];
    }
    __syncthreads();
    f32_passes<E, true>(buf, d, lane, tw, 1, d.npass - 1);
    float2 z[kFxNB<E, 4>][4];
    f32_last4<E, true>(buf, d, lane, tw, z);
    float2* out = reinterpret_cast<float2*>(outp) + kx;
    if (active) {
#pragma unroll
        for (int b = 0; b < kFxNB<E, 4>; ++b)
#pragma unroll
            for (int r = 0; r < 4; ++r) out[(size_t)(lane + b * T + r * (M / 4)) * d.ldI] = z[b][r];
    }
}

// The inverse x-transform of u + i v of one row: z[b][r] = element
// lane + b T + r M / 4.  A thread's radix-3 butterflies of the first pass come
// in pairs (q, K - q), whose inputs z(k), z(M - k) belong to the same two
// entries of the half spectra; q = 0 pairs 0 with K / 2 and takes z(K) besides.
template <int E>
__device__ __forceinline__ void f32_row_inverse(const Dims& d, const float2* urow, const float2* vrow, bool active,
                                                const float2* __restrict__ tw, int lane, float2* buf,
                                                float2 (*z)[4]) {
    constexpr int NP = E == 12 ? 2 : 1;   // pairs per thread: K / 2 over T = 3 K / E
    const int K = d.K, T = d.Tg;
    const float2 zero = make_float2(0.f, 0.f);
    float2 ua[NP], va[NP], ub[NP], vb[NP], um = zero, vm = zero;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int q = lane + p * T;
        ua[p] = va[p] = ub[p] = vb[p] = zero;
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
    }
    auto zp = [](float2 a, float2 b) { return make_float2(a.x - b.y, a.y + b.x); };    // z(k)
    auto zm = [](float2 a, float2 b) { return make_float2(a.x + b.y, b.x - a.y); };    // z(M - k)
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int q = lane + p * T;
        if (E != 12 && q >= K / 2) continue;
        const int q2 = q ? K - q : K / 2;
        const bool first = p == 0 && lane == 0;
        float2 v[3], w[3];
        v[1] = w[1] = zero;
        v[0] = first ? make_float2(ua[0].x, va[0].x) : zp(ua[p], va[p]);   // kx = 0: real parts only
        w[0] = zp(ub[p], vb[p]);
        v[2] = first ? zm(um, vm) : zm(ub[p], vb[p]);
        w[2] = first ? zm(ub[p], vb[p]) : zm(ua[p], va[p]);
        if (first) {
            v[1] = zp(um, vm);
            bf3<true>(v);
        } else {
            bf3_bzero<true>(v);
        }
        bf3_bzero<true>(w);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            buf[3 * q + r] = v[r];
            buf[3 * q2 + r] = w[r];
        }
    }
    __syncthreads();
    f32_passes<E, true>(buf, d, lane, tw, 1, d.npass - 1);
    f32_last4<E, true>(buf, d, lane, tw, z);
}

// The forward x-transform of a row held as z (destroyed); put(k, P(k),
// P(M - k)) for k in [0, K] (P(M) = P(0)).
template <int E, typename Put>
__device__ __forceinline__ void f32_row_forward(const Dims& d, float2 (*z)[4], const float2* __restrict__ tw, int lane,
                                                float2* buf, Put put) {
    const int M = d.M, K = d.K, T = d.Tg;
    __syncthreads();   // every thread is done with the buffer
#pragma unroll
    for (int b = 0; b < kFxNB<E, 4>; ++b)
#pragma unroll
        for (int r = 0; r < 4; ++r) buf[lane + b * T + r * (M / 4)] = z[b][r];
    __syncthreads();
    f32_passes<E, false>(buf, d, lane, tw, 0, d.npass - 1);
    f32_last4<E, false>(buf, d, lane, tw, z);
    __syncthreads();
#pragma unroll
    for (int b = 0; b < kFxNB<E, 4>; ++b)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int n = lane + b * T + r * (M / 4);
            if (n <= K || n >= M - K) buf[n] = z[b][r];
        }
    __syncthreads();
    for (int k = lane; k <= K; k += T) put(k, buf[k], buf[k == 0 ? 0 : M - k]);
}

// K2, Basdevant form, of one row (see xpass_bas_body).
template <int E>
__device__ __forceinline__ void f32_xpass_body(const Dims& d, float2* Iu, float2* Iv, const float2* __restrict__ tw,
                                               int G, float scale, int blk, float2* bufs) {
    const int g = threadIdx.x / d.Tg;
    const int lane = threadIdx.x - g * d.Tg;
    const int y = blk * G + g;
    const bool active = y < d.rows && g < G;
    float2* buf = bufs + (size_t)g * d.M;
    float2* urow = Iu + (size_t)(active ? y : 0) * d.ldI;
    float2* vrow = Iv + (size_t)(active ? y : 0) * d.ldI;
    float2 z[kFxNB<E, 4>][4];
    f32_row_inverse<E>(d, urow, vrow, active, tw, lane, buf, z);
#pragma unroll
    for (int b = 0; b < kFxNB<E, 4>; ++b)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float2 a = z[b][r];
            z[b][r] = make_float2(a.x * a.y, a.y * a.y - a.x * a.x);
        }
    f32_row_forward<E>(d, z, tw, lane, buf, [&](int k, float2 p, float2 q) {
        if (!active) return;
        if (scale == 1.f) {   // products of prescaled u, v: no multiply
            urow[k] = make_float2(p.x + q.x, p.y - q.y);
            vrow[k] = make_float2(p.y + q.y, q.x - p.x);
        } else {
            urow[k] = make_float2((p.x + q.x) * scale, (p.y - q.y) * scale);
            vrow[k] = make_float2((p.y + q.y) * scale, (q.x - p.x) * scale);
        }
    });
}

// K3's transform: column kx of one product, read from the half-spectral rows;
// sink(jc, value) gets the retained rows.  SYNC: a barrier between the last
// pass's loads and the sinks (which write to buf).
template <int E, bool SYNC, typename Sink>
__device__ __forceinline__ void f32_yfwd_column(const Dims& d, const float2* __restrict__ I, bool active, int kx,
                                                const float2* __restrict__ tw, int lane, float2* buf, Sink sink) {
    constexpr int NB = kFxNB<E, 3>;
    const int M = d.M, K = d.K, T = d.Tg;
    float2 x[NB][3];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * T;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            x[b][r] = make_float2(0.f, 0.f);
            if (active && fx_on<E, 3>(j, M)) x[b][r] = __ldcg(&I[(size_t)(j + r * K) * d.ldI + kx]);
        }
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = lane + b * T;
        if (!fx_on<E, 3>(j, M)) continue;
        bf3<false>(x[b]);
#pragma unroll
        for (int r = 0; r < 3; ++r) buf[3 * j + r] = x[b][r];
    }
    __syncthreads();
    f32_passes<E, false>(buf, d, lane, tw, 1, d.npass - 1);
    float2 z[kFxNB<E, 4>][4];
    f32_last4<E, false>(buf, d, lane, tw, z);
    if (SYNC) __syncthreads();
#pragma unroll
    for (int b = 0; b < kFxNB<E, 4>; ++b)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int n = lane + b * T + r * (M / 4);
            if (n <= K) sink(n, z[b][r]);
            else if (n >= M - K) sink(n - M + d.KY, z[b][r]);
        }
}

// K3 in one kernel (see yfwd_body): 2G transforms, blockDim / T at a time,
// their retained rows left in shared memory, then the epilogue.
template <int E>
__device__ __forceinline__ bool f32_yfwd_body(const Dims& d, const float2* __restrict__ Iu,
                                              const float2* __restrict__ Iv, float2* S0, float2* S1, float2* Sdw,
                                              const float2* __restrict__ src, int stage, double dt, const Phys& ph,
                                              const float2* __restrict__ tw, int G, int blk, float2* bufs) {
    const int t = threadIdx.x / d.Tg;
    const int lane = threadIdx.x - t * d.Tg;
    const int kx0 = blk * G;
    const int gtot = min(G, d.KX - kx0);
    const int nconc = blockDim.x / d.Tg;
    for (int t0 = 0; t0 < 2 * G; t0 += nconc) {
        const int i = t0 + t, f = i >= G, gg = i - f * G;   // buffer i: field f, column gg
        float2* buf = bufs + (size_t)i * d.M;
        f32_yfwd_column<E, true>(d, f ? Iv : Iu, gg < gtot, kx0 + gg, tw, lane, buf,
                                 [&](int jc, float2 v) { buf[jc] = v; });
    }
    __syncthreads();
    bool bad = false;
    const DivBy byKY(d.KY);
    for (int idx = threadIdx.x; idx < gtot * d.KY; idx += blockDim.x) {
        const int gg = gtot == 1 ? 0 : byKY(idx);
        const int jc = idx - gg * d.KY;
        bad |= stage_point<float>(d, bufs[(size_t)gg * d.M + jc], bufs[(size_t)(G + gg) * d.M + jc], kx0 + gg, jc, S0,
                                  S1, Sdw, src, stage, dt, ph);
    }
    return bad;
}

}  // namespace s2d
