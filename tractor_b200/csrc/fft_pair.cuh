// Two N-point FFTs at once (N = 32 .. 256) by a group of N/16 threads, each
// holding 16 complex values of both in packed FP32 (f32x2.cuh): a radix-16
// pass, one shared-memory exchange, a radix-N/16 pass (Stockham).
//
// Pass 1: thread t holds x[t + G m], G = N/16, m = 0..15, and computes the
// 16-point DFT y[16 t + q] = sum_m x[t + G m] W_16^{s m q}.
// Pass 2: for j = t + G g, g = 0 .. 16/G - 1, the G values y[j + 16 m] take
// the twiddles W_N^{s m j} and give X[j + 16 q] = sum_m y'[j + 16 m] W_G^{s m q}.
// W_M = exp(2 pi i / M), s = +1 (inverse, unnormalised) or -1.
//
// Every instruction works on both transforms, so a transform costs half the
// instructions of one held alone (the renderer is bound by instruction issue
// and fetch).  Real and imaginary parts are exchanged one after the other
// through a buffer of N + G elements of 8 bytes per group (one pad element per
// 16: every half warp's accesses fall into different banks, for each N), so
// that 16 warps' buffers leave room for a whole transpose.
#pragma once
#include "f32x2.cuh"

namespace tb {

// The same element of the two transforms.
struct C2 {
    f32x2 re, im;
};

__device__ __forceinline__ C2 add(C2 a, C2 b) { return C2{add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ C2 sub(C2 a, C2 b) { return C2{sub2(a.re, b.re), sub2(a.im, b.im)}; }
// A factor wr + i wi for both transforms: wr and wi twice each.  Tables of
// them hold (wr, wr, wi, wi).
struct Factor {
    f32x2 re, im;
};
__device__ __forceinline__ Factor factor(const float4* table, int i) {
    const ulonglong2 f = reinterpret_cast<const ulonglong2*>(table)[i];
    return Factor{f.x, f.y};
}
__device__ __forceinline__ C2 cmul2(C2 a, Factor w) {
    return C2{sub2(mul2(a.re, w.re), mul2(a.im, w.im)), fma2(a.re, w.im, mul2(a.im, w.re))};
}
__device__ __forceinline__ C2 cmulc(C2 a, Factor w) {   // by the conjugate
    return C2{fma2(a.im, w.im, mul2(a.re, w.re)), sub2(mul2(a.im, w.re), mul2(a.re, w.im))};
}
template <int S> __device__ __forceinline__ C2 cmul_const(C2 a, float wr, float wi) {
    const f32x2 r = both(wr), i = both(S * wi), n = both(-S * wi);
    return C2{fma2(a.im, n, mul2(a.re, r)), fma2(a.im, r, mul2(a.re, i))};
}
// a + s i b and a - s i b
template <int S> __device__ __forceinline__ C2 add_si(C2 a, C2 b) {
    return S > 0 ? C2{sub2(a.re, b.im), add2(a.im, b.re)} : C2{add2(a.re, b.im), sub2(a.im, b.re)};
}
template <int S> __device__ __forceinline__ C2 sub_si(C2 a, C2 b) { return add_si<-S>(a, b); }

template <int S> __device__ __forceinline__ void dft4(C2& a0, C2& a1, C2& a2, C2& a3) {
    const C2 s02 = add(a0, a2), d02 = sub(a0, a2), s13 = add(a1, a3), d13 = sub(a1, a3);
    a0 = add(s02, s13);
    a2 = sub(s02, s13);
    a1 = add_si<S>(d02, d13);
    a3 = sub_si<S>(d02, d13);
}

// In place, natural order: DFTs of length 4 over the stride-4 subsequences,
// the twiddles W_16^{s n2 k1}, DFTs of length 4 across them.
template <int S> __device__ __forceinline__ void dft16(C2 (&a)[16]) {
    constexpr float C1 = 0.92387953251128674f, S1 = 0.38268343236508978f;
    constexpr float R = 0.70710678118654752f;
#pragma unroll
    for (int n = 0; n < 4; n++) dft4<S>(a[n], a[4 + n], a[8 + n], a[12 + n]);
    // a[4 k1 + n2]: W_16^{n2 k1}
    a[5] = cmul_const<S>(a[5], C1, S1);
    a[9] = cmul_const<S>(a[9], R, R);
    a[13] = cmul_const<S>(a[13], S1, C1);
    a[6] = cmul_const<S>(a[6], R, R);
    {
        const C2 v = a[10];   // s i v
        const f32x2 zero = 0ull;
        a[10] = S > 0 ? C2{sub2(zero, v.im), v.re} : C2{v.im, sub2(zero, v.re)};
    }
    a[14] = cmul_const<S>(a[14], -R, R);
    a[7] = cmul_const<S>(a[7], S1, C1);
    a[11] = cmul_const<S>(a[11], -R, R);
    a[15] = cmul_const<S>(a[15], -C1, -S1);
    C2 b[16];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        dft4<S>(a[4 * k], a[4 * k + 1], a[4 * k + 2], a[4 * k + 3]);
#pragma unroll
        for (int q = 0; q < 4; q++) b[k + 4 * q] = a[4 * k + q];
    }
#pragma unroll
    for (int m = 0; m < 16; m++) a[m] = b[m];
}

template <int S> __device__ __forceinline__ void dft8(C2* a) {
    C2 e0 = a[0], e1 = a[2], e2 = a[4], e3 = a[6], o0 = a[1], o1 = a[3], o2 = a[5], o3 = a[7];
    dft4<S>(e0, e1, e2, e3);
    dft4<S>(o0, o1, o2, o3);
    const f32x2 r = both(0.70710678118654752f);
    const C2 p1 = add_si<S>(o1, o1), p3 = sub_si<S>(o3, o3);   // o (1 + s i), o (1 - s i)
    o1 = C2{mul2(p1.re, r), mul2(p1.im, r)};
    o3 = C2{mul2(p3.re, r), mul2(p3.im, r)};                   // -(W_8^3 o3)
    a[0] = add(e0, o0);
    a[4] = sub(e0, o0);
    a[1] = add(e1, o1);
    a[5] = sub(e1, o1);
    a[2] = add_si<S>(e2, o2);
    a[6] = sub_si<S>(e2, o2);
    a[3] = sub(e3, o3);
    a[7] = add(e3, o3);
}

// 8-byte elements of a group's exchange buffer.
template <int N> __host__ __device__ constexpr int pair_xbuf() { return N + N / 16; }
__device__ __forceinline__ int pair_pad(int i) { return i + (i >> 4); }

// Pass-2 twiddles: entry 16 m + j = exp(2 pi i m j / N), m < N/16, j < 16.  By
// `count` threads numbered `tid`.
template <int N> __device__ void build_pair_twiddles(float4* tw, int tid, int count) {
    for (int e = tid; e < N; e += count) {
        double s, c;
        sincospi(2.0 * (double)((e >> 4) * (e & 15)) / N, &s, &c);
        tw[e] = make_float4((float)c, (float)c, (float)s, (float)s);
    }
}

// Runs both transforms on the G = N/16 threads t of a group.  `v[m]` =
// x[t + G m] on entry; `store(g, q, value)` receives the outputs X[t + G g +
// 16 q] (16 calls per thread, g and q known when compiling).  Whole warps.
template <int N, int S, class Store>
__device__ __forceinline__ void fft_pair(C2 (&v)[16], int t, f32x2* xb, const float4* tw,
                                         Store store) {
    constexpr int G = N / 16;
    dft16<S>(v);
#pragma unroll
    for (int q = 0; q < 16; q++) xb[pair_pad(16 * t + q)] = v[q].re;
    __syncwarp();
    // v[g G + m] = y[t + G g + 16 m]
#pragma unroll
    for (int i = 0; i < 16; i++) v[i].re = xb[pair_pad(t + G * (i / G) + 16 * (i % G))];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 16; q++) xb[pair_pad(16 * t + q)] = v[q].im;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; i++) v[i].im = xb[pair_pad(t + G * (i / G) + 16 * (i % G))];
    __syncwarp();
#pragma unroll
    for (int g = 0; g < 16 / G; g++) {
#pragma unroll
        for (int m = 1; m < G; m++) {
            const Factor w = factor(tw, 16 * m + t + G * g);
            C2& x = v[g * G + m];
            x = S > 0 ? cmul2(x, w) : cmulc(x, w);
        }
        if constexpr (G == 16) {
            dft16<S>(v);
        } else if constexpr (G == 8) {
            dft8<S>(v + 8 * g);
        } else if constexpr (G == 4) {
            dft4<S>(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
        } else {
            const C2 a = v[2 * g], b = v[2 * g + 1];
            v[2 * g] = add(a, b);
            v[2 * g + 1] = sub(a, b);
        }
#pragma unroll
        for (int q = 0; q < G; q++) store(g, q, v[g * G + q]);
    }
}

}  // namespace tb
