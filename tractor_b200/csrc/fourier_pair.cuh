// The pixelized-PSF renderer's main path (included by fourier_render.cu, whose
// helpers it uses): value items whose Lanczos-3 shift is a spectral product
// (the output window keeps 3 px from the FFT box's edges, or there is no
// shift), on packed transforms of two columns or two row pairs at a time.
//
// A CTA of 16 warps works in groups, one item per group: at FFT size 256 the
// whole CTA renders one galaxy, at 128 two groups of 8 warps one each, at 64
// seven of 2 warps (shared memory), at 32 sixteen of one warp, every group in
// its own part of shared memory with its own named barrier.  The sizes run one after another (largest first, the
// small ones fill the end), each from a list of items and a counter.
//
// An item of size N, sz/2 + 1 = N/2 + 1 columns:
//   1. column pass: N/4 jobs of two adjacent columns.  The
//      mixture spectrum of 16 rows per thread (spectrum_pair), times the PSF
//      spectrum and the y taps' response, an inverse transform along y; the
//      kept rows go to S1.  Columns 0 and N/2 share a transform (their
//      Hermitian parts are real after it, which is what irfftn keeps).
//   2. row pass: jobs of four rows: two complex transforms along x of two
//      real rows each, times the x taps' response, straight to the output.
// S1 holds rows r and r + 2 side by side: S1[(pair N/2+1 + v) 4 + slot], pair =
// 2 (r / 4) + r % 2, slot = (r / 2) % 2 (+ 2: imaginary part), so that a row
// job reads one float4 per element of a pair of rows.
//
// Bound: instruction issue and fetch.  One 221 KB CTA of 16 warps per galaxy
// with one transform per half warp (fourier_render_kernel) spends 58 K cycles
// on a galaxy of size 256 and a 128 x 128 window, mostly waiting for
// instructions; packing halves the transforms' instructions.
// Measured, with the preparation: 256 galaxies of size 256 on 128 x 128 patches
// 87 us fused, 78 us fourier_render_kernel, 74 us here; 2,000 on ragged 25-253
// px patches 568, 516, 346; 2,000 on 100 x 100 (size 128) 252, 225, 146.  A
// galaxy of size 256 takes 49 K cycles (columns 33 K, rows 11 K, the rest its
// preparation, which nothing overlaps), at 1.7 instructions per cycle: held by
// fixed latencies at 16 warps (128 registers) and the phases' barriers.

constexpr int kPairThreads = 512;
constexpr int kPairMaxK = 32;       // components of an item on this path
constexpr int kPairRows256 = 132;   // rows of S1 at N = 256 (windows of 128 and a few more)

// Exponents (log2 units, relative to the component) below this are dropped
// from a spectrum: 2^-44 of a component's flux is far below FP32's rounding of
// the sum over frequencies.
constexpr float kSpecFloor = -44.f;
template <int N>
struct PairPlan {
    static constexpr int kThreads = N >= 128 ? 2 * N : N;     // of a group
    static constexpr int kLanes = kThreads / (N / 16);        // transforms (pairs) at once
    static constexpr int kGroups = N == 64 ? 7 : kPairThreads / kThreads;
    static constexpr int kRows = N == 256 ? kPairRows256 : N; // rows of S1
    static constexpr int NH = N / 2 + 1;
    static constexpr int kXbuf = kLanes * tb::pair_xbuf<N>() * 8;
    static constexpr int kS1 = kRows * NH * 8;
    static constexpr int kBytes = kXbuf + kS1 + (NH + 2 * N) * 16 /* hx, hy, tw */ +
                                  4 * N * 4 /* gsp, edge */ + 2 * kPairMaxK * 16 /* comp, aux */ +
                                  16 * 4 /* taps */ + 16 /* slot */;
    static_assert(kRows % 4 == 0 && kBytes % 16 == 0, "layout");
};
constexpr int kPairSmem = PairPlan<256>::kBytes > 2 * PairPlan<128>::kBytes
                              ? PairPlan<256>::kBytes : 2 * PairPlan<128>::kBytes;
static_assert(kPairSmem <= 232448 && PairPlan<64>::kGroups * PairPlan<64>::kBytes <= kPairSmem &&
              PairPlan<32>::kGroups * PairPlan<32>::kBytes <= kPairSmem, "shared memory of an SM");

// Work lists of one call, by FFT size (index 0: 256, 1: 128, 2: 64, 3: 32) and
// the items left to fourier_render_kernel (4).
struct PairWs {
    int32_t count[5];
    int32_t next[5];
    int32_t pad[54];
};

struct PairGroup {
    tb::f32x2* xbuf;
    float* s1;
    float4 *hx, *hy, *tw;   // tap responses and twiddles (tb::factor)
    float* gsp;         // mixture spectrum of columns 0 and N/2
    float2* edge;       // their common transform input
    float4* comp;       // (amp, ca, cb, cd): exponent ca v^2 + cb v w + cd w^2 (log2 units)
    float4* aux;        // (g, slope, -1/cd, -): see stage_aux
    float* taps;
    int* slot;
    int tid, bar;
    template <int N>
    __device__ __forceinline__ void sync() const {
        if constexpr (PairPlan<N>::kThreads == 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(PairPlan<N>::kThreads) : "memory");
    }
};

// What a column needs to know of a component: g = ca - cb^2 / (4 cd) (its
// largest exponent over w is g v^2, at w = slope v) and -1/cd.
__device__ __forceinline__ float4 stage_aux(float4 c) {
    const bool flat = c.w > -1e-20f;   // a point-like core: constant
    return make_float4(flat ? 0.f : c.y - c.z * c.z / (4.f * c.w),
                       flat ? 0.f : -c.z / (2.f * c.w), flat ? 1e30f : -1.f / c.w, 0.f);
}

// Mixture spectrum of the columns va and vb = va + 1/N at the rows w = w0 +
// q/16, q = 0..15 (this thread's, in increasing order of signed frequency):
// acc[q].  Components that stay below kSpecFloor in the column are left out,
// and of the others the runs of four rows that they do not reach; `span` is
// the largest t/N of the threads of a column, so that a column's threads
// agree.  (Carrying a run's exponentials from its first row, four ex2 for
// eight values, was no faster here and raised the patches' error against 64
// bits from 1.7e-7 to 2.0e-7.)
__device__ __forceinline__ void spectrum_pair(const float4* comp, const float4* aux, int K,
                                              float va, float vb, float w0, float first,
                                              float span, tb::f32x2 (&acc)[16]) {
    using namespace tb;
#pragma unroll
    for (int q = 0; q < 16; q++) acc[q] = 0ull;
    const f32x2 v2 = pack(va, vb), vv = mul2(v2, v2);
    for (int k = 0; k < K; k++) {
        const float4 a = aux[k];
        const float top = a.x * va * va;
        if (top < kSpecFloor) continue;
        const float4 c = comp[k];
        const f32x2 amp = both(c.x), al = mul2(vv, both(c.y)), be = mul2(v2, both(c.z));
        const f32x2 cd = both(c.w);
        const float h2 = (top - kSpecFloor) * a.z + 1e-30f, half = h2 * rsqrtf(h2);
        const float lo = fminf(a.y * va, a.y * vb) - half - span - 3.f / 16.f;
        const float hi = fmaxf(a.y * va, a.y * vb) + half;
#pragma unroll
        for (int g = 0; g < 4; g++) {
            const float wf = first + 0.25f * g;      // the run's lowest row of any thread
            if (wf < lo || wf > hi) continue;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const f32x2 w = both(w0 + (float)(4 * g + i) / 16.f);
                const float2 e = unpack(fma2(w, fma2(cd, w, be), al));
                acc[4 * g + i] = fma2(amp, pack(ex2(e.x), ex2(e.y)), acc[4 * g + i]);
            }
        }
    }
}

// Mixture spectrum of columns 0 and N/2, every row, into gsp (read by the job
// of columns 0 and 1).
template <int N>
__device__ __forceinline__ void spectrum_edges(const PairGroup& sh, int K) {
    for (int e = sh.tid; e < 2 * N; e += PairPlan<N>::kThreads) {
        const int j = e & (N - 1);
        const float w = (float)(j < N / 2 ? j : j - N) / (float)N;
        float g;
        spectrum_rows<1>(sh.comp, K, e < N ? 0.f : 0.5f, &w, &g);
        sh.gsp[e] = g;
    }
}

// The transform input of columns 0 and N/2 together at every row, into
// `edge`: Xh(w) = (X(w) + conj X(-w)) / 2 of each, the second times i.
template <int N>
__device__ __forceinline__ void edge_columns(const PairGroup& sh, const float* __restrict__ spec) {
    const float2* P = reinterpret_cast<const float2*>(spec);
    const float2* Pn = P + (int64_t)(N / 2) * N;
    for (int j = sh.tid; j < N; j += PairPlan<N>::kThreads) {
        const int jn = (N - j) & (N - 1);
        const float4 hj = sh.hy[j], hn = sh.hy[jn];
        const float2 h = make_float2(hj.x, hj.z), hm = make_float2(hn.x, hn.z);
        const float2 a = cmulf(__ldg(P + j), h), b = cmulf(__ldg(P + jn), hm);
        const float2 an = cmulf(__ldg(Pn + j), h), bn = cmulf(__ldg(Pn + jn), hm);
        const float g0 = sh.gsp[j], g0n = sh.gsp[jn], gN = sh.gsp[N + j], gNn = sh.gsp[N + jn];
        const float2 x0 = make_float2(0.5f * (g0 * a.x + g0n * b.x), 0.5f * (g0 * a.y - g0n * b.y));
        const float2 xN = make_float2(0.5f * (gN * an.x + gNn * bn.x),
                                      0.5f * (gN * an.y - gNn * bn.y));
        sh.edge[j] = make_float2(x0.x - xN.y, x0.y + xN.x);
    }
}

__device__ __forceinline__ int s1_index(int r, int NH, int v) {
    return ((2 * (r >> 2) + (r & 1)) * NH + v) * 4 + ((r >> 1) & 1);
}

// Column pass: rows [rlo, rlo + nrows) of every column into S1.
template <int N>
__device__ __forceinline__ void pair_columns(const PairGroup& sh, int K,
                                             const float* __restrict__ spec, int rlo, int nrows) {
    using namespace tb;
    constexpr int G = N / 16, NH = PairPlan<N>::NH;
    const int t = sh.tid % G, grp = sh.tid / G;
    f32x2* xb = sh.xbuf + grp * pair_xbuf<N>();
    const float2* P = reinterpret_cast<const float2*>(spec) + t;
    const float w0 = (float)t / (float)N - 0.5f;
    for (int j0 = 0; j0 < N / 4; j0 += PairPlan<N>::kLanes) {
        const bool act = j0 + grp < N / 4;
        const int va = 2 * (act ? j0 + grp : N / 4 - 1);
        C2 x[16];
        {
            f32x2 acc[16];
            spectrum_pair(sh.comp, sh.aux, K, (float)va / N, (float)(va + 1) / N, w0, -0.5f,
                          (float)(G - 1) / N, acc);
            const float2* Pa = P + va * N;
#pragma unroll
            for (int m = 0; m < 16; m++) {
                const float2 pa = __ldg(Pa + G * m), pb = __ldg(Pa + N + G * m);
                const f32x2 a = acc[(m + 8) & 15];   // row t + G m
                x[m] = cmul2(C2{mul2(a, pack(pa.x, pb.x)), mul2(a, pack(pa.y, pb.y))},
                             factor(sh.hy, t + G * m));
            }
            if (j0 == 0) {   // columns 0 and N/2 in place of column 0
#pragma unroll
                for (int m = 0; m < 16; m++) {
                    const float2 e = sh.edge[t + G * m];
                    const float2 re = unpack(x[m].re), im = unpack(x[m].im);
                    x[m] = C2{pack(va == 0 ? e.x : re.x, re.y), pack(va == 0 ? e.y : im.x, im.y)};
                }
            }
        }
        // the first column's imaginary part, or column N/2's real one (the
        // imaginary parts of those two columns are zero: pair_item)
        const int other = va == 0 ? 4 * (N / 2) : 2;
        fft_pair<N, +1>(x, t, xb, sh.tw, [&](int g, int q, C2 z) {
            const int r0 = t + G * g - rlo, r = r0 + 16 * q;
            if (!act || (unsigned)r >= (unsigned)nrows) return;
            // 16 rows on: 8 pairs of rows
            float* s = sh.s1 + s1_index(r0 & 15, NH, va) + ((r0 >> 4) + q) * (32 * NH);
            const float2 re = unpack(z.re), im = unpack(z.im);
            s[0] = re.x;
            s[other] = im.x;
            s[4] = re.y;
            s[6] = im.y;
        });
        __syncwarp();
    }
}

// Row pass: the rows of S1 to output rows row0 .., columns [c0, c1) of the box.
template <int N>
__device__ __forceinline__ void pair_rows(const tb_fft_item& it, const PairGroup& sh, int nrows,
                                          float* O, int64_t ldo, int row0, int c0, int c1,
                                          float osc) {
    using namespace tb;
    constexpr int G = N / 16, NH = PairPlan<N>::NH;
    const int t = sh.tid % G, grp = sh.tid / G;
    f32x2* xb = sh.xbuf + grp * pair_xbuf<N>();
    const int nq = (nrows + 3) / 4;
    const int mode = it.mode;
    const f32x2 scale = both(osc);
    for (int i0 = 0; i0 < nq; i0 += PairPlan<N>::kLanes) {
        const bool act = i0 + grp < nq;
        const int i = act ? i0 + grp : nq - 1;
        const ulonglong2* H1 = reinterpret_cast<const ulonglong2*>(sh.s1) + 2 * i * NH;   // rows 4 i, 4 i + 2
        const ulonglong2* H2 = H1 + NH;                                                   // 4 i + 1, 4 i + 3
        C2 x[16];
#pragma unroll
        for (int m = 0; m < 16; m++) {
            // element n = t + G m: column n, or (n > N/2) the conjugate of N - n
            const int q = m < 8 ? t + G * m : G * (16 - m) - t;
            const ulonglong2 f1 = H1[q], f2 = H2[q];
            const Factor h = factor(sh.hx, q);
            C2 h1 = cmul2(C2{f1.x, f1.y}, h), h2 = cmul2(C2{f2.x, f2.y}, h);
            // columns 0 and N/2 are real
            if ((m == 0 || m == 8) && t == 0) h1.im = h2.im = 0ull;
            x[m] = m < 8 ? C2{sub2(h1.re, h2.im), add2(h1.im, h2.re)}
                         : C2{add2(h1.re, h2.im), sub2(h2.re, h1.im)};
        }
        const int last = act ? nrows - 4 * i : 0;
        float* p0 = O + (int64_t)(row0 + 4 * i) * ldo + t;
        float *p1 = p0 + ldo, *p2 = p1 + ldo, *p3 = p2 + ldo;
        const bool plain = mode == TB_MOG_STORE && last >= 4;
        const int lo = c0 - t, hi = c1 - t;
        fft_pair<N, +1>(x, t, xb, sh.tw, [&](int g, int q, C2 z) {
            const int c = G * g + 16 * q;
            if (c < lo || c >= hi) return;
            const float2 re = unpack(mul2(z.re, scale)), im = unpack(mul2(z.im, scale));
            if (plain) {
                p0[c] = re.x;
                p1[c] = im.x;
                p2[c] = re.y;
                p3[c] = im.y;
            } else {
                float dummy = 0.f;
                if (last > 0) put<false>(p0 + c, re.x, mode, dummy);
                if (last > 1) put<false>(p1 + c, im.x, mode, dummy);
                if (last > 2) put<false>(p2 + c, re.y, mode, dummy);
                if (last > 3) put<false>(p3 + c, im.y, mode, dummy);
            }
        });
        __syncwarp();
    }
}

// Frequency response of seven taps at index fr of an N-point transform: sum_k
// tap_k exp(2 pi i fr (k - 3) / N).
template <int N>
__device__ __forceinline__ float2 tap_response(const float* tap, int fr) {
    float c = tap[3], s = 0.f;
#pragma unroll
    for (int k = 1; k <= 3; k++) {
        float sk, ck;
        sincospif(2.f * (float)((fr * k) & (N - 1)) / (float)N, &sk, &ck);
        c = fmaf(tap[3 + k] + tap[3 - k], ck, c);
        s = fmaf(tap[3 + k] - tap[3 - k], sk, s);
    }
    return make_float2(c, s);
}

// Tap responses of an item, twice each, for the packed products.
template <int N>
__device__ __forceinline__ void pair_responses(const PairGroup& sh) {
    for (int f = sh.tid; f < PairPlan<N>::NH + N; f += PairPlan<N>::kThreads) {
        const bool isx = f < PairPlan<N>::NH;
        const int fr = isx ? f : f - PairPlan<N>::NH;
        const float2 r = tap_response<N>(isx ? sh.taps : sh.taps + 8, fr);
        (isx ? sh.hx : sh.hy)[fr] = make_float4(r.x, r.x, r.y, r.y);
    }
}

template <int N>
__device__ void pair_item(const tb_fft_item& it, const PairGroup& sh,
                          const double* __restrict__ amp, const double* __restrict__ var,
                          const float* __restrict__ psf_spec, float* __restrict__ out) {
    constexpr int kThreads = PairPlan<N>::kThreads, NH = PairPlan<N>::NH;
    const int mw = it.mw, mh = it.mh, sx = it.sx, sy = it.sy, K = it.K;
    float* O = out + it.out_off;
    const int64_t ldo = it.ldo > 0 ? it.ldo : mw;
    const int gr0 = max(0, -sy), gr1 = min(N, mh - sy);
    const int gc0 = max(0, -sx), gc1 = min(N, mw - sx);
    const bool empty = gr0 >= gr1 || gc0 >= gc1;
    if (it.mode == TB_MOG_STORE && (empty || gr0 + sy > 0 || gr1 + sy < mh || gc0 + sx > 0 ||
                                    gc1 + sx < mw)) {
        // the mask's pixels outside the transform's window
        for (int i = sh.tid; i < mh * mw; i += kThreads) {
            const int r = i / mw - sy, c = i % mw - sx;
            if (empty || r < gr0 || r >= gr1 || c < gc0 || c >= gc1)
                O[(int64_t)(i / mw) * ldo + i % mw] = 0.f;
        }
    }
    if (empty) return;
    const double c2 = -2.0 * TB_PI * TB_PI * TB_LOG2E;
    for (int k = sh.tid; k < K; k += kThreads) {
        const int c = it.c0 + k;
        const float4 f = make_float4((float)amp[c], (float)(c2 * var[4 * c]),
                                     (float)(c2 * 2.0 * var[4 * c + 1]), (float)(c2 * var[4 * c + 3]));
        sh.comp[k] = f;
        sh.aux[k] = stage_aux(f);
    }
    // the taps by the group's first and last warps
    if (sh.tid < 32) taps_warp(it.mux, false, sh.taps);
    if (sh.tid >= kThreads - 32) taps_warp(it.muy, false, sh.taps + 8);
    sh.template sync<N>();
    pair_responses<N>(sh);
    spectrum_edges<N>(sh, K);
    sh.template sync<N>();
    const float* spec = psf_spec + it.spec_off;
    edge_columns<N>(sh, spec);
    const float osc = it.scale / (float)(N * N);
    for (int a = gr0; a < gr1; a += PairPlan<N>::kRows) {
        const int nrows = min(PairPlan<N>::kRows, gr1 - a);
        // columns 0 and N/2 are real; rows that complete the last four are zero
        for (int r = sh.tid; r < nrows; r += kThreads) {
            float* s = sh.s1 + s1_index(r, NH, 0);
            s[2] = s[4 * (N / 2) + 2] = 0.f;
        }
        for (int e = sh.tid; e < ((4 - nrows % 4) % 4) * NH; e += kThreads) {
            float* s = sh.s1 + s1_index(nrows + e / NH, NH, e % NH);
            s[0] = s[2] = 0.f;
        }
        if (a == gr0) sh.template sync<N>();   // `edge` is complete
        pair_columns<N>(sh, K, spec, a, nrows);
        sh.template sync<N>();
        pair_rows<N>(it, sh, nrows, O + sx, ldo, a + sy, gc0, gc1, osc);
        sh.template sync<N>();
    }
}

// The groups of a CTA that take items from a list of `count`.  A list that is all
// of the call is spread over the CTAs: with fewer items than groups, those of the
// first CTAs would take them all and share an SM while others idle (the gradient of
// 8 galaxies of 40 px 62 -> 57 us, of 256 72 -> 60; 256 renders 38 -> 33).  Beside
// other lists, whose items keep CTAs busy for longer, the rest must make do with
// the CTAs that are free, and every group takes items.
__device__ __forceinline__ int active_groups(int groups, int count, int total) {
    return count == total ? min(groups, (count + (int)gridDim.x - 1) / (int)gridDim.x) : groups;
}

// The items of one FFT size, taken from their list by the CTA's groups.
template <int N>
__device__ void pair_size(unsigned char* smem, const tb_fft_item* __restrict__ items,
                          const int32_t* __restrict__ list, int count, int total, int32_t* next,
                          const double* __restrict__ amp, const double* __restrict__ var,
                          const float* __restrict__ psf_spec, float* __restrict__ out) {
    using Plan = PairPlan<N>;
    if (count == 0) return;   // the same in every thread
    const int g = threadIdx.x / Plan::kThreads;
    unsigned char* p = smem + g * Plan::kBytes;
    PairGroup sh;
    sh.tid = threadIdx.x % Plan::kThreads;
    sh.bar = 1 + g;
    auto take = [&](int bytes) {
        unsigned char* q = p;
        p += bytes;
        return q;
    };
    sh.xbuf = reinterpret_cast<tb::f32x2*>(take(Plan::kXbuf));
    sh.s1 = reinterpret_cast<float*>(take(Plan::kS1));
    sh.hx = reinterpret_cast<float4*>(take(Plan::NH * 16));
    sh.hy = reinterpret_cast<float4*>(take(N * 16));
    sh.tw = reinterpret_cast<float4*>(take(N * 16));
    sh.gsp = reinterpret_cast<float*>(take(2 * N * 4));
    sh.edge = reinterpret_cast<float2*>(take(2 * N * 4));
    sh.comp = reinterpret_cast<float4*>(take(kPairMaxK * 16));
    sh.aux = reinterpret_cast<float4*>(take(kPairMaxK * 16));
    sh.taps = reinterpret_cast<float*>(take(16 * 4));
    sh.slot = reinterpret_cast<int*>(take(16));
    __syncthreads();   // the previous size's groups are done with shared memory
    if (g >= active_groups(Plan::kGroups, count, total)) return;
    tb::build_pair_twiddles<N>(sh.tw, sh.tid, Plan::kThreads);
    for (;;) {
        if (sh.tid == 0) *sh.slot = atomicAdd(next, 1);
        sh.template sync<N>();
        const int u = *sh.slot;
        if (u >= count) break;
        pair_item<N>(items[list[u]], sh, amp, var, psf_spec, out);
        sh.template sync<N>();
    }
}

// A list rendered as by fourier_render_kernel, a CTA per item.  A call, not
// inlined: each part of the kernel then has all 128 registers (4 bytes of spills
// in place of 168; a galaxy whose window reaches the box's edge 194 -> 143 us,
// 256 of 128 px 76 -> 74).
template <bool kDeriv>
__device__ __noinline__ void whole_cta_list(const tb_fft_item* __restrict__ items, int n_items,
                                            const double* __restrict__ amp,
                                            const double* __restrict__ var,
                                            const double* __restrict__ dcoef,
                                            const float* __restrict__ psf_spec,
                                            float* __restrict__ out, double* __restrict__ dots,
                                            int32_t* next, tb_status* st,
                                            const int32_t* __restrict__ list, int count,
                                            unsigned char* smem) {
    render_items<kDeriv>(items, n_items, amp, var, dcoef, psf_spec, out, dots, next, st, list,
                         count, smem);
}

// All items of a call: those outside this path first (an item at the box's edge
// takes several times as long as another; kDeriv: position derivatives among
// them), then the lists by size.
template <bool kDeriv>
__global__ void __launch_bounds__(kPairThreads, 1)
fourier_pair_kernel(const tb_fft_item* __restrict__ items, int n_items,
                    const double* __restrict__ amp, const double* __restrict__ var,
                    const float* __restrict__ psf_spec, float* __restrict__ out, PairWs* ws,
                    const int32_t* __restrict__ lists, tb_status* st) {
    static_assert(kPairThreads == kThreads && kPairSmem >= kSmemBytes, "one block shape for both");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int4 c = *reinterpret_cast<const int4*>(ws->count);   // (one load, not one for each list)
    const int rest = ws->count[4], total = c.x + c.y + c.z + c.w + rest;
    if (rest != 0)
        whole_cta_list<kDeriv>(items, n_items, amp, var, nullptr, psf_spec, out, nullptr,
                               &ws->next[4], st, lists + 4 * (int64_t)n_items, rest, smem_raw);
    pair_size<256>(smem_raw, items, lists, c.x, total, &ws->next[0], amp, var, psf_spec, out);
    pair_size<128>(smem_raw, items, lists + n_items, c.y, total, &ws->next[1], amp, var, psf_spec,
                   out);
    pair_size<64>(smem_raw, items, lists + 2 * (int64_t)n_items, c.z, total, &ws->next[2], amp,
                  var, psf_spec, out);
    pair_size<32>(smem_raw, items, lists + 3 * (int64_t)n_items, c.w, total, &ws->next[3], amp,
                  var, psf_spec, out);
}

// The list of an item: by FFT size, or 4 outside this path (a window at the
// box's edge, position derivatives, many components); -1 and a report for a
// bad one.
__device__ __forceinline__ int pair_list(const tb_fft_item& it, int i, tb_status* st) {
    if (!item_ok(it, nullptr)) {
        tb::report(st, TB_STATUS_BAD_ITEM, i, it.sz);
        return -1;
    }
    return it.dmode != TB_FFT_VALUE || it.K > kPairMaxK || !split_eligible(it) ? 4
           : it.sz == 256 ? 0 : it.sz == 128 ? 1 : it.sz == 64 ? 2 : 3;
}

// Sorts the items into their lists.  Up to kSortItems items one CTA does it all (alone:
// the counters and the status word are cleared here); more, many CTAs after
// memsets.
constexpr int kSortThreads = 512, kSortItems = 4096;

__global__ void __launch_bounds__(kSortThreads)
fourier_sort_kernel(const tb_fft_item* __restrict__ items, int n,
                    PairWs* ws, int32_t* __restrict__ lists,
                    tb_status* st, bool alone) {
    if (alone) {
        if (threadIdx.x < 10) ws->count[threadIdx.x] = 0;   // count[5], next[5]
        if (st && threadIdx.x == 0) *st = tb_status{};
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    for (int i0 = blockIdx.x * kSortThreads; i0 < n; i0 += gridDim.x * kSortThreads) {
        const int i = i0 + threadIdx.x;
        const int c = i < n ? pair_list(items[i], i, st) : -1;
        for (int q = 0; q < 5; q++) {   // one atomic per warp and list
            const unsigned m = __ballot_sync(0xffffffffu, c == q);
            if (m == 0) continue;
            int base = 0;
            if (lane == __ffs(m) - 1) base = atomicAdd(&ws->count[q], __popc(m));
            base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
            if (c == q) lists[q * (int64_t)n + base + __popc(m & ((1u << lane) - 1u))] = i;
        }
    }
}

// Galaxies prepared and sorted in one launch, a warp each (the lists' counters
// and the status word cleared before).
constexpr int kPrepSortThreads = 128;

__global__ void __launch_bounds__(kPrepSortThreads)
galaxy_prep_sort_kernel(const tb_galaxy_src* __restrict__ srcs, int n, tb_fft_image img,
                        tb_profile_tables Tg, tb_fft_item* __restrict__ items,
                        double* __restrict__ camp, double* __restrict__ cvar, int stride,
                        int32_t* __restrict__ flags, PairWs* ws, int32_t* __restrict__ lists,
                        tb_status* st) {
    const tb_profile_tables T = Tg;   // (read where they lie, as by tb_galaxy_fft_prep)
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * (kPrepSortThreads / 32) + (threadIdx.x >> 5);
    if (i >= n) return;   // whole warps leave together
    tb_fft_item it;
    tb::prep_galaxy_tables(srcs, i, img, T, lane, items, camp, cvar, stride, flags, it);
    if (lane != 0) return;
    const int c = pair_list(it, i, st);
    if (c >= 0) lists[c * (int64_t)n + atomicAdd(&ws->count[c], 1)] = i;
}
