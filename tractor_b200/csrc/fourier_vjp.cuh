// The vector-Jacobian product of the pixelized-PSF renderer as one adjoint
// pass per galaxy (included by fourier_render.cu after fourier_pair.cuh).
//
// A galaxy's patch is linear in its spectrum F: out = osc sum_{w,v} c_v Re[F P
// Hx Hy exp(2 pi i (w r + v c) / N)] over the rfft columns v (c_v = 1 at v = 0
// and N/2, else 2), with the PSF spectrum P and the Lanczos taps' responses Hx,
// Hy.  So with U the transform of the upstream gradient u (zero outside the
// window), the contraction with the patch of any derivative spectrum F_j is
//   sum u out_j = osc sum_{w,v} F_j W,  W = c_v Re(P Hx Hy conj U),
// and the position derivatives take the derivative taps' responses in W
// instead.  The galaxy's components share one evaluation: per component
// sums of E W, E W w, E W w^2 give the counts, the three shape parameters and
// the Sersic index (their spectra are E (da + ba v^2 + bb v w + bc w^2)), sums
// of E Wx and E Wy the position.  One forward transform and one evaluation per
// galaxy replace seven renders (spectrum, inverse transform, product with u).
//
// Groups, sizes and packed transforms as in fourier_pair.cuh.  Row pass: four
// rows of u as two complex transforms, stored as they come: S1[quad (N + 1) +
// n] = the two transforms' values (re, im, re, im) at n.  Column pass: two
// columns per job, their rows recovered from the transforms at v and N - v, a
// transform along r, then the sums.  Columns 0 and N/2 (real rows: one common
// transform) are left to a last step.
// Sums in FP32 per thread, in FP64 over the group, in a fixed order.
// With the preparation, 256 galaxies of 40 to 253 pixels: 558 us for seven
// renders and the sums against the gradient, now 199; of 200 pixels 1039, 225; the
// relative error against FP64 is the same (2.6e-7).

constexpr int kVjpMaxK = 16;

template <int N>
struct VjpPlan {
    using Pair = PairPlan<N>;
    static constexpr int NH = Pair::NH;
    static constexpr int kRows = N == 256 ? 132 : N - 4;   // rows of S1
    static constexpr int kWarps = Pair::kThreads / 32;
    static constexpr int kS1 = kRows / 4 * (N + 1) * 16;
    static constexpr int kHx = (2 * NH * 8 + 15) / 16 * 16;
    static constexpr int kBytes = Pair::kXbuf + kS1 + kHx + 2 * N * 16 /* hy */ + N * 16 /* tw */ +
                                  2 * N * 8 /* edge */ + 6 * kVjpMaxK * 16 /* comp .. */ +
                                  7 * kWarps * 8 /* red */ + (7 * kWarps % 2) * 8 +
                                  32 * 4 /* taps */ + 16 /* slot */;
    static_assert(kRows % 4 == 0 && kBytes % 16 == 0, "layout");
};
constexpr int kVjpSmem = 232448 - 1024;   // (and the static part)
static_assert(VjpPlan<256>::kBytes <= kVjpSmem &&
              VjpPlan<128>::Pair::kGroups * VjpPlan<128>::kBytes <= kVjpSmem &&
              VjpPlan<64>::Pair::kGroups * VjpPlan<64>::kBytes <= kVjpSmem &&
              VjpPlan<32>::Pair::kGroups * VjpPlan<32>::kBytes <= kVjpSmem && kSmemBytes <= kVjpSmem,
              "shared memory of an SM");

struct VjpGroup {
    tb::f32x2* xbuf;
    float4* s1;
    float2 *hx, *dhx;     // x taps' and derivative taps' responses
    float4 *hy, *dhy;     // the y ones, twice each (tb::factor)
    float4* tw;
    float2* edge;         // U of columns 0 and N/2
    float4 *comp, *aux;   // as PairGroup
    float4* dc;           // [4][kVjpMaxK]: (da, ba, bb, bc) of s0, s1, s2 and the index
    double* red;
    float* taps;          // x, y, d/dx, d/dy, 8 floats each
    int* slot;
    int tid, bar;
    template <int N>
    __device__ __forceinline__ void sync() const {
        if constexpr (PairPlan<N>::kThreads == 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(PairPlan<N>::kThreads) : "memory");
    }
};

// Row pass: the transforms of rows [rlo, rlo + nrows) of u into S1.
template <int N>
__device__ __forceinline__ void vjp_rows(const VjpGroup& sh, const float* __restrict__ u,
                                         int64_t ldo, int row0, int nrows, int c0, int c1) {
    using namespace tb;
    constexpr int G = N / 16;
    const int t = sh.tid % G, grp = sh.tid / G;
    f32x2* xb = sh.xbuf + grp * pair_xbuf<N>();
    const int nq = (nrows + 3) / 4;
    for (int i0 = 0; i0 < nq; i0 += PairPlan<N>::kLanes) {
        const bool act = i0 + grp < nq;
        const int i = act ? i0 + grp : nq - 1;
        const float* p = u + (int64_t)(row0 + 4 * i) * ldo;
        const int last = nrows - 4 * i;
        C2 x[16];
#pragma unroll
        for (int m = 0; m < 16; m++) {
            const int c = t + G * m;
            const bool in = c >= c0 && c < c1;
            const float r0 = in ? __ldg(p + c) : 0.f;
            const float r1 = in && last > 1 ? __ldg(p + ldo + c) : 0.f;
            const float r2 = in && last > 2 ? __ldg(p + 2 * ldo + c) : 0.f;
            const float r3 = in && last > 3 ? __ldg(p + 3 * ldo + c) : 0.f;
            x[m] = C2{pack(r0, r2), pack(r1, r3)};
        }
        float4* s = sh.s1 + i * (N + 1) + t;
        fft_pair<N, -1>(x, t, xb, sh.tw, [&](int g, int q, C2 z) {
            const float2 re = unpack(z.re), im = unpack(z.im);
            if (act) s[G * g + 16 * q] = make_float4(re.x, im.x, re.y, im.y);
        });
        __syncwarp();
    }
}

// Element (row r, column v) of the rows' transforms from S1: row r is the real
// (part 0) or imaginary (part 1) input of its transform.
template <int N>
__device__ __forceinline__ float2 vjp_element(const float2* s, int v, int part) {
    const float2 z = s[2 * v], y = s[2 * ((N - v) & (N - 1))];
    return part == 0 ? make_float2(0.5f * (z.x + y.x), 0.5f * (z.y - y.y))
                     : make_float2(0.5f * (z.y + y.y), 0.5f * (y.x - z.x));
}

// Column pass over the interior columns 1 .. N/2 - 1: adds this thread's share
// of the seven sums (x, y, counts, s0, s1, s2, index; unscaled) and leaves U of
// columns 0 and N/2 in `edge`.
template <int N>
__device__ __forceinline__ void vjp_columns(const VjpGroup& sh, int K,
                                            const float* __restrict__ spec, int rlo, int nrows,
                                            float (&dot)[7]) {
    using namespace tb;
    constexpr int G = N / 16;
    const int t = sh.tid % G, grp = sh.tid / G;
    f32x2* xb = sh.xbuf + grp * pair_xbuf<N>();
    const float2* P = reinterpret_cast<const float2*>(spec) + t;
    const float2* S = reinterpret_cast<const float2*>(sh.s1);
    const float w0 = (float)t / (float)N - 0.5f, span = (float)(G - 1) / N;
    for (int j0 = 0; j0 < N / 4; j0 += PairPlan<N>::kLanes) {
        const bool act = j0 + grp < N / 4;
        const int va = 2 * (act ? j0 + grp : N / 4 - 1), vb = va + 1;
        C2 x[16];
        const int base = t - rlo, part = base & 1;
#pragma unroll
        for (int m = 0; m < 16; m++) {
            const int r = base + G * m;
            const bool in = (unsigned)r < (unsigned)nrows;
            const float2* s = S + (in ? ((r >> 2) * (N + 1)) * 2 + ((r >> 1) & 1) : 0);
            float2 a = vjp_element<N>(s, va, part), b = vjp_element<N>(s, vb, part);
            if (j0 == 0) {
                // columns 0 and N/2 (real) as one transform in place of column 0
                const float2 z0 = s[0], zN = s[N];
                const float2 e = part == 0 ? make_float2(z0.x, zN.x) : make_float2(z0.y, zN.y);
                a.x = va == 0 ? e.x : a.x;
                a.y = va == 0 ? e.y : a.y;
            }
            x[m] = C2{in ? pack(a.x, b.x) : 0ull, in ? pack(a.y, b.y) : 0ull};
        }
        C2 U[16];   // row t + G m
        fft_pair<N, -1>(x, t, xb, sh.tw, [&](int g, int q, C2 z) { U[g + (16 / G) * q] = z; });
        __syncwarp();
        if (j0 == 0) {
            // U_0 = (Z(w) + conj Z(-w)) / 2, U_N/2 = (Z(w) - conj Z(-w)) / 2i
            float2* zb = reinterpret_cast<float2*>(xb);
#pragma unroll
            for (int m = 0; m < 16; m++)
                zb[t + G * m] = make_float2(unpack(U[m].re).x, unpack(U[m].im).x);
            __syncwarp();
#pragma unroll
            for (int m = 0; m < 16; m++) {
                const int j = t + G * m;
                const float2 z = zb[j], y = zb[(N - j) & (N - 1)];
                if (va == 0) {
                    sh.edge[j] = make_float2(0.5f * (z.x + y.x), 0.5f * (z.y - y.y));
                    sh.edge[N + j] = make_float2(0.5f * (z.y + y.y), 0.5f * (y.x - z.x));
                }
            }
            __syncwarp();
        }
        if (!act) continue;
        // twice the interior columns; column 0 is left to vjp_edges
        const f32x2 weight = pack(va == 0 ? 0.f : 2.f, 2.f);
        const float2 hxa = sh.hx[va], hxb = sh.hx[vb], dxa = sh.dhx[va], dxb = sh.dhx[vb];
        const f32x2 hr = pack(hxa.x, hxb.x), hi = pack(hxa.y, hxb.y);
        const f32x2 dr = pack(dxa.x, dxb.x), di = pack(dxa.y, dxb.y);
        const float fa = (float)va / N, fb = (float)vb / N;
        const f32x2 v2 = pack(fa, fb), vv = mul2(v2, v2);
#pragma unroll
        for (int h = 0; h < 2; h++) {   // the rows of negative, then of positive frequency
            f32x2 W[8], Wx[8], Wy[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int m = i + 8 * (1 - h), j = G * m;
                const float2 pa = __ldg(P + va * N + j), pb = __ldg(P + vb * N + j);
                const f32x2 pr = mul2(weight, pack(pa.x, pb.x)), pi = mul2(weight, pack(pa.y, pb.y));
                // Z = P conj U
                const C2 z = C2{fma2(pi, U[m].im, mul2(pr, U[m].re)),
                                sub2(mul2(pi, U[m].re), mul2(pr, U[m].im))};
                const C2 zy = cmul2(z, factor(sh.hy, t + j)), zd = cmul2(z, factor(sh.dhy, t + j));
                W[i] = sub2(mul2(zy.re, hr), mul2(zy.im, hi));
                Wx[i] = sub2(mul2(zy.re, dr), mul2(zy.im, di));
                Wy[i] = sub2(mul2(zd.re, hr), mul2(zd.im, hi));
            }
            const float wh = w0 + 0.5f * h;
            for (int k = 0; k < K; k++) {
                const float4 a = sh.aux[k];
                const float top = a.x * fa * fa;
                if (top < kSpecFloor) continue;
                const float h2 = (top - kSpecFloor) * a.z + 1e-30f, half = h2 * rsqrtf(h2);
                const float lo = fminf(a.y * fa, a.y * fb) - half - span - 3.f / 16.f;
                const float hi_w = fmaxf(a.y * fa, a.y * fb) + half;
                const float4 c = sh.comp[k];
                const f32x2 al = mul2(vv, both(c.y)), be = mul2(v2, both(c.z)), cd = both(c.w);
                f32x2 s0 = 0ull, s1 = 0ull, s2 = 0ull, sx = 0ull, sy = 0ull;
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    const float wf = -0.5f + 0.5f * h + 0.25f * g;
                    if (wf < lo || wf > hi_w) continue;
#pragma unroll
                    for (int i = 4 * g; i < 4 * g + 4; i++) {
                        const f32x2 w = both(wh + (float)i / 16.f);
                        const float2 e = unpack(fma2(w, fma2(cd, w, be), al));
                        const f32x2 E = pack(ex2(e.x), ex2(e.y));
                        const f32x2 q = mul2(E, W[i]), qw = mul2(q, w);
                        s0 = add2(s0, q);
                        s1 = add2(s1, qw);
                        s2 = fma2(qw, w, s2);
                        sx = fma2(E, Wx[i], sx);
                        sy = fma2(E, Wy[i], sy);
                    }
                }
                const float2 q0 = unpack(s0), q1 = unpack(s1), q2 = unpack(s2);
                const float2 qx = unpack(sx), qy = unpack(sy);
                dot[0] = fmaf(c.x, qx.x + qx.y, dot[0]);
                dot[1] = fmaf(c.x, qy.x + qy.y, dot[1]);
                dot[2] = fmaf(c.x, q0.x + q0.y, dot[2]);
                const float m0 = q0.x + q0.y, mv = fa * fa * q0.x + fb * fb * q0.y;
                const float mw = fa * q1.x + fb * q1.y, m2 = q2.x + q2.y;
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    const float4 d = sh.dc[p * kVjpMaxK + k];
                    dot[3 + p] += d.x * m0 + d.y * mv + d.z * mw + d.w * m2;
                }
            }
        }
    }
}

// The sums over columns 0 and N/2, an element per thread and turn.
template <int N>
__device__ __forceinline__ void vjp_edges(const VjpGroup& sh, int K,
                                          const float* __restrict__ spec, float (&dot)[7]) {
    const float2* P = reinterpret_cast<const float2*>(spec);
    for (int e = sh.tid; e < 2 * N; e += PairPlan<N>::kThreads) {
        const int j = e & (N - 1), col = e < N ? 0 : N / 2;
        const float v = (float)col / N, w = (float)(j < N / 2 ? j : j - N) / (float)N;
        const float2 U = sh.edge[e], p = __ldg(P + (int64_t)col * N + j);
        const float2 z = make_float2(p.x * U.x + p.y * U.y, p.y * U.x - p.x * U.y);
        const float4 hy = sh.hy[j], dy = sh.dhy[j];
        const float2 zy = cmulf(z, make_float2(hy.x, hy.z)), zd = cmulf(z, make_float2(dy.x, dy.z));
        const float2 hx = sh.hx[col], dx = sh.dhx[col];
        const float W = zy.x * hx.x - zy.y * hx.y, Wx = zy.x * dx.x - zy.y * dx.y;
        const float Wy = zd.x * hx.x - zd.y * hx.y;
        for (int k = 0; k < K; k++) {
            const float4 c = sh.comp[k];
            const float E = tb::ex2(fmaf(w, fmaf(c.w, w, c.z * v), c.y * v * v));
            dot[0] = fmaf(c.x * E, Wx, dot[0]);
            dot[1] = fmaf(c.x * E, Wy, dot[1]);
            dot[2] = fmaf(c.x * E, W, dot[2]);
#pragma unroll
            for (int p = 0; p < 4; p++) {
                const float4 d = sh.dc[p * kVjpMaxK + k];
                const float pre = d.x + d.y * v * v + w * (d.z * v + d.w * w);
                dot[3 + p] = fmaf(pre * E, W, dot[3 + p]);
            }
        }
    }
}

// One galaxy: items[0 .. 7) in tb_galaxy_fft_jac_prep's order.
template <int N>
__device__ void vjp_source(const tb_fft_item* __restrict__ items, const VjpGroup& sh,
                           const double* __restrict__ amp, const double* __restrict__ var,
                           const double* __restrict__ dcoef, const float* __restrict__ psf_spec,
                           const float* __restrict__ grad, double* __restrict__ dots) {
    constexpr int kThreads = PairPlan<N>::kThreads, NH = PairPlan<N>::NH;
    const tb_fft_item& it = items[2];
    const int mw = it.mw, mh = it.mh, sx = it.sx, sy = it.sy, K = it.K;
    const int64_t ldo = it.ldo > 0 ? it.ldo : mw;
    const int gr0 = max(0, -sy), gr1 = min(N, mh - sy);
    const int gc0 = max(0, -sx), gc1 = min(N, mw - sx);
    const double c2 = -2.0 * TB_PI * TB_PI * TB_LOG2E;
    for (int e = sh.tid; e < 5 * K; e += kThreads) {
        const int k = e % K, p = e / K, c = it.c0 + k;
        if (p == 4) {
            const float4 f = make_float4((float)amp[c], (float)(c2 * var[4 * c]),
                                         (float)(c2 * 2.0 * var[4 * c + 1]),
                                         (float)(c2 * var[4 * c + 3]));
            sh.comp[k] = f;
            sh.aux[k] = stage_aux(f);
        } else {
            const double* d = dcoef + 4 * ((int64_t)items[3 + p].dc0 + k);
            const double m2 = -2.0 * TB_PI * TB_PI * amp[c];
            sh.dc[p * kVjpMaxK + k] = make_float4((float)d[0], (float)(m2 * d[1]),
                                                  (float)(m2 * 2.0 * d[2]), (float)(m2 * d[3]));
        }
    }
    for (int q = sh.tid / 32; q < 4; q += kThreads / 32)
        taps_warp(q % 2 == 0 ? it.mux : it.muy, q >= 2, sh.taps + 8 * q);
    sh.template sync<N>();
    for (int f = sh.tid; f < 2 * (NH + N); f += kThreads) {
        const bool d = f >= NH + N;
        const int g = d ? f - NH - N : f, fr = g < NH ? g : g - NH;
        const float2 r = tap_response<N>(sh.taps + 8 * ((g < NH ? 0 : 1) + (d ? 2 : 0)), fr);
        if (g < NH) (d ? sh.dhx : sh.hx)[fr] = r;
        else (d ? sh.dhy : sh.hy)[fr] = make_float4(r.x, r.x, r.y, r.y);
    }
    const float* spec = psf_spec + it.spec_off;
    const float* u = grad + it.out_off + sx;
    float dot[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int a = gr0; a < gr1; a += VjpPlan<N>::kRows) {
        const int nrows = min(VjpPlan<N>::kRows, gr1 - a);
        vjp_rows<N>(sh, u, ldo, a + sy, nrows, gc0, gc1);
        sh.template sync<N>();
        vjp_columns<N>(sh, K, spec, a, nrows, dot);
        sh.template sync<N>();
        vjp_edges<N>(sh, K, spec, dot);
    }
    // the group's sums, in FP64 and a fixed order
    const int lane = sh.tid & 31, warp = sh.tid >> 5;
#pragma unroll
    for (int p = 0; p < 7; p++) {
        double d = (double)dot[p];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if (lane == 0) sh.red[p * VjpPlan<N>::kWarps + warp] = d;
    }
    sh.template sync<N>();
    if (sh.tid < 7) {
        double d = 0.0;
        for (int q = 0; q < VjpPlan<N>::kWarps; q++) d += sh.red[sh.tid * VjpPlan<N>::kWarps + q];
        dots[items[sh.tid].dot_off] = d * ((double)items[sh.tid].scale / ((double)N * N));
    }
}

template <int N>
__device__ void vjp_size(unsigned char* smem, const tb_fft_item* __restrict__ items,
                         const int32_t* __restrict__ list, int count, int total, int32_t* next,
                         const double* __restrict__ amp, const double* __restrict__ var,
                         const double* __restrict__ dcoef, const float* __restrict__ psf_spec,
                         const float* __restrict__ grad, double* __restrict__ dots) {
    using Plan = VjpPlan<N>;
    if (count == 0) return;   // the same in every thread
    const int g = threadIdx.x / Plan::Pair::kThreads;
    __syncthreads();   // the previous size's groups are done with shared memory
    if (g >= active_groups(Plan::Pair::kGroups, count, total)) return;
    unsigned char* p = smem + g * Plan::kBytes;
    auto take = [&](int bytes) {
        unsigned char* q = p;
        p += bytes;
        return q;
    };
    VjpGroup sh;
    sh.tid = threadIdx.x % Plan::Pair::kThreads;
    sh.bar = 1 + g;
    sh.xbuf = reinterpret_cast<tb::f32x2*>(take(Plan::Pair::kXbuf));
    sh.s1 = reinterpret_cast<float4*>(take(Plan::kS1));
    sh.hx = reinterpret_cast<float2*>(take(Plan::kHx));
    sh.dhx = sh.hx + Plan::NH;
    sh.hy = reinterpret_cast<float4*>(take(N * 16));
    sh.dhy = reinterpret_cast<float4*>(take(N * 16));
    sh.tw = reinterpret_cast<float4*>(take(N * 16));
    sh.edge = reinterpret_cast<float2*>(take(2 * N * 8));
    sh.comp = reinterpret_cast<float4*>(take(kVjpMaxK * 16));
    sh.aux = reinterpret_cast<float4*>(take(kVjpMaxK * 16));
    sh.dc = reinterpret_cast<float4*>(take(4 * kVjpMaxK * 16));
    sh.red = reinterpret_cast<double*>(take(7 * Plan::kWarps * 8 + (7 * Plan::kWarps % 2) * 8));
    sh.taps = reinterpret_cast<float*>(take(32 * 4));
    sh.slot = reinterpret_cast<int*>(take(16));
    tb::build_pair_twiddles<N>(sh.tw, sh.tid, Plan::Pair::kThreads);
    for (;;) {
        if (sh.tid == 0) *sh.slot = atomicAdd(next, 1);
        sh.template sync<N>();
        const int u = *sh.slot;
        if (u >= count) break;
        vjp_source<N>(items + 7 * (int64_t)list[u], sh, amp, var, dcoef, psf_spec, grad, dots);
        sh.template sync<N>();
    }
}

__global__ void __launch_bounds__(kPairThreads, 1)
fourier_vjp_kernel(const tb_fft_item* __restrict__ items, int n,
                   const double* __restrict__ amp, const double* __restrict__ var,
                   const double* __restrict__ dcoef, const float* __restrict__ psf_spec,
                   float* __restrict__ grad, double* __restrict__ dots, PairWs* ws,
                   const int32_t* __restrict__ lists, tb_status* st) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int4 c = *reinterpret_cast<const int4*>(ws->count);
    const int rest = ws->count[4], total = c.x + c.y + c.z + c.w + rest;
    if (rest != 0)
        whole_cta_list<true>(items, 7 * n, amp, var, dcoef, psf_spec, grad, dots, &ws->next[4], st,
                             lists + 4 * (int64_t)n, rest, smem_raw);
    vjp_size<256>(smem_raw, items, lists, c.x, total, &ws->next[0], amp, var, dcoef, psf_spec, grad,
                  dots);
    vjp_size<128>(smem_raw, items, lists + n, c.y, total, &ws->next[1], amp, var, dcoef, psf_spec,
                  grad, dots);
    vjp_size<64>(smem_raw, items, lists + 2 * (int64_t)n, c.z, total, &ws->next[2], amp, var, dcoef,
                 psf_spec, grad, dots);
    vjp_size<32>(smem_raw, items, lists + 3 * (int64_t)n, c.w, total, &ws->next[3], amp, var, dcoef,
                 psf_spec, grad, dots);
}

// Sorts the galaxies by FFT size; the seven items of one whose window does not
// keep 3 px from the box's edges (or with many components) go to list 4.
__global__ void __launch_bounds__(128)
fourier_vjp_sort_kernel(const tb_fft_item* __restrict__ items, int n,
                        const double* __restrict__ dcoef, PairWs* ws, int32_t* __restrict__ lists,
                        double* __restrict__ dots, tb_status* st) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const tb_fft_item* I = items + 7 * (int64_t)i;
    const tb_fft_item it = I[2];
    bool ok = true;
    for (int p = 0; p < 7; p++) ok = ok && item_ok(I[p], dcoef) && I[p].mode == TB_FFT_DOT;
    if (!ok) {
        tb::report(st, TB_STATUS_BAD_ITEM, i, it.sz);
        return;
    }
    const int N = it.sz;
    const int gr0 = max(0, -it.sy), gr1 = min(N, it.mh - it.sy);
    const int gc0 = max(0, -it.sx), gc1 = min(N, it.mw - it.sx);
    if (it.K == 0 || gr0 >= gr1 || gc0 >= gc1) {   // no patch
        for (int p = 0; p < 7; p++) dots[I[p].dot_off] = 0.0;
        return;
    }
    if (it.K <= kVjpMaxK && gc0 >= 3 && gc1 <= N - 3 && gr0 >= 3 && gr1 <= N - 3) {
        const int c = N == 256 ? 0 : N == 128 ? 1 : N == 64 ? 2 : 3;
        lists[c * (int64_t)n + atomicAdd(&ws->count[c], 1)] = i;
    } else {
        const int at = atomicAdd(&ws->count[4], 7);
        for (int p = 0; p < 7; p++) lists[4 * (int64_t)n + at + p] = 7 * i + p;
    }
}
