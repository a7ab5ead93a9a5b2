// Batched EM fit of 2-D Gaussian mixtures to images (sm_100a): the batched
// form of em_fit_2d_reg (tractor/emfit.i:274-557), which
// GaussianMixturePSF.fromStamp (tractor/psf.py:536-597) runs on a PSF stamp.
//
// One CTA per image, all iterations inside the kernel, FP64 throughout (as
// the reference).  Each iteration:
//   * per component: C^-1 and amp / (2 pi sqrt det C) (a non-positive
//     determinant stops the fit, as the reference returns -1 there);
//   * E step: the responsibility of component k at pixel (x, y) is
//     z_k / sum_j z_j (as z_k times the sum's reciprocal) with
//     z_k = scale_k exp(-dsq_k / 2), 0 for dsq >= 100 (z itself where the
//     sum is 0, as the reference leaves it);
//   * M step from the weighted moments w = img z_k / sum z (sum w, sum w x,
//     sum w y, sum w x^2, sum w x y, sum w y^2), summed per thread, then over
//     the block in a fixed order (every launch gives the same result):
//     mean = (sum w x, sum w y) / sum w, covariance = (alpha I + sum w
//     (x - mean)(x - mean)^T) / (sum w + alpha) with sum w (x - m)^2 =
//     sum w x^2 - m sum w x, amplitude = sum w.
// The reference sums the second moments about the new mean in a second pass
// over the pixels; the expansion above is the same sum in one pass (the
// difference is FP64 rounding).
//
// Bound: FP64 issue and latency (60 % of the issue slots, 37 % of the FP64 pipe;
// the rest waits on the chain of a pixel's exponentials, their sum and its
// reciprocal).  A thread keeps one column of pixels, so a component's exponent
// is a quadratic in y alone, its moments three sums (w, w y, w y^2) and the x
// moments follow once per column; the exponential is exp2_tab; each warp takes
// the M step and the next iteration's parameters itself, so an iteration has
// one block barrier.  100 iterations, 1024 stamps of 25 x 25 (against a pixel
// stride per thread with exp(), divisions and a butterfly per moment): 1
// component 487 -> 410 us, 3 components 1033 -> 797, 8 components 4589 -> 2661;
// 256 stamps of 63 x 63, 3 components 3080 -> 2391.
//
// Rounding: EM converges slowly, so the fixed point amplifies every rounding of an
// iteration, those shared by all pixels most.  Hence the exponents' coefficients
// to the last bit (`prepare`), the exponential's table in two parts, and, where it
// costs no turn, a thread's runs of columns in mirrored pairs, whose first moments
// cancel before they are rounded together.  After 1000 iterations, against
// extended precision, over eight sets of stamps (15 to 27 px, 1 to 3 components)
// the geometric means of the rms errors are 4.9e-16 in the amplitudes, 6.9e-16 in
// the means and 6.9e-15 in the variances; with one pixel at a time, exp() and
// divisions 4.6e-16, 7.0e-16 and 7.1e-15; without those three 5.3e-16, 1.0e-15 and
// 8.4e-15 (1024 stamps, 3 components: 7.5 in place of 7.8 ms).
#include <type_traits>

#include "tb_common.cuh"

namespace {

constexpr int kEmThreads = 64;
constexpr int kWarps = kEmThreads / 32;

// 1 / d, as accurate as the division to its last bit or so: Newton's
// iteration from the hardware's estimate; the division itself where the
// estimate would be flushed.
__device__ __forceinline__ double em_reciprocal(double d) {
    if (!(fabs(d) > 1e-290 && fabs(d) < 1e290)) return 1.0 / d;
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    r = fma(r, fma(-d, r, 1.0), r);
    return fma(r, fma(-d, r, 1.0), r);
}

// The sums over the warp of each lane's a[0 .. N): every exchange leaves a lane
// half of the values it had (about N shuffles instead of 5 N); at the end it
// holds `count` sums, of the elements `first` on.
template <int M, int N, int O>
__device__ __forceinline__ void halve(double (&a)[M], int lane, int& first, int& count) {
    if constexpr (O > 0) {
        constexpr int H = (N + 1) / 2;
        if constexpr (N > 1) {
            const bool hi = lane & O;
#pragma unroll
            for (int i = 0; i < H; i++) {
                const double up = i + H < N ? a[i + H] : 0.0;
                const double send = hi ? a[i] : up, keep = hi ? up : a[i];
                a[i] = keep + __shfl_xor_sync(0xffffffffu, send, O);
            }
            first += hi ? H : 0;
            count = hi ? count - H : min(count, H);
        } else {
            a[0] += __shfl_xor_sync(0xffffffffu, a[0], O);
        }
        halve<M, H, O / 2>(a, lane, first, count);
    }
}

// out[e] = the sum over the warp of a[e], e < M <= 64.
template <int M>
__device__ __forceinline__ void warp_sums(double (&a)[M], int lane, double* out) {
    int first = 0, count = M;
    halve<M, M, 16>(a, lane, first, count);
#pragma unroll
    for (int i = 0; i < (M > 32 ? 2 : 1); i++)
        if (i < count) out[first + i] = a[i];   // (equal values from lanes that share one)
}

// (resident CTAs: 7 up to 5 components, which hold 1024 stamps in one wave: 3
// components 7.8 ms, with 8 and fewer registers 8.5; 5 components 1306 us, with 6 a
// second wave 2000)
template <int K>
__global__ void __launch_bounds__(kEmThreads, K <= 5 ? 7 : 4)
em_fit_kernel(const double* __restrict__ img, int n, int ny, int nx,
              const int32_t* __restrict__ xy0, double* __restrict__ amp,
              double* __restrict__ mean, double* __restrict__ var, double alpha, int steps,
              int32_t* __restrict__ status) {
    constexpr int kM = 6 * K;   // moments per image
    // per warp: the current mixture, and what the E step reads of it (all
    // exponents in log2 units)
    __shared__ double par[kWarps][K][8];   // mean x, y, c00, c01, c11, scale
    __shared__ double red[2][kWarps][kM];
    // (one component's responsibility is 1 but for rounding, whatever the exponential)
    constexpr bool kFine = K > 1;
    __shared__ std::conditional_t<kFine, double2, double> exp_tab[tb::kExpTab];
    const int s = blockIdx.x;
    if (s >= n) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double* im = img + (int64_t)s * ny * nx;
    double* A = amp + (int64_t)s * K;
    double* Mu = mean + (int64_t)s * K * 2;
    double* V = var + (int64_t)s * K * 4;
    const int x0 = xy0 ? xy0[2 * s] : -(nx / 2);
    const int y0 = xy0 ? xy0[2 * s + 1] : -(ny / 2);
    // The columns are cut into `groups` runs of `rows` pixels, taken by the
    // threads in turn: the cut that keeps the threads busiest, a run's start
    // counted as half a pixel (as two, 300 iterations of 1024 stamps of 23 x 23, 3
    // components, took 2574 us, 2490 with the rounding of before; now 2259).
    int groups = 1, rows = ny;
    {
        int best = 0x7fffffff;
        for (int g = 1; g <= max(8, kEmThreads / nx) && g <= ny; g++) {
            const int r = (ny + g - 1) / g;
            const int cost = (nx * g + kEmThreads - 1) / kEmThreads * (2 * r + 1);
            if (cost < best) { best = cost; groups = g; rows = r; }
        }
    }
    const int step_x = kEmThreads % nx, step_g = kEmThreads / nx;
    // runs q and N - 1 - q (mirrored at the image's centre) by the same thread,
    // where that takes no more turns
    const int N = nx * groups;
    const bool mirror = 2 * (((N + 1) / 2 + kEmThreads - 1) / kEmThreads) <=
                        (N + kEmThreads - 1) / kEmThreads;
    const double tpd = 4.0 * TB_PI * TB_PI;   // (2 pi)^D, D = 2
    tb::exp2_tab_init(exp_tab);
    // component `lane` of this warp's copy: the exponents' coefficients and the
    // scale from its mixture; whether its determinant is positive.  `tame`: its
    // exponent is <= 0 (but for rounding) and finite at every pixel, as the
    // table-driven exponential needs it.
    bool tame = true;
    auto prepare = [&](double w, double mx, double my, double v00, double v01, double v10,
                       double v11) -> bool {
        const double det = v00 * v11 - v01 * v10;
        double* p = par[warp][lane];
        p[0] = mx;
        p[1] = my;
        // q + ql = -log2(e) / (2 det): the quotient's remainder, the constant's
        // second part and the rounding of det
        const double c = -0.5 * TB_LOG2E, q = c / det;
        double ql = 0.0;
        if constexpr (kFine) {
            const double b = v01 * v10, be = fma(v01, v10, -b);
            const double dl = (fma(v00, v11, -det) - b) - be;
            ql = ((fma(-q, det, c) - 0.5 * 2.0355273740931033e-17) - q * dl) *
                 (q * -1.3862943611198906);   // (1 / c)
        }
        p[2] = fma(v11, q, v11 * ql);
        p[3] = -fma(v01 + v10, q, (v01 + v10) * ql);
        p[4] = fma(v00, q, v00 * ql);
        p[5] = w / sqrt(tpd * det);
        const double off = v01 + v10;
        tame = p[2] < 0.0 && p[4] < 0.0 && 4.0 * v00 * v11 > off * off && p[2] > -1e100 &&
               p[4] > -1e100 && fabs(mx) < 1e50 && fabs(my) < 1e50;
        return !(det <= 0.0);
    };
    bool ok = true;
    double fw = 0.0, fmx = 0.0, fmy = 0.0, f00 = 0.0, f01 = 0.0, f10 = 0.0, f11 = 0.0;
    if (lane < K) {
        fw = A[lane];
        fmx = Mu[2 * lane];
        fmy = Mu[2 * lane + 1];
        f00 = V[4 * lane];
        f01 = V[4 * lane + 1];
        f10 = V[4 * lane + 2];
        f11 = V[4 * lane + 3];
        ok = prepare(fw, fmx, fmy, f00, f01, f10, f11) || steps <= 0;
    }
    __syncthreads();   // the table
    int bad = 0;
    for (int step = 0; step < steps; step++) {
        if (!__all_sync(0xffffffffu, ok)) {   // the same in every warp
            bad = 1;
            break;
        }
        double acc[kM];
#pragma unroll
        for (int v = 0; v < kM; v++) acc[v] = 0.0;
        auto e_step = [&](auto table) {
            int qx = tid % nx, qr = tid / nx;
            bool back = false;
            while (qr < groups) {
                if (qx >= nx) {
                    qx -= nx;
                    if (++qr >= groups) break;
                }
                const int q = qr * nx + qx;
                if (mirror && 2 * q >= N) break;
                const int ix = back ? nx - 1 - qx : qx, run = back ? groups - 1 - qr : qr;
                const int ra = run * rows, rb = min(ny, ra + rows);
                const double x = (double)(x0 + ix);
                double ca[K], cb[K], S0[K], Sy[K];
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const double dx = x - par[warp][k][0];
                    ca[k] = par[warp][k][2] * dx * dx;
                    cb[k] = par[warp][k][3] * dx;
                    S0[k] = Sy[k] = 0.0;
                }
                const double* px = im + ra * nx + ix;
                double y = (double)(y0 + ra);
                double dnext = ra < rb ? *px : 0.0;
                for (int iy = ra; iy < rb; iy++, y += 1.0) {
                    const double yy = y * y, d = dnext;
                    px += nx;
                    if (iy + 1 < rb) dnext = *px;
                    double z[K];
                    double zsum = 0.0;
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        const double dy = y - par[warp][k][1];
                        const double e = fma(dy, fma(par[warp][k][4], dy, cb[k]), ca[k]);
                        const double E = decltype(table)::value ? tb::exp2_tab(e, exp_tab) : exp2(e);
                        z[k] = e <= -50.0 * TB_LOG2E ? 0.0 : par[warp][k][5] * E;   // dsq >= 100: 0
                        zsum += z[k];
                    }
                    double dr;
                    if (((unsigned)__double2hiint(zsum) << 1) - (323u << 21) < (1400u << 21)) {   // 1e-211 .. 1e210
                        dr = d * em_reciprocal(zsum);
                    } else {
                        // a pixel whose z sum to 0 keeps them unnormalised (all 0
                        // unless some amplitude is negative), as the reference does
                        const double rz = zsum != 0.0 ? 1.0 / zsum : 1.0;
#pragma unroll
                        for (int k = 0; k < K; k++) z[k] *= rz;
                        dr = d;
                    }
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        const double wi = dr * z[k];
                        S0[k] += wi;
                        Sy[k] = fma(wi, y, Sy[k]);
                        acc[6 * k + 5] = fma(wi, yy, acc[6 * k + 5]);
                    }
                }
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const double xs = x * S0[k];
                    acc[6 * k + 0] += S0[k];
                    acc[6 * k + 1] += xs;
                    acc[6 * k + 2] += Sy[k];
                    acc[6 * k + 3] = fma(xs, x, acc[6 * k + 3]);
                    acc[6 * k + 4] = fma(x, Sy[k], acc[6 * k + 4]);
                }
                back = mirror && !back && 2 * q + 1 < N;   // the middle run is its own mirror image
                if (!back) {
                    qx += step_x;
                    qr += step_g;
                }
            }
        };
        if (__all_sync(0xffffffffu, tame)) e_step(std::true_type{});
        else e_step(std::false_type{});
        double* r = red[step & 1][warp];
        warp_sums<kM>(acc, lane, r);
        __syncthreads();   // (the other half of `red` is read before the next one)
        if (lane < K) {
            double m[6];
#pragma unroll
            for (int q = 0; q < 6; q++) {
                double t = 0.0;
                for (int w2 = 0; w2 < kWarps; w2++) t += red[step & 1][w2][6 * lane + q];
                m[q] = t;
            }
            fw = m[0];
            const double rw = 1.0 / fw, rden = 1.0 / (fw + alpha);
            fmx = m[1] * rw;
            fmy = m[2] * rw;
            f00 = (alpha + (m[3] - fmx * m[1])) * rden;
            f01 = f10 = (m[4] - fmx * m[2]) * rden;
            f11 = (alpha + (m[5] - fmy * m[2])) * rden;
            ok = prepare(fw, fmx, fmy, f00, f01, f10, f11);
        }
        __syncwarp();
    }
    if (warp == 0 && lane < K) {
        A[lane] = fw;
        Mu[2 * lane] = fmx;
        Mu[2 * lane + 1] = fmy;
        V[4 * lane] = f00;
        V[4 * lane + 1] = f01;
        V[4 * lane + 2] = f10;
        V[4 * lane + 3] = f11;
    }
    if (tid == 0 && status) status[s] = bad;
}

// The EM fit with a flat sky term (em_fit_2d_reg2, tractor/emfit2.c), the
// fit GaussianMixturePSF.fromStamp(v2=True) runs (tractor/psf.py:579-588).
// Per iteration, per component: the symmetrised covariance's determinant (a
// non-positive one stops the fit), its inverse, amp / sqrt((2 pi)^2 det) and
// the cut maxD = -2 log(approx sqrt((2 pi)^2 det)); per pixel: a pixel <= 0
// adds |img| to the sky and nothing else; z_k = 0 where dsq >= maxD_k; a
// pixel whose z sum to 0 adds img to the sky; otherwise psky joins the sum,
// img psky / sum goes to the sky and w_k = img z_k / sum; the weighted
// moments (sum w, sum w x, sum w y and the second moments about the OLD
// mean, as emfit2.c accumulates them in one pass) and the sky sum are
// summed per thread over a fixed pixel stride, then over the block in a
// fixed order; then mean = sum w x / sum w, covariance = (alpha I + second
// moments) / (sum w + alpha), amplitude = sum w, psky = sky / npix.  psky
// starts at 0.01 x the image mean; its last value is the fit's sky level.
template <int K>
__global__ void __launch_bounds__(kEmThreads, 8)
em_fit_sky_kernel(const double* __restrict__ img, int n, int ny, int nx,
                  const int32_t* __restrict__ xy0, double* __restrict__ amp,
                  double* __restrict__ mean, double* __restrict__ var, double alpha, int steps,
                  double approx, double* __restrict__ skyamp, int32_t* __restrict__ status) {
    constexpr int kM = 6 * K + 1;   // moments per image, then the sky sum
    __shared__ double w_s[K], mu_s[K][2], v_s[K][4];
    __shared__ double iv_s[K][3], sc_s[K], maxd_s[K];
    __shared__ double red[kWarps][kM];
    __shared__ double psky_s;
    __shared__ int bad;
    const int s = blockIdx.x;
    if (s >= n) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double* im = img + (int64_t)s * ny * nx;
    double* A = amp + (int64_t)s * K;
    double* Mu = mean + (int64_t)s * K * 2;
    double* V = var + (int64_t)s * K * 4;
    const int x0 = xy0 ? xy0[2 * s] : -(nx / 2);
    const int y0 = xy0 ? xy0[2 * s + 1] : -(ny / 2);
    const int npix = nx * ny;
    const int ix0 = tid % nx, iy0 = tid / nx;
    const int step_x = kEmThreads % nx, step_y = kEmThreads / nx;
    const double tpd = 4.0 * TB_PI * TB_PI;
    if (tid < K) {
        w_s[tid] = A[tid];
        mu_s[tid][0] = Mu[2 * tid];
        mu_s[tid][1] = Mu[2 * tid + 1];
#pragma unroll
        for (int d = 0; d < 4; d++) v_s[tid][d] = V[4 * tid + d];
    }
    if (tid == 0) {
        bad = 0;
        psky_s = 0.0;
    }
    // the image sum (fixed-order block reduction) for the first sky level
    {
        double t = 0.0;
        for (int i = tid; i < npix; i += kEmThreads) t += im[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) red[warp][0] = t;
        __syncthreads();
        if (tid == 0 && steps > 0) {
            double sum = 0.0;
            for (int w2 = 0; w2 < kWarps; w2++) sum += red[w2][0];
            psky_s = 0.01 * sum / (double)npix;
        }
        __syncthreads();
    }
    for (int step = 0; step < steps; step++) {
        if (tid < K) {
            const double* Vk = v_s[tid];
            const double v12 = (Vk[1] + Vk[2]) / 2.0;
            const double det = Vk[0] * Vk[3] - v12 * v12;
            if (det <= 0.0) bad = 1;
            iv_s[tid][0] = Vk[3] / det;
            iv_s[tid][1] = -2.0 * v12 / det;
            iv_s[tid][2] = Vk[0] / det;
            sc_s[tid] = w_s[tid] / sqrt(tpd * det);
            maxd_s[tid] = log(approx * sqrt(tpd * det)) / -0.5;
        }
        __syncthreads();
        if (bad) break;   // the same value in every thread
        const double psky = psky_s;
        double acc[kM];
#pragma unroll
        for (int v = 0; v < kM; v++) acc[v] = 0.0;
        int ix = ix0, iy = iy0;
        for (int i = tid; i < npix; i += kEmThreads) {
            const double x = (double)(x0 + ix), y = (double)(y0 + iy);
            ix += step_x;
            iy += step_y;
            if (ix >= nx) {
                ix -= nx;
                iy++;
            }
            const double d = im[i];
            if (d <= 0.0) {
                acc[6 * K] += fabs(d);
                continue;
            }
            double z[K];
            double zsum = 0.0;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const double dx = x - mu_s[k][0], dy = y - mu_s[k][1];
                const double dsq = iv_s[k][0] * dx * dx + iv_s[k][1] * dx * dy +
                                   iv_s[k][2] * dy * dy;
                z[k] = dsq >= maxd_s[k] ? 0.0 : sc_s[k] * exp(-0.5 * dsq);
                zsum += z[k];
            }
            if (zsum == 0.0) {
                acc[6 * K] += d;
                continue;
            }
            zsum += psky;
            acc[6 * K] += d * (psky / zsum);
#pragma unroll
            for (int k = 0; k < K; k++) {
                const double wi = d * z[k] / zsum;
                const double dx = x - mu_s[k][0], dy = y - mu_s[k][1];
                acc[6 * k + 0] += wi;
                acc[6 * k + 1] += wi * x;
                acc[6 * k + 2] += wi * y;
                acc[6 * k + 3] += wi * dx * dx;
                acc[6 * k + 4] += wi * dx * dy;
                acc[6 * k + 5] += wi * dy * dy;
            }
        }
#pragma unroll
        for (int v = 0; v < kM; v++) {
            double a = acc[v];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (lane == 0) red[warp][v] = a;
        }
        __syncthreads();
        if (tid < K) {
            double m[6];
#pragma unroll
            for (int q = 0; q < 6; q++) {
                double t = 0.0;
                for (int w2 = 0; w2 < kWarps; w2++) t += red[w2][6 * tid + q];
                m[q] = t;
            }
            const double ws = m[0];
            mu_s[tid][0] = m[1] / ws;
            mu_s[tid][1] = m[2] / ws;
            const double den = ws + alpha;
            v_s[tid][0] = (alpha + m[3]) / den;
            v_s[tid][1] = m[4] / den;
            v_s[tid][2] = v_s[tid][1];
            v_s[tid][3] = (alpha + m[5]) / den;
            w_s[tid] = ws;
        }
        if (tid == 0) {
            double t = 0.0;
            for (int w2 = 0; w2 < kWarps; w2++) t += red[w2][6 * K];
            psky_s = t / (double)npix;
        }
        __syncthreads();
    }
    if (tid < K) {
        A[tid] = w_s[tid];
        Mu[2 * tid] = mu_s[tid][0];
        Mu[2 * tid + 1] = mu_s[tid][1];
#pragma unroll
        for (int d = 0; d < 4; d++) V[4 * tid + d] = v_s[tid][d];
    }
    if (tid == 0) {
        if (skyamp) skyamp[s] = psky_s;
        if (status) status[s] = bad;
    }
}

template <int K>
int launch_sky(const double* img, int n, int ny, int nx, const int32_t* xy0, double* amp,
               double* mean, double* var, double alpha, int steps, double approx, double* sky,
               int32_t* status, cudaStream_t s) {
    em_fit_sky_kernel<K><<<n, kEmThreads, 0, s>>>(img, n, ny, nx, xy0, amp, mean, var, alpha,
                                                  steps, approx, sky, status);
    return cudaGetLastError() == cudaSuccess ? TB_OK : TB_ERR_LAUNCH;
}

template <int K>
int launch(const double* img, int n, int ny, int nx, const int32_t* xy0, double* amp,
           double* mean, double* var, double alpha, int steps, int32_t* status,
           cudaStream_t s) {
    em_fit_kernel<K><<<n, kEmThreads, 0, s>>>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps,
                                              status);
    return cudaGetLastError() == cudaSuccess ? TB_OK : TB_ERR_LAUNCH;
}

}  // namespace

extern "C" int tb_em_fit_2d(const double* img, int32_t n, int32_t ny, int32_t nx,
                            const int32_t* xy0, double* amp, double* mean, double* var,
                            int32_t K, double alpha, int32_t steps, int32_t* status,
                            void* stream) {
    if (n < 0 || ny < 1 || nx < 1 || (int64_t)ny * nx > (1 << 24) || K < 1 ||
        K > TB_EM_MAX_K || steps < 0)
        return TB_ERR_ARG;
    if (n == 0) return TB_OK;
    if (!img || !amp || !mean || !var) return TB_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    switch (K) {
        case 1: return launch<1>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, status, s);
        case 2: return launch<2>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, status, s);
        case 3: return launch<3>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, status, s);
        case 4: return launch<4>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, status, s);
        case 5: return launch<5>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, status, s);
        case 6: return launch<6>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, status, s);
        case 7: return launch<7>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, status, s);
        default: return launch<8>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, status, s);
    }
}

extern "C" int tb_em_fit_2d_sky(const double* img, int32_t n, int32_t ny, int32_t nx,
                                const int32_t* xy0, double* amp, double* mean, double* var,
                                int32_t K, double alpha, int32_t steps, double approx,
                                double* skyamp, int32_t* status, void* stream) {
    if (n < 0 || ny < 1 || nx < 1 || (int64_t)ny * nx > (1 << 24) || K < 1 ||
        K > TB_EM_MAX_K || steps < 0 || !(approx > 0.0))
        return TB_ERR_ARG;
    if (n == 0) return TB_OK;
    if (!img || !amp || !mean || !var) return TB_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    switch (K) {
        case 1: return launch_sky<1>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, approx, skyamp, status, s);
        case 2: return launch_sky<2>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, approx, skyamp, status, s);
        case 3: return launch_sky<3>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, approx, skyamp, status, s);
        case 4: return launch_sky<4>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, approx, skyamp, status, s);
        case 5: return launch_sky<5>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, approx, skyamp, status, s);
        case 6: return launch_sky<6>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, approx, skyamp, status, s);
        case 7: return launch_sky<7>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, approx, skyamp, status, s);
        default: return launch_sky<8>(img, n, ny, nx, xy0, amp, mean, var, alpha, steps, approx, skyamp, status, s);
    }
}
