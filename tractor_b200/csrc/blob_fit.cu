// Batched blob fitting (sm_100a): Levenberg-Marquardt on many independent
// blobs at once, each blob a few galaxies seen in several bands.  It is the
// batched form of Tractor.optimize / optimize_loop with LsqrOptimizer
// (tractor/lsqr_optimizer.py:280-326) over getDerivs + getChiImage
// (tractor/engine.py:279-339, 455-473), with ConstrainedOptimizer's bounds and
// maximum steps (tractor/constrained_optimizer.py:12-159).
//
// One iteration:
//   tb_fit_prep  one warp per source: the profile mixture (exp / deV /
//                Sersic) and its derivative with respect to the Sersic index,
//                the pixel-space shape factor M = T T^T and its derivatives
//                with respect to (log r_e, ee1, ee2) -- FP64 central
//                differences of the exact FP64 maps (sersic.py:288-342,
//                ellipses.py:165-263);
//   tb_fit_pass  persistent CTAs take units of a few 32 x 8 pixel tiles of a
//                (blob, band) image: the model (every source's PSF-convolved
//                mixture, as galaxy.py:307-326) and the analytic derivative
//                columns (position, flux, shape, index), weighted by inverr;
//                A^T A, A^T r and r^T r into the unit's own slice (no atomics);
//   tb_fit_step  sums the slices (many CTAs per blob), then one CTA per blob:
//                accepts or rejects the trial parameters, solves the
//                Marquardt-damped normal equations (FP64 LDL^T, one refinement
//                step), limits the step (bounds, maximum steps: scaled as a
//                whole, or, for a blob slow to converge, minimised within them)
//                and writes the next trial parameters.
#include "ldl.cuh"
#include "profile_eval.cuh"

namespace {

constexpr int kPrepThreads = 128;      // 4 sources per block
constexpr int kMaxGalK = 10;           // galaxy components of one source
constexpr int kThreads = 256;          // pass CTA = one 32 x 8 tile, one pixel per thread
constexpr int kTileW = 32;
constexpr int kTileH = 8;
constexpr int kCols = 7;               // columns per (source, band): x y flux logre ee1 ee2 n

constexpr int kCompStride = kMaxGalK * TB_FIT_MAX_PSF;   // component slots per (source, band)

// Per-source summary written by tb_fit_prep.
struct SrcTab {
    double flux[TB_FIT_MAX_BANDS];
    double M[3];                   // T T^T (xx, xy, yy)
    double dM[3][3];               // d(T T^T) / d(logre, ee1, ee2)
    int32_t K[TB_FIT_MAX_BANDS];   // components in each band (galaxy x PSF)
    int32_t ok;
};

// One PSF-convolved component of a (source, band), written by tb_fit_prep in
// both precisions (FP32 for tb_fit_pass, FP64 for tb_fit_refine and
// tb_fit_model_vjp).  The mean stays FP64 (absolute pixels); a pass makes it
// tile-relative.  The shape derivative of component k is dC_k = v_k dM (dM
// per source), the index derivative dC_k = dv_k M: the passes accumulate per
// source the moments sum_k val_k v_k (u u^T - C_k^-1) and sum_k val_k dv_k
// (u u^T - C_k^-1), u = C_k^-1 (pixel - mean), over components and apply dM
// / M once per source and pixel.
template <class T>
struct __align__(16) FitC {
    double mx, my;
    T i00, i01, i11;          // C^-1
    T s, sn;                  // a / (2 pi sqrt det), d a / d n / (2 pi sqrt det)
    T v, dv;                  // the galaxy component's variance and d/dn
    T pad;
};

// ---------------------------------------------------------------------------
// prep
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(kPrepThreads)
fit_prep_kernel(const tb_fit_source* __restrict__ srcs, int n, const double* __restrict__ params,
                int n_bands, const tb_fit_unit* __restrict__ units, int n_units,
                tb_profile_tables Tg, double cd0, double cd1, double cd2, double cd3,
                SrcTab* __restrict__ tab, FitC<float>* __restrict__ comps,
                FitC<double>* __restrict__ comps64, const tb_fit_state* __restrict__ state) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const tb_profile_tables T = tb::stage_tables(Tg, smem_raw);
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * (kPrepThreads / 32) + (threadIdx.x >> 5);
    if (i >= n) return;
    const tb_fit_source s = srcs[i];
    // a converged or stopped blob's tables stay as they are (nothing reads them)
    if (state && s.blob >= 0 && (int64_t)(s.blob + 1) * n_bands <= n_units &&
        state[s.blob].status != 0)
        return;
    const double* p = params + (int64_t)i * TB_FIT_NPAR;
    const double cd[4] = {cd0, cd1, cd2, cd3};
    int ok = s.blob >= 0 && (int64_t)(s.blob + 1) * n_bands <= n_units;
    double a = 0.0, v = 0.0, da = 0.0, dv = 0.0;
    int K = 0;
    if (s.profile == TB_PROFILE_SERSIC) {
        K = tb::sersic_with_slope(T, p[8], lane, kMaxGalK, a, v, da, dv);
        if (K < 0) {
            ok = 0;
            K = 0;
        } else {
            // components sorted by variance (sersic.py:338-341); the sort is
            // a permutation of lanes, kept fixed for the derivative
            const int rank = tb::variance_rank(v, K, lane);
            double a2 = 0.0, v2 = 0.0, da2 = 0.0, dv2 = 0.0;
            for (int j = 0; j < K; j++) {
                const int rj = __shfl_sync(0xffffffffu, rank, j);
                const double aj = __shfl_sync(0xffffffffu, a, j);
                const double vj = __shfl_sync(0xffffffffu, v, j);
                const double daj = __shfl_sync(0xffffffffu, da, j);
                const double dvj = __shfl_sync(0xffffffffu, dv, j);
                if (rj == lane) { a2 = aj; v2 = vj; da2 = daj; dv2 = dvj; }
            }
            a = a2; v = v2; da = da2; dv = dv2;
        }
    } else if (s.profile == TB_PROFILE_EXP || s.profile == TB_PROFILE_DEV) {
        K = tb::warp_profile(T, s.profile, 0.0, lane, kMaxGalK, a, v);
        if (K < 0) { ok = 0; K = 0; }
    } else if (s.profile == TB_PROFILE_POINT) {
        K = 1;
        a = lane == 0 ? 1.0 : 0.0;
    } else {
        ok = 0;
    }
    double M[3] = {0.0, 0.0, 0.0};
    double dM[3][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
    if (s.profile != TB_PROFILE_POINT) {
        double re;
        tb::shape_with_slopes(cd, TB_SHAPE_ELLIPSE_ESOFT, p[5], p[6], p[7], lane, M, dM, re);
    }
    bool fin = isfinite(p[0]) && isfinite(p[1]);
    for (int q = 0; q < 3; q++) fin = fin && isfinite(M[q]);
    ok = ok && fin;
    // components per band: PSF component p (outer) x galaxy component gi
    // (inner), mixture_profiles.py:158-172
    int Kb[TB_FIT_MAX_BANDS] = {0, 0, 0};
    for (int bd = 0; bd < n_bands; bd++) {
        ok = __all_sync(0xffffffffu, ok);   // a lane may have met a bad component
        const tb_fit_unit* u = ok ? units + (int64_t)s.blob * n_bands + bd : units;
        const int Kp = u->psf_K;
        if (Kp < 1 || Kp > TB_FIT_MAX_PSF) ok = 0;
        const int Kt = ok ? K * Kp : 0;
        Kb[bd] = Kt;
        for (int k0 = 0; k0 < Kt; k0 += 32) {
            const int k = k0 + lane;
            const int gi = (Kt > 0 && k < Kt) ? k % K : 0;
            const int pp = (Kt > 0 && k < Kt) ? k / K : 0;
            const double ag = __shfl_sync(0xffffffffu, a, gi);
            const double vg = __shfl_sync(0xffffffffu, v, gi);
            const double dag = __shfl_sync(0xffffffffu, da, gi);
            const double dvg = __shfl_sync(0xffffffffu, dv, gi);
            if (k >= Kt) continue;
            const double C00 = vg * M[0] + u->psf_var[4 * pp];
            const double C01 = vg * M[1] + 0.5 * (u->psf_var[4 * pp + 1] + u->psf_var[4 * pp + 2]);
            const double C11 = vg * M[2] + u->psf_var[4 * pp + 3];
            const double det = C00 * C11 - C01 * C01;
            const double i00 = C11 / det, i01 = -C01 / det, i11 = C00 / det;
            const double norm = 1.0 / (2.0 * TB_PI * sqrt(det));
            const bool good = det > 0.0 && isfinite(norm);
            if (!good) ok = 0;
            FitC<double> c;
            c.mx = p[0] + u->psf_mean[2 * pp];
            c.my = p[1] + u->psf_mean[2 * pp + 1];
            c.i00 = i00;
            c.i01 = i01;
            c.i11 = i11;
            c.s = ag * u->psf_amp[pp] * norm;
            c.sn = dag * u->psf_amp[pp] * norm;
            c.v = vg;
            c.dv = dvg;
            c.pad = 0.0;
            const int64_t at = ((int64_t)i * n_bands + bd) * kCompStride + k;
            comps64[at] = c;
            comps[at] = FitC<float>{c.mx, c.my, (float)i00, (float)i01, (float)i11, (float)c.s,
                                    (float)c.sn, (float)vg, (float)dvg, 0.f};
        }
    }
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0) {
        SrcTab t;
        for (int bd = 0; bd < TB_FIT_MAX_BANDS; bd++) {
            t.flux[bd] = bd < n_bands ? p[2 + bd] : 0.0;
            t.K[bd] = bd < n_bands ? Kb[bd] : 0;
        }
        t.ok = ok;
        for (int q = 0; q < 3; q++) {
            t.M[q] = M[q];
            for (int j = 0; j < 3; j++) t.dM[j][q] = dM[j][q];
        }
        tab[i] = t;
    }
}

// ---------------------------------------------------------------------------
// pass (tb_fit_pass, FP32) and refinement pass (tb_fit_refine and
// tb_fit_model_vjp, FP64): one kernel, compiled for both precisions.
//
// Near the optimum the gradient is a sum of terms that cancel, FP32 chi^2
// cannot verify gains below ~1e-4, and an FP32 A^T A (FP32 columns: the index
// column is a difference of nearly equal sums) is too inexact for the steps
// of an ill-conditioned blob to converge; the final iterations of a fit take
// all of them in FP64.
//
// Bound: issue in the component loop (FP64: 31 operations per pixel and
// component: exponent 3, exponential 10, value and C^-1 u 5, moments 13).  So
// each warp stages, per pixel row, only the components that reach its row of
// a source's mask; the trace terms are folded into the second moments; and
// the products A^T A, A^T r go to the FP64 tensor core (mma m8n8k4),
// accumulated in two registers per 8 x 8 block over a whole run of tiles with
// the same sources: no block barrier inside a run, no reduction per pixel.
// 300 blobs (192-512 px, 3 bands): first FP32 pass 2.5 -> 1.7 ms, first FP64
// pass about 10 -> 3.1 ms; FP32 is latency-bound (2.3 instructions per cycle
// and SM, FMA pipe 31 %, LSU 35 %, FP64 tensor 11 %), FP64 at 42 % of its pipe.
// Model + gradient of 100 blobs 3.4 -> 1.8 ms of kernels.
// ---------------------------------------------------------------------------
constexpr int kWarps = kThreads / 32;
constexpr int kSlots = 4;              // sources whose columns a warp holds at once
constexpr int kLd = 36;                // elements per column row (see frag)
constexpr int kXs = 8 * kLd;           // elements per source: 7 columns and r

// What a launch computes: the normal equations and chi^2 of the running
// blobs; chi^2 of the tiles no mask reaches (FP32); the model (FP64); the
// columns contracted with an upstream gradient (FP64).
enum Mode { kEquations, kConstant, kModel, kVjp };

// One source of the unit, copied to shared memory once per unit.
template <class T>
struct UnitSrc {
    int32_t x0, y0, x1, y1;   // mask [x0, x1) x [y0, y1), image pixels; an empty mask is all 0
    int32_t K, profile;       // components (galaxy x PSF) in the unit's band
    T counts;                 // flux in the unit's band
    T M[3];                   // T T^T (xx, xy, yy)
    T dM[3][3];               // its shape derivatives
};

// One component staged for one pixel row of a tile (dy = row - mean y) by
// the warp that owns the row: tile-relative mean x, exponent
// e(dx) = h00 dx^2 + bx dx + c0 in log2 units, C^-1 u = (i00 dx + uxy,
// i01 dx + uyy).
template <class T>
struct __align__(16) RowC {
    T mx, h00, bx, c0;
    T i00, i01, uxy, uyy;
    T i11, s, sn, v;
    T dv, pad[sizeof(T) == 8 ? 1 : 3];
};

template <class T>
struct PassSmem {
    UnitSrc<T> us[TB_FIT_MAX_SRC];
    RowC<T> wc[kWarps][32];                 // a warp's staged components
    T X[kWarps][kSlots * kXs];              // a warp's weighted columns and residuals
    double exp_tab[tb::kExpTab];
    double red[kWarps];
    int64_t slot;
    int skip;
};

__device__ __forceinline__ float exp2_of(float e, const double*) { return tb::ex2(e); }
__device__ __forceinline__ double exp2_of(double e, const double* tab) {
    return tb::exp2_tab(e, tab);
}

// Position of the (q+1)-th set bit of m (q < popc(m)).
__device__ __forceinline__ int nth_bit(unsigned m, int q) {
    for (int i = 0; i < q; i++) m &= m - 1u;
    return __ffs(m) - 1;
}

// Parameter slot of column i (x y flux(band) logre ee1 ee2 n) of source sI;
// -1 where the profile has no such parameter.
__device__ __forceinline__ int param_slot(int sI, int profile, int band, int i) {
    if (i >= 3 && profile == TB_PROFILE_POINT) return -1;
    if (i == 6 && profile != TB_PROFILE_SERSIC) return -1;
    const int base = sI * TB_FIT_NPAR;
    return i < 2 ? base + i : i == 2 ? base + 2 + band : base + 2 + i;
}

// Stages, by one warp, those of the components cs[k0 .. min(k0 + 32, K)) that
// reach pixels [xa, xb] (tile-relative, inclusive) of row py of the tile at
// column ox into wc[0 ..), in their order; returns how many.  Along a row the
// exponent is a concave quadratic in dx whose maximum over the segment is at
// its vertex clamped to the segment: a component whose Mahalanobis^2 stays
// above 100 there (FP32, with a margin of 2) is exactly zero at every pixel
// (exponents below -50 count as 0) and is left out.  Components with
// non-finite coefficients are always staged.
template <class T>
__device__ __forceinline__ int stage_row(RowC<T>* wc, const FitC<T>* __restrict__ cs, int k0,
                                         int K, int ox, int py, int xa, int xb) {
    const int lane = threadIdx.x & 31;
    const int k = k0 + lane;
    bool keep = false;
    T mx = 0, dy = 0, i00 = 0, i01 = 0, i11 = 0;
    __syncwarp();   // the warp's previous components are no longer read
    if (k < K) {
        const FitC<T>& c = cs[k];
        mx = (T)(c.mx - (double)ox);
        dy = (T)((double)py - c.my);
        i00 = c.i00;
        i01 = c.i01;
        i11 = c.i11;
        const float a = (float)i00, bb = (float)(i01 * dy), cc = (float)(i11 * dy * dy);
        const float lo = (float)((T)xa - mx), hi = (float)((T)xb - mx);
        const bool ok = isfinite(a) && isfinite(bb) && isfinite(cc) && isfinite(lo) && a > 0.f;
        const float dx = fminf(fmaxf(__fdividef(-bb, a), lo), hi);
        keep = !ok || !(fmaf(dx, fmaf(a, dx, 2.f * bb), cc) > 102.f);
    }
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (keep) {
        const FitC<T>& c = cs[k];
        RowC<T>& f = wc[__popc(bal & ((1u << lane) - 1u))];
        f.mx = mx;
        f.h00 = (T)(-0.5 * TB_LOG2E) * i00;
        f.bx = (T)-TB_LOG2E * i01 * dy;
        f.c0 = (T)(-0.5 * TB_LOG2E) * i11 * dy * dy;
        f.i00 = i00;
        f.i01 = i01;
        f.uxy = i01 * dy;
        f.uyy = i11 * dy;
        f.i11 = i11;
        f.s = c.s;
        f.sn = c.sn;
        f.v = c.v;
        f.dv = c.dv;
    }
    __syncwarp();   // staged components visible to the whole warp
    return __popc(bal);
}

// Source S's model at this thread's pixel (column lane of the tile at ox,
// row py): counts x its unit-flux mixture; 0 outside its mask.  Called by
// whole warps.
template <class T>
__device__ __forceinline__ T source_model(PassSmem<T>& sm, const UnitSrc<T>& S,
                                          const FitC<T>* __restrict__ cs, int ox, int py) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int xa = max(S.x0 - ox, 0), xb = min(S.x1 - ox, kTileW);
    if (py < S.y0 || py >= S.y1 || xa >= xb) return 0;   // warp-uniform
    RowC<T>* wc = sm.wc[warp];
    T val = 0;
    for (int k0 = 0; k0 < S.K; k0 += 32) {
        const int n = stage_row<T>(wc, cs, k0, S.K, ox, py, xa, xb - 1);
#pragma unroll 2
        for (int g = 0; g < n; g++) {
            const RowC<T>& c = wc[g];
            const T dx = (T)lane - c.mx;
            const T e = fma(dx, fma(c.h00, dx, c.bx), c.c0);
            const T E = exp2_of(e, sm.exp_tab);
            val = fma(e >= (T)(-50.0 * TB_LOG2E) ? E : (T)0, c.s, val);
        }
    }
    return lane >= xa && lane < xb ? S.counts * val : (T)0;
}

// Source S's seven derivative columns, times w, at this thread's pixel of
// row py into X[0 .. 7)[lane] (0 outside its mask); returns its model there.
// Per component the moments of u that d/d(mean, C, amplitude) produce,
// d/dC = 1/2 (u u^T - C^-1), combined once per source with dM (shape) and M
// (index).  Called by whole warps; no block barrier.
template <class T>
__device__ __forceinline__ T source_columns(PassSmem<T>& sm, const UnitSrc<T>& S,
                                            const FitC<T>* __restrict__ cs, int ox, int py, T w,
                                            T* X) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int xa = max(S.x0 - ox, 0), xb = min(S.x1 - ox, kTileW);
    T S0 = 0, Sx = 0, Sy = 0, Axx = 0, Axy = 0, Ayy = 0, Dxx = 0, Dxy = 0, Dyy = 0, Sn = 0;
    const bool row = py >= S.y0 && py < S.y1 && xa < xb;   // warp-uniform
    if (row) {
        RowC<T>* wc = sm.wc[warp];
        for (int k0 = 0; k0 < S.K; k0 += 32) {
            const int n = stage_row<T>(wc, cs, k0, S.K, ox, py, xa, xb - 1);
#pragma unroll 2
            for (int g = 0; g < n; g++) {
                const RowC<T>& c = wc[g];
                const T dx = (T)lane - c.mx;
                const T e = fma(dx, fma(c.h00, dx, c.bx), c.c0);
                T E = exp2_of(e, sm.exp_tab);
                if (!(e >= (T)(-50.0 * TB_LOG2E))) E = 0;
                const T ux = fma(c.i00, dx, c.uxy), uy = fma(c.i01, dx, c.uyy);
                const T val = c.s * E;
                S0 += val;
                Sx = fma(val, ux, Sx);
                Sy = fma(val, uy, Sy);
                const T pxx = fma(ux, ux, -c.i00), pxy = fma(ux, uy, -c.i01),
                        pyy = fma(uy, uy, -c.i11);
                const T vv = val * c.v, vd = val * c.dv;
                Axx = fma(vv, pxx, Axx);
                Axy = fma(vv, pxy, Axy);
                Ayy = fma(vv, pyy, Ayy);
                Dxx = fma(vd, pxx, Dxx);
                Dxy = fma(vd, pxy, Dxy);
                Dyy = fma(vd, pyy, Dyy);
                Sn = fma(c.sn, E, Sn);
            }
        }
    }
    const bool in = row && lane >= xa && lane < xb;
    const T cn = in ? S.counts : (T)0;
    const T cw = cn * w, h = (T)0.5 * cw;
    X[lane] = cw * Sx;
    X[kLd + lane] = cw * Sy;
    X[2 * kLd + lane] = in ? w * S0 : (T)0;
#pragma unroll
    for (int j = 0; j < 3; j++)
        X[(3 + j) * kLd + lane] =
            h * (S.dM[j][0] * Axx + (T)2 * S.dM[j][1] * Axy + S.dM[j][2] * Ayy);
    X[6 * kLd + lane] =
        h * (S.M[0] * Dxx + (T)2 * S.M[1] * Dxy + S.M[2] * Dyy) + cw * Sn;
    return cn * S0;
}

// A^T A and A^T r are contractions over pixels: with X_s the 8 x 32 matrix of
// source s's seven weighted columns and the residual over a warp's 32
// pixels, X_a X_b^T is a chain of eight FP64 m8n8k4 tensor-core products
// (FP32 columns are widened first).  Their A and B fragments are the same
// element per lane, X[lane / 4][4 step + lane % 4]; the row stride of 36
// elements puts the lanes of a (half, FP64) warp in different banks.
template <class T>
__device__ __forceinline__ double frag(const T* X, int step) {
    const int lane = threadIdx.x & 31;
    return (double)X[(lane >> 2) * kLd + 4 * step + (lane & 3)];
}

// Where a unit adds its products.  kVjp: g alone, by parameter slot (P per
// slice).  kEquations: compact slices that hold only the m sources whose masks
// meet the unit (`mask`), seven columns each: a (7 m)^2 block of H (upper
// triangle) and 7 m of g, so that a unit of a few tiles in a large blob neither
// clears nor passes on a P x P block; the mask itself, and the band above it,
// go to the slice's last g slot (7 m < 9 m <= P).
struct SliceOut {
    double *H, *g;
    unsigned mask;
    int ld;                   // 7 m
    int P, band;
};

__device__ __forceinline__ int compact_row(unsigned mask, int src) {
    return kCols * __popc(mask & ((1u << src) - 1u));
}

// The warps' NB 8 x 8 blocks summed (in warp order) and added to their
// destinations: element (i, j) of block q, between sources sa(q) <= sb(q)
// (-1: no such source), to H (upper triangle) or, in the residual's column,
// to g.  The blocks pass through the component staging area, a round at a
// time.  Called by the whole block.
template <class T, int NB, class SA, class SB>
__device__ __forceinline__ void flush(PassSmem<T>& sm, const double (&c)[NB][2], SA sa, SB sb,
                                      const SliceOut& o) {
    constexpr int kRound = (int)(32 * sizeof(RowC<T>) / (64 * sizeof(double)));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncwarp();   // the warp's staged components are read
#pragma unroll
    for (int q0 = 0; q0 < NB; q0 += kRound) {
#pragma unroll
        for (int q = q0; q < NB && q < q0 + kRound; q++)
            reinterpret_cast<double2*>(sm.wc[warp])[(q - q0) * 32 + lane] =
                make_double2(c[q][0], c[q][1]);
        __syncthreads();
        const int nb = NB - q0 < kRound ? NB - q0 : kRound;
        for (int e = threadIdx.x; e < nb * 64; e += kThreads) {
            const int q = q0 + (e >> 6), i = (e >> 3) & 7, j = e & 7;
            const int a = sa(q), b = sb(q);
            if (a < 0 || b < 0 || i == 7 || (j == 7 ? a != b : !o.H || (a == b && j < i))) continue;
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < kWarps; w++) s += reinterpret_cast<const double*>(sm.wc[w])[e];
            if (o.H) {
                const int di = compact_row(o.mask, a) + i;
                if (j == 7) o.g[di] += s;
                else o.H[di * o.ld + compact_row(o.mask, b) + j] += s;
            } else {
                const int di = param_slot(a, sm.us[a].profile, o.band, i);
                if (di >= 0) o.g[di] += s;
            }
        }
        __syncthreads();
    }
}

// Block q of R sources: q < R a source's own block, then the pairs (0, 1),
// (0, 2), .. (R - 2, R - 1).
__host__ __device__ constexpr int pair_a(int q, int R) {
    if (q < R) return q;
    int a = 0, n = q - R;
    while (n >= R - 1 - a) { n -= R - 1 - a; a++; }
    return a;
}
__host__ __device__ constexpr int pair_b(int q, int R) {
    if (q < R) return q;
    int a = 0, n = q - R;
    while (n >= R - 1 - a) { n -= R - 1 - a; a++; }
    return a + 1 + n;
}

// The unit a CTA works on.
template <class T>
struct PassUnit {
    const FitC<T>* comps;     // its band of source s: comps + s * cstride
    int64_t cstride, pix_off;
    const int32_t* tiles;
    const float* data;        // data, or (VJP) the upstream gradient
    const float* inverr;      // null: no weights (VJP)
    int W, Hh;
    SliceOut out;
};

// This thread's pixel (0 outside the image): its value and weight.
template <class T>
__device__ __forceinline__ void load_pixel(const PassUnit<T>& u, int px, int py, T& d, T& w) {
    d = w = 0;
    if (px < u.W && py < u.Hh) {
        const int64_t pix = u.pix_off + (int64_t)py * u.W + px;
        d = (T)u.data[pix];
        w = u.inverr ? (T)u.inverr[pix] : (T)1;
    }
}

// Tiles [t0, t1), all met by exactly the R sources `hit`: each warp adds its
// rows' products into register blocks without a block barrier, then one
// flush.  kResid: r = (data - model) inverr, every pair's block, chi^2;
// otherwise (one source) r = data.
template <class T, int R, bool kResid>
__device__ void run_tiles(PassSmem<T>& sm, const PassUnit<T>& u, unsigned hit, int t0, int t1,
                          double& chi2) {
    constexpr int NB = R * (R + 1) / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T* X = sm.X[warp];
    double c[NB][2];
#pragma unroll
    for (int q = 0; q < NB; q++) c[q][0] = c[q][1] = 0.0;
    for (int t = t0; t < t1; t++) {
        const int ox = (u.tiles[t] & 0x3ff) * kTileW;
        const int py = ((u.tiles[t] >> 10) & 0x3ff) * kTileH + warp;
        T d, w;
        load_pixel(u, ox + lane, py, d, w);
        T m = 0;
        bool any = false;
        unsigned hm = hit;
        __syncwarp();   // the previous tile's fragments are read
#pragma unroll 1
        for (int s = 0; s < R; s++, hm &= hm - 1) {
            const int sI = __ffs(hm) - 1;
            const UnitSrc<T>& S = sm.us[sI];
            any = any || (py >= S.y0 && py < S.y1);
            m += source_columns<T>(sm, S, u.comps + sI * u.cstride, ox, py, w, X + s * kXs);
        }
        const T r = kResid ? (d - m) * w : d;
        if (kResid) chi2 += (double)(r * r);
        if (!any) continue;   // warp-uniform: every column is 0 in this row
#pragma unroll
        for (int s = 0; s < R; s++) X[s * kXs + 7 * kLd + lane] = r;
        __syncwarp();
#pragma unroll
        for (int step = 0; step < 8; step++) {
            double f[R];
#pragma unroll
            for (int s = 0; s < R; s++) f[s] = frag(X + s * kXs, step);
#pragma unroll
            for (int q = 0; q < NB; q++) tb::mma884(c[q], f[pair_a(q, R)], f[pair_b(q, R)]);
        }
    }
    auto src = [&](int i) { return nth_bit(hit, i); };
    flush<T, NB>(sm, c, [&](int q) { return src(pair_a(q, R)); },
                 [&](int q) { return src(pair_b(q, R)); }, u.out);
}

// A tile that more than kSlots sources meet: the model first, then groups of
// three sources (their own and mutual blocks), each followed by its blocks
// with every later source, whose columns are evaluated again.
template <class T>
__device__ void crowded_tile(PassSmem<T>& sm, const PassUnit<T>& u, unsigned hit, int code,
                             double& chi2) {
    constexpr int kG3 = kSlots - 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int R = __popc(hit);
    T* X = sm.X[warp];
    const int ox = (code & 0x3ff) * kTileW, py = ((code >> 10) & 0x3ff) * kTileH + warp;
    T d, w;
    load_pixel(u, ox + lane, py, d, w);
    T m = 0;
    for (unsigned hm = hit; hm; hm &= hm - 1) {
        const int sI = __ffs(hm) - 1;
        m += source_model<T>(sm, sm.us[sI], u.comps + sI * u.cstride, ox, py);
    }
    const T r = (d - m) * w;
    chi2 += (double)(r * r);
    for (int q0 = 0; q0 < R; q0 += kG3) {
        __syncwarp();
        for (int s = 0; s < kG3; s++) {
            T* Xs = X + s * kXs;
            if (q0 + s < R) {
                const int sI = nth_bit(hit, q0 + s);
                source_columns<T>(sm, sm.us[sI], u.comps + sI * u.cstride, ox, py, w, Xs);
            } else {
#pragma unroll
                for (int c = 0; c < 7; c++) Xs[c * kLd + lane] = 0;
            }
            Xs[7 * kLd + lane] = r;
        }
        __syncwarp();
        auto src = [&](int i) { return q0 + i < R ? nth_bit(hit, q0 + i) : -1; };
        {
            constexpr int NB = kG3 * (kG3 + 1) / 2;
            double c[NB][2];
#pragma unroll
            for (int q = 0; q < NB; q++) c[q][0] = c[q][1] = 0.0;
#pragma unroll
            for (int step = 0; step < 8; step++) {
                double f[kG3];
#pragma unroll
                for (int s = 0; s < kG3; s++) f[s] = frag(X + s * kXs, step);
#pragma unroll
                for (int q = 0; q < NB; q++) tb::mma884(c[q], f[pair_a(q, kG3)], f[pair_b(q, kG3)]);
            }
            flush<T, NB>(sm, c, [&](int q) { return src(pair_a(q, kG3)); },
                         [&](int q) { return src(pair_b(q, kG3)); }, u.out);
        }
        for (int i = q0 + kG3; i < R; i++) {
            const int sI = nth_bit(hit, i);
            T* Xb = X + kG3 * kXs;
            __syncwarp();
            source_columns<T>(sm, sm.us[sI], u.comps + sI * u.cstride, ox, py, w, Xb);
            Xb[7 * kLd + lane] = r;
            __syncwarp();
            double c[kG3][2];
#pragma unroll
            for (int q = 0; q < kG3; q++) c[q][0] = c[q][1] = 0.0;
#pragma unroll
            for (int step = 0; step < 8; step++) {
                const double fb = frag(Xb, step);
#pragma unroll
                for (int q = 0; q < kG3; q++) tb::mma884(c[q], frag(X + q * kXs, step), fb);
            }
            flush<T, kG3>(sm, c, src, [&](int) { return sI; }, u.out);
        }
    }
}

// Two CTAs per SM: 128 registers hold the ten blocks of four sources without
// spills in FP32 (three CTAs at 80 registers measured 8 % slower, four 17 %).
template <class T>
__global__ void __launch_bounds__(kThreads, 2)
fit_pass_kernel(const tb_fit_unit* __restrict__ units, const int32_t* __restrict__ order,
                int n_units, const tb_fit_blob* __restrict__ blobs,
                const tb_fit_source* __restrict__ srcs, const SrcTab* __restrict__ tab,
                const FitC<T>* __restrict__ gcomps, const float* __restrict__ data,
                const float* __restrict__ inverr, double* __restrict__ hbuf,
                double* __restrict__ gbuf, double* __restrict__ chi2_part,
                const tb_fit_state* __restrict__ state, int n_bands,
                const int32_t* __restrict__ tiles, double* chi2_const, Mode mode,
                float* __restrict__ model_out, int32_t* counter, tb_status* st) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PassSmem<T>& sm = *reinterpret_cast<PassSmem<T>*>(smem_raw);
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    if (sizeof(T) == 8) tb::exp2_tab_init(sm.exp_tab);   // read after next_unit's barriers
    for (;;) {
        const int64_t oi = tb::next_unit(counter, &sm.slot);   // barriers on both sides
        if (oi >= n_units) break;
        const int ui = order[oi];
        if (ui < 0 || ui >= n_units) {
            if (tid == 0) tb::report(st, TB_STATUS_BAD_ITEM, (int)oi, ui);
            continue;
        }
        const tb_fit_unit& u = units[ui];
        const tb_fit_blob b = blobs[u.blob];
        if (mode == kEquations && state[u.blob].status != 0) continue;   // converged or stopped
        const int P = b.P;
        const int nsrc = b.n_src;
        // checks, and the unit's sources into shared memory (lane = source);
        // a blob without sources is taken as any other (its slices hold nothing)
        if (warp == 0) {
            const bool unit_bad = nsrc < 0 || nsrc > TB_FIT_MAX_SRC || P != nsrc * TB_FIT_NPAR ||
                                  u.psf_K < 1 || u.psf_K > TB_FIT_MAX_PSF || u.band < 0 ||
                                  u.band >= n_bands || u.slice < 0 || u.slice >= b.n_slices ||
                                  u.t0 < 0 || u.t1 < u.t0 || u.t1 > b.n_active;
            bool src_bad = false;
            if (!unit_bad && lane < nsrc) {
                const SrcTab& S = tab[b.src0 + lane];
                const int K = S.K[u.band];
                src_bad = !S.ok || K < 0 || K > kCompStride;
                const tb_fit_source fs = srcs[b.src0 + lane];
                const bool live = fs.w > 0 && fs.h > 0;
                UnitSrc<T> U;
                U.x0 = live ? fs.x0 : 0;
                U.y0 = live ? fs.y0 : 0;
                U.x1 = live ? fs.x0 + fs.w : 0;
                U.y1 = live ? fs.y0 + fs.h : 0;
                U.K = K;
                U.profile = fs.profile;
                U.counts = (T)S.flux[u.band];
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    U.M[q] = (T)S.M[q];
#pragma unroll
                    for (int j = 0; j < 3; j++) U.dM[j][q] = (T)S.dM[j][q];
                }
                sm.us[lane] = U;
            }
            const bool bad = unit_bad || __any_sync(0xffffffffu, src_bad);
            if (lane == 0) {
                sm.skip = unit_bad ? 1 : bad ? -1 : 0;   // -1: its slice is its own
                if (bad) tb::report(st, TB_STATUS_BAD_ITEM, ui, nsrc);
            }
        }
        __syncthreads();
        if (sm.skip) {
            // (a gradient is summed over every slice, whatever the status says)
            if (mode == kVjp && sm.skip < 0)
                for (int e = tid; e < P; e += kThreads)
                    gbuf[b.g_off + (int64_t)u.slice * P + e] = 0.0;
            if (tid == 0) {
                if (mode == kConstant) chi2_const[b.unit0 + u.slice] = INFINITY;
                else if (mode == kEquations) chi2_part[b.unit0 + u.slice] = INFINITY;
            }
            continue;
        }
        PassUnit<T> pu;
        pu.comps = gcomps + ((int64_t)b.src0 * n_bands + u.band) * kCompStride;
        pu.cstride = (int64_t)n_bands * kCompStride;
        pu.pix_off = u.pix_off;
        // the unit's range of the tiles some source's mask reaches; kConstant:
        // the others (their chi^2 does not depend on the parameters), covered
        // by the unit that starts the range
        pu.tiles = tiles + b.tile_off + (mode == kConstant ? b.n_active : u.t0);
        pu.data = data;
        pu.inverr = mode == kVjp ? nullptr : inverr;
        pu.W = u.W;
        pu.Hh = u.H;
        const int n_t = mode == kConstant ? (u.t0 == 0 ? b.n_tiles - b.n_active : 0) : u.t1 - u.t0;
        // the sources whose masks meet a tile (the same for every warp)
        auto reach = [&](int t) -> unsigned {
            const int ox = (pu.tiles[t] & 0x3ff) * kTileW, oy = ((pu.tiles[t] >> 10) & 0x3ff) * kTileH;
            bool hit = false;
            if (lane < nsrc) {
                const UnitSrc<T>& U = sm.us[lane];
                hit = U.x1 > ox && U.x0 < ox + kTileW && U.y1 > oy && U.y0 < oy + kTileH;
            }
            return __ballot_sync(0xffffffffu, hit);
        };
        pu.out = SliceOut{nullptr, nullptr, 0u, 0, P, u.band};
        if (mode == kEquations || mode == kVjp) {
            pu.out.g = gbuf + b.g_off + (int64_t)u.slice * P;
            for (int e = tid; e < P; e += kThreads) pu.out.g[e] = 0.0;
        }
        if (mode == kEquations) {
            for (int t = 0; t < n_t; t++) pu.out.mask |= reach(t);
            pu.out.ld = kCols * __popc(pu.out.mask);
            pu.out.H = hbuf + b.h_off + (int64_t)u.slice * P * P;
            for (int e = tid; e < pu.out.ld * pu.out.ld; e += kThreads) pu.out.H[e] = 0.0;
        }
        double chi2 = 0.0;
        for (int t = 0, t1; t < n_t; t = t1) {
            // a run of tiles that the same sources meet
            const unsigned hit = mode == kConstant ? 0u : reach(t);
            t1 = t + 1;
            while (t1 < n_t && (mode == kConstant || reach(t1) == hit)) t1++;
            if (sizeof(T) == 8 && mode == kModel) {
                for (int q = t; q < t1; q++) {
                    const int ox = (pu.tiles[q] & 0x3ff) * kTileW;
                    const int py = ((pu.tiles[q] >> 10) & 0x3ff) * kTileH + warp;
                    T m = 0;
                    for (unsigned hm = hit; hm; hm &= hm - 1) {
                        const int sI = __ffs(hm) - 1;
                        m += source_model<T>(sm, sm.us[sI], pu.comps + sI * pu.cstride, ox, py);
                    }
                    if (ox + lane < u.W && py < u.H)
                        model_out[u.pix_off + (int64_t)py * u.W + ox + lane] = (float)m;
                }
                continue;
            }
            if (sizeof(T) == 8 && mode == kVjp) {
                // the upstream gradient does not depend on the model: one source at a time
                for (unsigned hm = hit; hm; hm &= hm - 1)
                    run_tiles<T, 1, false>(sm, pu, hm & (0u - hm), t, t1, chi2);
                continue;
            }
            switch (__popc(hit)) {
                case 0:
                    for (int q = t; q < t1; q++) {
                        T d, w;
                        load_pixel(pu, (pu.tiles[q] & 0x3ff) * kTileW + lane,
                                   ((pu.tiles[q] >> 10) & 0x3ff) * kTileH + warp, d, w);
                        const T r = d * w;
                        chi2 += (double)(r * r);
                    }
                    break;
                case 1: run_tiles<T, 1, true>(sm, pu, hit, t, t1, chi2); break;
                case 2: run_tiles<T, 2, true>(sm, pu, hit, t, t1, chi2); break;
                case 3: run_tiles<T, 3, true>(sm, pu, hit, t, t1, chi2); break;
                case 4: run_tiles<T, 4, true>(sm, pu, hit, t, t1, chi2); break;
                default:
                    for (int q = t; q < t1; q++) crowded_tile<T>(sm, pu, hit, pu.tiles[q], chi2);
            }
        }
        if (mode == kModel || mode == kVjp) continue;
        // chi^2 of the unit: fixed-order block reduction
        for (int o = 16; o > 0; o >>= 1) chi2 += __shfl_xor_sync(0xffffffffu, chi2, o);
        if (lane == 0) sm.red[warp] = chi2;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int w2 = 0; w2 < kWarps; w2++) s += sm.red[w2];
            if (mode == kConstant) chi2_const[b.unit0 + u.slice] = s;
            else chi2_part[b.unit0 + u.slice] = s + (chi2_const ? chi2_const[b.unit0 + u.slice] : 0.0);
            if (mode == kEquations && P > 0)
                pu.out.g[P - 1] = __longlong_as_double((long long)u.band << 32 | pu.out.mask);
        }
    }
}

// ---------------------------------------------------------------------------
// step
// ---------------------------------------------------------------------------

constexpr int kStepThreads = 256;

__device__ double max_step(int off) {
    // PixPos [1, 1] (wcs.py:384), fluxes unlimited, EllipseESoft inherits
    // EllipseE's [1, 0.1, 0.1] (ellipses.py:48), SersicIndex 0.1 (sersic.py:352)
    switch (off) {
        case 0: case 1: case 5: return 1.0;
        case 6: case 7: case 8: return 0.1;
        default: return 0.0;   // none
    }
}

// A blob's trial chi^2: its slices' parts summed by one warp in a fixed
// order (every lane gets the sum).  The assembly and the step kernel both
// decide on it, so both must sum alike.
__device__ __forceinline__ double trial_chi2(const double* __restrict__ part, int ns) {
    double c = 0.0;
    for (int k = threadIdx.x & 31; k < ns; k += 32) c += part[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    return c;
}

__device__ __forceinline__ bool accept_trial(const tb_fit_state& S, double c2) {
    return isfinite(c2) && (S.accepted == 0 || c2 < S.chi2);
}

// The slices of an accepted trial summed into the blob's accepted H (full,
// symmetric) and g.  A kernel of its own, kAsmCtas CTAs per blob, a warp per
// row: summing a large blob's slices took the one CTA of the step longer than
// factoring the result.  A row takes only the slices that hold its source
// (and, a flux, its band's), an element only those that hold both.
constexpr int kAsmCtas = 16;

__global__ void __launch_bounds__(kStepThreads)
fit_assemble_kernel(const tb_fit_blob* __restrict__ blobs,
                    const tb_fit_source* __restrict__ srcs, double* __restrict__ hbuf,
                    double* __restrict__ gbuf, const double* __restrict__ chi2_part,
                    const tb_fit_state* __restrict__ state) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const tb_fit_state& S = state[blockIdx.x];
    if (S.status != 0) return;
    const tb_fit_blob b = blobs[blockIdx.x];
    const int P = b.P, ns = b.n_slices;
    const int64_t PP = (int64_t)P * P;
    const int r0 = blockIdx.y * (kStepThreads / 32) + warp;
    if (r0 >= P) return;   // whole warps
    if (!accept_trial(S, trial_chi2(chi2_part + b.unit0, ns))) return;
    const double* Hp = hbuf + b.h_off;
    const double* gp = gbuf + b.g_off;
    double* Ha = hbuf + b.h_off + ns * PP;
    double* ga = gbuf + b.g_off + (int64_t)ns * P;
    // column within a source's seven of parameter slot `off` in `band`, or -1
    auto column = [](int off, int band) {
        return off < 2 ? off : off < 2 + TB_FIT_MAX_BANDS ? (off - 2 == band ? 2 : -1) : off - 2;
    };
    // whether a source of this profile has the parameter
    auto has = [&](int src, int off) {
        const int profile = srcs[b.src0 + src].profile;
        return off < 2 + TB_FIT_MAX_BANDS ||
               (profile != TB_PROFILE_POINT && (off < TB_FIT_NPAR - 1 || profile == TB_PROFILE_SERSIC));
    };
    for (int r = r0; r < P; r += kAsmCtas * (kStepThreads / 32)) {
        const int a = r / TB_FIT_NPAR, ao = r % TB_FIT_NPAR;
        const bool ha = has(a, ao);
        double gs = 0.0;
        for (int c0 = r; c0 < P; c0 += 32) {
            const int c = c0 + lane;
            const int s = c / TB_FIT_NPAR, so = c % TB_FIT_NPAR;
            const bool hs = c < P && ha && has(s, so);
            double h = 0.0;
            for (int k0 = 0; k0 < ns; k0 += 32) {
                // this row's slices among k0 .. k0 + 31
                const int kk = k0 + lane;
                const long long tail =
                    kk < ns ? __double_as_longlong(gp[(int64_t)kk * P + P - 1]) : 0ll;
                const unsigned mk = (unsigned)tail;
                const int band = (int)(tail >> 32);
                const int ca_l = ha ? column(ao, band) : -1;
                unsigned sl = __ballot_sync(0xffffffffu, ca_l >= 0 && ((mk >> a) & 1u));
                if (c0 == r && ((sl >> lane) & 1u))
                    gs += gp[(int64_t)kk * P + compact_row(mk, a) + ca_l];
                while (sl) {   // eight slices' loads in flight at a time
                    double x[8];
#pragma unroll
                    for (int t = 0; t < 8; t++) {
                        const int q = sl ? __ffs(sl) - 1 : 0;
                        const unsigned m = __shfl_sync(0xffffffffu, mk, q);
                        const int ca = __shfl_sync(0xffffffffu, ca_l, q);
                        const int bq = __shfl_sync(0xffffffffu, band, q);
                        const int cb = hs ? column(so, bq) : -1;
                        x[t] = sl && cb >= 0 && ((m >> s) & 1u)
                            ? Hp[(k0 + q) * PP + (compact_row(m, a) + ca) * kCols * __popc(m) +
                                 compact_row(m, s) + cb] : 0.0;
                        sl &= sl - 1;
                    }
#pragma unroll
                    for (int t = 0; t < 8; t++) h += x[t];
                }
            }
            if (c < P) {
                Ha[(int64_t)r * P + c] = h;
                Ha[(int64_t)c * P + r] = h;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) gs += __shfl_xor_sync(0xffffffffu, gs, o);
        if (lane == 0) ga[r] = gs;
    }
}

constexpr int kStepMaxP = TB_FIT_MAX_SRC * TB_FIT_NPAR;
constexpr int kStepSharedP = 128;      // largest padded size factored in shared memory
constexpr int kStepSmem = 8 * (tb::packed_size(kStepSharedP) + 7 * kStepSharedP);   // 73 KB
static_assert(kStepSmem >= 8 * 7 * ((kStepMaxP + 7) / 8 * 8), "the vectors always fit");
static_assert(3 * (kStepSmem + 2048) <= 228 * 1024, "three blobs per SM");

// Where the whole step would be scaled below kLimited of it, the parameters
// beyond their limits are held there and the others solved again, kBoxRounds
// times at most; in iterations after kPatience.  (80 fits of 1 to 28 blobs: 659 ms
// with 0.2, 685 with 0.5, 720 without; 2,000 blobs, four seeds: 1522, 1514 and 1666
// ms, with 16 iterations of patience 1599.)
constexpr double kLimited = 0.2;
constexpr int kBoxRounds = 4;
constexpr int kPatience = 8;

// One CTA per blob.  Up to 128 parameters the factor lives in shared memory
// (73 KB, three blobs per SM), above in the blob's global area.
//
// Bound: the chain of columns.  A column at a time through L2, one barrier
// each, took 0.6 ms for 126 parameters; four columns at a time (every thread
// factors the 4 x 4 diagonal block itself and finishes one row of the panel,
// then the trailing tiles are updated by FP64 tensor-core products of rank 4)
// is two barriers per four columns and 256 multiply-adds per instruction.
// Kernel time per step: 126 parameters 615 -> 175 us (with the assembly), 36
// parameters 87 -> 29 us.
//
// The step is scaled as a whole to its limits (ConstrainedOptimizer), so one
// all but undetermined parameter (the shape of a source a tenth of a pixel wide)
// can cut the step of all the others to 1e-5 of it, one iteration after the
// other: such a blob took 97 iterations, others, thousands of units of chi^2
// from their optimum, reached the limit of 100.  A blob that is still running
// after kPatience iterations therefore takes, where the quadratic model expects
// more of it, the step that minimises the model within the limits (each
// parameter beyond its limit held there, the others solved for): 26 iterations
// for the first, 12 to 50 for the others.  Most blobs stop before, and their
// steps are what they were.
__global__ void __launch_bounds__(kStepThreads, 3)
fit_step_kernel(const tb_fit_blob* __restrict__ blobs, int n_blobs, int n_bands,
                const tb_fit_source* __restrict__ srcs, double* __restrict__ params,
                double* __restrict__ trial, double* __restrict__ hbuf, double* __restrict__ gbuf,
                const double* __restrict__ chi2_part, tb_fit_state* __restrict__ state,
                double tol, int max_iter) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red[kStepThreads / 32], red2[kStepThreads / 32];
    __shared__ int s_active, s_accept, s_slow;
    __shared__ double s_lambda, s_scale, s_pa, s_pb;
    const int bi = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    (void)n_bands;
    if (bi >= n_blobs) return;
    const tb_fit_blob b = blobs[bi];
    tb_fit_state& S = state[bi];
    const int status0 = S.status;
    __syncthreads();   // every thread has read the status before thread 0 updates it
    if (status0 != 0) return;
    const int P = b.P;
    const int n = (P + 7) / 8 * 8;
    const int ns = b.n_slices;
    double* dsc = reinterpret_cast<double*>(smem_raw);
    double* dinv = dsc + n;
    double* y = dinv + n;
    double* xs = y + n;
    double* rdg = xs + n;
    double* gm = rdg + n;      // gradient, with the held parameters at their limits
    double* held = gm + n;     // their steps; 0 for the others
    double* Ha = hbuf + b.h_off + (int64_t)ns * P * P;   // accepted H
    double* L = n <= kStepSharedP ? held + n : Ha + (int64_t)P * P;   // factor
    double* ga = gbuf + b.g_off + (int64_t)ns * P;
    double* pa = params + (int64_t)b.src0 * TB_FIT_NPAR;
    double* pt = trial + (int64_t)b.src0 * TB_FIT_NPAR;
    auto col = [&](int j) { return L + tb::packed_col(j, n); };

    const double c2 = warp == 0 ? trial_chi2(chi2_part + b.unit0, ns) : 0.0;
    if (tid == 0) {
        const bool first = S.accepted == 0;
        const bool acc = accept_trial(S, c2);
        int status = 0;
        if (acc) {
            // damping from the gain ratio rho = actual / predicted (Nielsen's
            // rule: lambda x max(1/3, 1 - (2 rho - 1)^3); x 0.3 without a
            // prediction)
            const double gain = first ? INFINITY : 0.5 * (S.chi2 - c2);
            double fct = 0.3;
            if (!first && S.pred > 0.0 && isfinite(S.pred)) {
                const double t = 2.0 * (gain / S.pred) - 1.0;
                fct = fmax(1.0 / 3.0, 1.0 - t * t * t);
            }
            S.dlnp = gain;
            S.chi2 = c2;
            S.accepted += 1;
            S.lambda = fmax(S.lambda * fct, 1e-9);
        } else {
            S.lambda *= 10.0;
            S.rejected += 1;
            if (!(S.lambda < 1e12) || !isfinite(c2) && first) status = 2;
        }
        S.iters += 1;
        if (status == 0 && S.iters >= max_iter) status = 3;
        s_accept = acc;
        s_lambda = S.lambda;
        s_slow = S.iters > kPatience;
        s_active = status == 0;
        S.status = status;
    }
    __syncthreads();
    if (s_accept) {
        for (int e = tid; e < P; e += kStepThreads) pa[e] = pt[e];
    }
    __syncthreads();
    if (!s_active) {
        // stopped: the trial parameters are the accepted ones
        for (int e = tid; e < P; e += kStepThreads) pt[e] = pa[e];
        return;
    }
    const double lam = s_lambda;
    // Marquardt scaling: D = sqrt(diag H); (D^-1 H D^-1 + lambda I) x = D^-1 g
    for (int i = tid; i < P; i += kStepThreads) {
        const double a = Ha[(int64_t)i * P + i];
        double d = (a > 0.0 && isfinite(a)) ? sqrt(a) : 0.0;
        // a Sersic index held at a bound that the gradient pushes against is
        // left out of the step (projected step; the bound-constrained optimum)
        if (i % TB_FIT_NPAR == TB_FIT_NPAR - 1 &&
            srcs[b.src0 + i / TB_FIT_NPAR].profile == TB_PROFILE_SERSIC &&
            ((pa[i] >= TB_FIT_SERSIC_MAX && ga[i] > 0.0) ||
             (pa[i] <= TB_FIT_SERSIC_MIN && ga[i] < 0.0)))
            d = 0.0;
        // frozen parameters are left out of the step
        if ((srcs[b.src0 + i / TB_FIT_NPAR].frozen >> (i % TB_FIT_NPAR)) & 1) d = 0.0;
        dsc[i] = d;
        dinv[i] = d == 0.0 ? 0.0 : 1.0 / d;
        gm[i] = ga[i];
        held[i] = 0.0;
    }
    for (int i = P + tid; i < n; i += kStepThreads) dinv[i] = dsc[i] = 0.0;
    __syncthreads();
    // take(i, sum_j H_ij value(j)) for every row i by one thread each, four rows
    // of a warp at a time (Ha is symmetric); elements of columns whose value is
    // 0 are not used
    auto rows_of_H = [&](auto value, auto take) {
        for (int i0 = 4 * warp; i0 < P; i0 += 4 * (kStepThreads / 32)) {
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
            for (int j = lane; j < P; j += 32) {
                const double vj = value(j);
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const double h = i0 + t < P ? Ha[(int64_t)(i0 + t) * P + j] : 0.0;
                    acc[t] = fma(vj != 0.0 ? h : 0.0, vj, acc[t]);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int t = 0; t < 4; t++) acc[t] += __shfl_xor_sync(0xffffffffu, acc[t], o);
#pragma unroll
            for (int t = 0; t < 4; t++)
                if (lane == t && i0 + t < P) take(i0 + t, acc[t]);
        }
    };
    // the parameters a multiple of the step y away
    auto write_trial = [&](double scale) {
        for (int i = tid; i < P; i += kStepThreads) {
            double v = pa[i] + scale * y[i];
            if (i % TB_FIT_NPAR == TB_FIT_NPAR - 1 &&
                srcs[b.src0 + i / TB_FIT_NPAR].profile == TB_PROFILE_SERSIC)
                v = fmin(fmax(v, TB_FIT_SERSIC_MIN), TB_FIT_SERSIC_MAX);
            pt[i] = v;
        }
    };
    double scaled_gain = 0.0;
    for (int round = 0;; round++) {
        // LDL^T of the scaled matrix, right-looking: column k is left as d_k
        // (diagonal) and c_ik = d_k l_ik below it, and subtracts c_ik c_jk / d_k
        // from the trailing columns.
        for (int j0 = 0; j0 < n; j0 += kStepThreads / 32) {
            const int j = j0 + warp;
            const double dj = dinv[j];
#pragma unroll 4
            for (int i = j + lane; i < n; i += 32) {
                const double h = i < P ? Ha[(int64_t)j * P + i] : 0.0;   // (j <= i)
                const bool live = dinv[i] != 0.0 && dj != 0.0;
                col(j)[i] = live ? h * dinv[i] * dj + (i == j ? lam : 0.0) : (i == j ? 1.0 : 0.0);
            }
        }
        __syncthreads();
        const bool bad = tb::ldl_factor<kStepThreads>(L, rdg, n) != 0;
        if (bad) {
            if (round > 0) return;   // the scaled step stands
            // not positive definite: treat as a rejected step with more damping
            if (tid == 0) {
                S.lambda *= 10.0;
                if (!(S.lambda < 1e12)) S.status = 2;
            }
            for (int e = tid; e < P; e += kStepThreads) pt[e] = pa[e];
            return;
        }
        for (int i = tid; i < n; i += kStepThreads) {
            xs[i] = 0.0;
            y[i] = i < P ? gm[i] * dinv[i] : 0.0;
        }
        __syncthreads();
        // solution and one refinement step
        for (int pass = 0; pass < 2; pass++) {
            if (pass == 1) {
                rows_of_H([&](int j) { return dinv[j] * xs[j]; }, [&](int i, double hx) {
                    y[i] = dinv[i] != 0.0 ? gm[i] * dinv[i] - (hx * dinv[i] + lam * xs[i])
                                          : -xs[i];
                });
                __syncthreads();
            }
            if (warp == 0) tb::ldl_solve(L, rdg, y, n);
            __syncthreads();
            for (int i = tid; i < P; i += kStepThreads) xs[i] += y[i];
            __syncthreads();
        }
        if (round == 0) {
            // Predicted log-likelihood gain of this damped step,
            // 1/2 (x . D^-1 g + lambda x . x); the blob has converged when it is
            // below tol while the damping is moderate (optimize_loop stops on the
            // gain of the last step, dchisq; the prediction is immune to FP32
            // noise in chi^2).
            {
                // a = x^T y0, b = x^T x: the gain predicted for the step is
                // (a + lambda b) / 2, for the step scaled by s it is
                // s a - s^2 (a - lambda b) / 2
                double pa_ = 0.0, pb_ = 0.0;
                for (int i = tid; i < P; i += kStepThreads) {
                    const double y0 = dsc[i] == 0.0 ? 0.0 : ga[i] / dsc[i];
                    pa_ += xs[i] * y0;
                    pb_ += xs[i] * xs[i];
                }
                for (int o = 16; o > 0; o >>= 1) {
                    pa_ += __shfl_xor_sync(0xffffffffu, pa_, o);
                    pb_ += __shfl_xor_sync(0xffffffffu, pb_, o);
                }
                if (lane == 0) {
                    red[warp] = pa_;
                    red2[warp] = pb_;
                }
                __syncthreads();
                if (tid == 0) {
                    double ta = 0.0, tb2 = 0.0;
                    for (int w2 = 0; w2 < kStepThreads / 32; w2++) {
                        ta += red[w2];
                        tb2 += red2[w2];
                    }
                    s_pa = ta;
                    s_pb = tb2;
                    const double t = ta + lam * tb2;
                    S.pred = 0.5 * t;
                    s_active = !(0.5 * t < tol && lam <= 1.0);
                    if (!s_active) S.status = 1;
                }
                __syncthreads();
                if (!s_active) {
                    for (int e = tid; e < P; e += kStepThreads) pt[e] = pa[e];
                    return;
                }
            }
            // step = x / D, limited by maximum steps and the Sersic-index bounds
            // (ConstrainedOptimizer scales the whole step, constrained_optimizer.py)
            double lim = 1.0;
            for (int i = tid; i < P; i += kStepThreads) {
                const double dlt = dsc[i] == 0.0 ? 0.0 : xs[i] / dsc[i];
                y[i] = dlt;
                const int off = i % TB_FIT_NPAR;
                const double ms = max_step(off);
                if (ms > 0.0 && fabs(dlt) > ms) lim = fmin(lim, ms / fabs(dlt));
                if (off == TB_FIT_NPAR - 1 &&
                    srcs[b.src0 + i / TB_FIT_NPAR].profile == TB_PROFILE_SERSIC) {
                    const double nv = pa[i] + dlt;
                    if (nv > TB_FIT_SERSIC_MAX && dlt > 0.0)
                        lim = fmin(lim, (TB_FIT_SERSIC_MAX - pa[i]) / dlt);
                    if (nv < TB_FIT_SERSIC_MIN && dlt < 0.0)
                        lim = fmin(lim, (TB_FIT_SERSIC_MIN - pa[i]) / dlt);
                }
            }
            for (int o = 16; o > 0; o >>= 1)
                lim = fmin(lim, __shfl_xor_sync(0xffffffffu, lim, o));
            if (lane == 0) red[warp] = lim;
            __syncthreads();
            if (tid == 0) {
                double l = 1.0;
                for (int w2 = 0; w2 < kStepThreads / 32; w2++) l = fmin(l, red[w2]);
                s_scale = fmax(l, 0.0);
                // the gain predicted for the trial as scaled (the next call's gain
                // ratio divides by it)
                S.pred = s_scale * s_pa - 0.5 * s_scale * s_scale * (s_pa - lam * s_pb);
            }
            __syncthreads();
            write_trial(s_scale);
            if (!s_slow || !(s_scale < kLimited)) return;
            scaled_gain = s_scale * s_pa - 0.5 * s_scale * s_scale * (s_pa - lam * s_pb);
        }
        // the step with the held parameters' shares, and whether more of it is
        // beyond its limits
        bool over = false;
        for (int i = tid; i < P; i += kStepThreads) {
            double dlt = held[i];
            if (dsc[i] != 0.0) {
                dlt = xs[i] / dsc[i];
                const int off = i % TB_FIT_NPAR;
                const double ms = max_step(off);
                double lo = ms > 0.0 ? -ms : -INFINITY, hi = ms > 0.0 ? ms : INFINITY;
                if (off == TB_FIT_NPAR - 1) {
                    lo = fmax(lo, TB_FIT_SERSIC_MIN - pa[i]);
                    hi = fmin(hi, TB_FIT_SERSIC_MAX - pa[i]);
                }
                if (dlt < lo || dlt > hi) {
                    over = true;
                    dlt = dlt < lo ? lo : hi;
                    dsc[i] = dinv[i] = 0.0;
                    held[i] = dlt;
                }
            }
            y[i] = dlt;
        }
        if (!__syncthreads_or(over)) {
            // (g - H y / 2) . y, into the trial if that is more than the scaled one's
            double gain = 0.0;
            rows_of_H([&](int j) { return y[j]; },
                      [&](int i, double hy) { gain += y[i] * (ga[i] - 0.5 * hy); });
            for (int o = 16; o > 0; o >>= 1) gain += __shfl_xor_sync(0xffffffffu, gain, o);
            if (lane == 0) red[warp] = gain;
            __syncthreads();
            gain = 0.0;
            for (int w2 = 0; w2 < kStepThreads / 32; w2++) gain += red[w2];
            if (!(gain > scaled_gain)) return;
            if (tid == 0) S.pred = gain;
            write_trial(1.0);
            return;
        }
        if (round == kBoxRounds) return;
        rows_of_H([&](int j) { return held[j]; }, [&](int i, double hh) { gm[i] = ga[i] - hh; });
        __syncthreads();
    }
}

__global__ void fit_reset_kernel(tb_fit_state* state, int n, double lambda0) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    tb_fit_state s;
    s.chi2 = INFINITY;
    s.dlnp = INFINITY;
    s.lambda = lambda0;
    s.pred = INFINITY;
    s.iters = 0;
    s.accepted = 0;
    s.rejected = 0;
    s.status = 0;
    state[i] = s;
}

}  // namespace

extern "C" int tb_fit_workspace(int32_t n_src, int32_t n_bands, int64_t* bytes) {
    if (n_src < 0 || n_bands < 1 || n_bands > TB_FIT_MAX_BANDS || !bytes) return TB_ERR_ARG;
    const int64_t tab = ((int64_t)n_src * (int64_t)sizeof(SrcTab) + 255) / 256 * 256;
    const int64_t nc = (int64_t)n_src * n_bands * kCompStride;
    *bytes = tab + nc * (int64_t)(sizeof(FitC<float>) + sizeof(FitC<double>));
    return TB_OK;
}

namespace {
inline SrcTab* ws_tab(void* ws) { return static_cast<SrcTab*>(ws); }
// component tables: FP64, then FP32
inline FitC<double>* ws_comps64(void* ws, int32_t n_src) {
    const int64_t tab = ((int64_t)n_src * (int64_t)sizeof(SrcTab) + 255) / 256 * 256;
    return reinterpret_cast<FitC<double>*>(static_cast<char*>(ws) + tab);
}
inline FitC<float>* ws_comps32(void* ws, int32_t n_src, int32_t n_bands) {
    return reinterpret_cast<FitC<float>*>(ws_comps64(ws, n_src) +
                                          (int64_t)n_src * n_bands * kCompStride);
}
inline const FitC<float>* ws_comps(void* ws, int32_t n_src, int32_t n_bands, float) {
    return ws_comps32(ws, n_src, n_bands);
}
inline const FitC<double>* ws_comps(void* ws, int32_t n_src, int32_t, double) {
    return ws_comps64(ws, n_src);
}

// One launch of the pass kernel in precision T over all units.
template <class T>
int launch_pass(const tb_fit_unit* units, const int32_t* order, int32_t n_units,
                const tb_fit_blob* blobs, const tb_fit_source* srcs, int32_t n_src,
                const void* workspace, const float* data, const float* inverr,
                const int32_t* tiles, double* hbuf, double* gbuf, double* chi2_part,
                double* chi2_const, const tb_fit_state* state, int32_t n_bands, Mode mode,
                float* model, int32_t* work_counter, tb_status* status, cudaStream_t s) {
    const int smem = (int)sizeof(PassSmem<T>);
    if (cudaFuncSetAttribute(fit_pass_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem) != cudaSuccess)
        return TB_ERR_LAUNCH;
    if (cudaMemsetAsync(work_counter, 0, sizeof(int32_t), s) != cudaSuccess) return TB_ERR_LAUNCH;
    if (status && cudaMemsetAsync(status, 0, sizeof(tb_status), s) != cudaSuccess)
        return TB_ERR_LAUNCH;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fit_pass_kernel<T>, kThreads,
                                                      smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    const int64_t want = (int64_t)tb::num_sms() * per_sm;
    const int grid = (int)(n_units < want ? n_units : want);
    void* ws = const_cast<void*>(workspace);
    fit_pass_kernel<T><<<grid, kThreads, smem, s>>>(
        units, order, n_units, blobs, srcs, ws_tab(ws), ws_comps(ws, n_src, n_bands, T()), data,
        inverr, hbuf, gbuf, chi2_part, state, n_bands, tiles, chi2_const, mode, model,
        work_counter, status);
    return cudaGetLastError() == cudaSuccess ? TB_OK : TB_ERR_LAUNCH;
}
}  // namespace

extern "C" int tb_fit_reset(tb_fit_state* state, int32_t n_blobs, double lambda0, void* stream) {
    if (n_blobs < 0 || (n_blobs > 0 && !state)) return TB_ERR_ARG;
    if (n_blobs == 0) return TB_OK;
    fit_reset_kernel<<<(n_blobs + 255) / 256, 256, 0, (cudaStream_t)stream>>>(state, n_blobs,
                                                                             lambda0);
    return cudaGetLastError() == cudaSuccess ? TB_OK : TB_ERR_LAUNCH;
}

extern "C" int tb_fit_prep(const tb_fit_source* srcs, int32_t n_src, const double* params,
                           int32_t n_bands, const tb_fit_unit* units, int32_t n_units,
                           const double* cd_inv, const tb_profile_tables* tables, void* workspace,
                           const tb_fit_state* state, void* stream) {
    if (n_src < 0 || n_bands < 1 || n_bands > TB_FIT_MAX_BANDS || n_units < 0) return TB_ERR_ARG;
    if (n_src == 0) return TB_OK;
    if (!srcs || !params || !units || !cd_inv || !tables || !workspace) return TB_ERR_ARG;
    const int smem = tb::tables_smem_bytes(*tables);
    if (smem > TB_PROFILE_SMEM_MAX) return TB_ERR_SIZE;
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(fit_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
            cudaSuccess)
        return TB_ERR_LAUNCH;
    const int per_block = kPrepThreads / 32;
    fit_prep_kernel<<<(n_src + per_block - 1) / per_block, kPrepThreads, smem,
                      (cudaStream_t)stream>>>(srcs, n_src, params, n_bands, units, n_units,
                                              *tables, cd_inv[0], cd_inv[1], cd_inv[2], cd_inv[3],
                                              ws_tab(workspace),
                                              ws_comps32(workspace, n_src, n_bands),
                                              ws_comps64(workspace, n_src), state);
    return cudaGetLastError() == cudaSuccess ? TB_OK : TB_ERR_LAUNCH;
}

extern "C" int tb_fit_pass(const tb_fit_unit* units, const int32_t* order, int32_t n_units,
                           const tb_fit_blob* blobs, const tb_fit_source* srcs, int32_t n_src,
                           const void* workspace, const float* data, const float* inverr,
                           const int32_t* tiles, double* hbuf, double* gbuf, double* chi2_part,
                           double* chi2_const, const tb_fit_state* state, int32_t n_bands,
                           int32_t mode, int32_t* work_counter, tb_status* status,
                           void* stream) {
    if (n_units < 0 || n_src < 0 || n_bands < 1 || n_bands > TB_FIT_MAX_BANDS) return TB_ERR_ARG;
    if (mode != 0 && mode != 1) return TB_ERR_ARG;
    if (n_units == 0) return TB_OK;
    if (!units || !order || !blobs || !srcs || !workspace || !data || !inverr || !tiles ||
        !hbuf || !gbuf || !chi2_part || !chi2_const || !state || !work_counter)
        return TB_ERR_ARG;
    return launch_pass<float>(units, order, n_units, blobs, srcs, n_src, workspace, data, inverr,
                              tiles, hbuf, gbuf, chi2_part, chi2_const, state, n_bands,
                              mode == 0 ? kEquations : kConstant, nullptr, work_counter, status,
                              (cudaStream_t)stream);
}

extern "C" int tb_fit_step(const tb_fit_blob* blobs, int32_t n_blobs, int32_t n_bands,
                           const tb_fit_source* srcs, double* params, double* trial,
                           double* hbuf, double* gbuf, const double* chi2_part,
                           tb_fit_state* state, double tol, int32_t max_iter, void* stream) {
    if (n_blobs < 0 || n_bands < 1 || n_bands > TB_FIT_MAX_BANDS) return TB_ERR_ARG;
    if (n_blobs == 0) return TB_OK;
    if (!blobs || !srcs || !params || !trial || !hbuf || !gbuf || !chi2_part || !state)
        return TB_ERR_ARG;
    if (cudaFuncSetAttribute(fit_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kStepSmem) != cudaSuccess)
        return TB_ERR_LAUNCH;
    fit_assemble_kernel<<<dim3(n_blobs, kAsmCtas), kStepThreads, 0, (cudaStream_t)stream>>>(
        blobs, srcs, hbuf, gbuf, chi2_part, state);
    fit_step_kernel<<<n_blobs, kStepThreads, kStepSmem, (cudaStream_t)stream>>>(
        blobs, n_blobs, n_bands, srcs, params, trial, hbuf, gbuf, chi2_part, state, tol, max_iter);
    return cudaGetLastError() == cudaSuccess ? TB_OK : TB_ERR_LAUNCH;
}

extern "C" int tb_fit_refine(const tb_fit_unit* units, const int32_t* order, int32_t n_units,
                             const tb_fit_blob* blobs, const tb_fit_source* srcs, int32_t n_src,
                             const void* workspace, const float* data, const float* inverr,
                             const int32_t* tiles, double* hbuf, double* gbuf,
                             double* chi2_out, const double* chi2_const,
                             const tb_fit_state* state, int32_t n_bands, int32_t* work_counter,
                             tb_status* status, void* stream) {
    if (n_units < 0 || n_src < 0 || n_bands < 1 || n_bands > TB_FIT_MAX_BANDS) return TB_ERR_ARG;
    if (n_units == 0) return TB_OK;
    if (!units || !order || !blobs || !srcs || !workspace || !data || !inverr || !tiles ||
        !hbuf || !gbuf || !chi2_out || !state || !work_counter)
        return TB_ERR_ARG;
    return launch_pass<double>(units, order, n_units, blobs, srcs, n_src, workspace, data, inverr,
                               tiles, hbuf, gbuf, chi2_out, const_cast<double*>(chi2_const), state,
                               n_bands, kEquations, nullptr, work_counter, status,
                               (cudaStream_t)stream);
}

extern "C" int tb_fit_model_vjp(const tb_fit_unit* units, const int32_t* order, int32_t n_units,
                                const tb_fit_blob* blobs, const tb_fit_source* srcs,
                                int32_t n_src, const void* workspace, const float* grad,
                                float* model, const int32_t* tiles, double* gbuf,
                                int32_t n_bands, int32_t mode, int32_t* work_counter,
                                tb_status* status, void* stream) {
    if (n_units < 0 || n_src < 0 || n_bands < 1 || n_bands > TB_FIT_MAX_BANDS) return TB_ERR_ARG;
    if (mode != TB_FIT_MODEL && mode != TB_FIT_VJP) return TB_ERR_ARG;
    if (n_units == 0) return TB_OK;
    if (!units || !order || !blobs || !srcs || !workspace || !tiles || !work_counter ||
        (mode == TB_FIT_MODEL && !model) || (mode == TB_FIT_VJP && (!grad || !gbuf)))
        return TB_ERR_ARG;
    return launch_pass<double>(units, order, n_units, blobs, srcs, n_src, workspace, grad, nullptr,
                               tiles, nullptr, gbuf, nullptr, nullptr, nullptr, n_bands,
                               mode == TB_FIT_MODEL ? kModel : kVjp, model, work_counter, status,
                               (cudaStream_t)stream);
}

