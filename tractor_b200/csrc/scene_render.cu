// Scene rendering (sm_100a): many sources into whole images, the batched
// Tractor.getModelImage (tractor/engine.py:424-445) for mixture-of-Gaussians
// PSFs.
//
// 1. tb_scene_prep: one warp per (source, image) record builds the source's
//    PSF-convolved mixture (galaxy.py:307-326 run_mog; point sources
//    psf.py:458-528) and its pixel rectangle (the ModelMask clipped to the
//    image, as Patch.addTo clips, patch.py:341-354).
// 2. Binning: every item is listed in each image tile (32 x tile_h) that its
//    rectangle touches -- a count pass, an exclusive scan, a fill pass.
// 3. tb_scene_render: a persistent kernel takes image tiles from a global
//    counter.  For a tile it sorts the listed items by index (catalog order),
//    stages their components -- culled against the part of the tile inside
//    each item's rectangle -- in shared memory, evaluates them (a few ex2 for
//    a thread's rows, carried down its columns), sums each source's components into a
//    per-source partial (the reference's patch), adds the partial inside the
//    rectangle to the tile accumulator, and writes every tile pixel once.
//    No float atomics; the result does not depend on scheduling.
#include "f32x2.cuh"
#include "profile_eval.cuh"

namespace {

constexpr int kPrepThreads = 128;   // 4 records (warps) per block
constexpr int kMaxGal = 32;         // galaxy components of one source (one per lane)
constexpr int kCap = 1024;          // items of one tile handled per chunk

// ---------------------------------------------------------------------------
// 1. prep
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(kPrepThreads)
scene_prep_kernel(const tb_scene_src* __restrict__ srcs, int n,
                  const tb_scene_image* __restrict__ images, int n_images,
                  const double* __restrict__ pamp, const double* __restrict__ pmean,
                  const double* __restrict__ pvar, tb_profile_tables Tg,
                  tb_scene_item* __restrict__ items, double* __restrict__ camp,
                  double* __restrict__ cmean, double* __restrict__ cvar, int stride) {
    // the tables are read where they lie (L1-cached), as in galaxy_fft_prep_kernel
    const tb_profile_tables T = Tg;
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * (kPrepThreads / 32) + (threadIdx.x >> 5);
    if (i >= n) return;   // whole warps leave together
    const tb_scene_src s = srcs[i];
    int flag = 0;
    const bool img_ok = s.image >= 0 && s.image < n_images;
    tb_scene_image im;
    if (img_ok) im = images[s.image];
    else {
        flag = 2;
        im = tb_scene_image{};
        im.cd_inv[0] = im.cd_inv[3] = 1.0;
    }

    // rectangle = ModelMask clipped to the image
    const int x0 = max(s.mx0, 0), y0 = max(s.my0, 0);
    const int x1 = min(s.mx0 + s.mw, im.W), y1 = min(s.my0 + s.mh, im.H);
    if (flag == 0 && (x1 <= x0 || y1 <= y0 || s.counts == 0.0)) flag = 1;
    const int Kp = im.psf_K;
    if (flag == 0 && (Kp <= 0 || Kp > 32)) flag = 2;

    // galaxy components: lane l holds component `slot` of the whole source
    // (composite: deV block, then exp block; galaxy.py:847-876)
    double a = 0.0, V00 = 0.0, V01 = 0.0, V11 = 0.0;
    int Kg = 0, slot = lane;
    const bool point = s.profile == TB_PROFILE_POINT;
    if (point) {
        Kg = 1;
        a = lane == 0 ? 1.0 : 0.0;
    } else if (s.profile == TB_PROFILE_COMPOSITE) {
        const double f = fmin(1.0, fmax(0.0, s.fdev));
        int Kd = 0, Ke = 0;
        double G[4], re, M00, M01, M11;
        if (f > 0.0) {
            double ad, vd;
            Kd = tb::warp_profile(T, TB_PROFILE_DEV, 0.0, lane, kMaxGal, ad, vd);
            tb::shape_basis(s.shape_type, s.sb0, s.sb1, s.sb2, G, re);
            tb::pixel_factor(im.cd_inv, G, M00, M01, M11);
            if (lane < Kd) {
                a = ad * f;
                V00 = vd * M00;
                V01 = vd * M01;
                V11 = vd * M11;
            }
        }
        if (f < 1.0 && Kd >= 0) {
            // exp component index of this lane (>= 32: none)
            const int el = lane >= Kd ? lane - Kd : 32 + lane;
            double ae, ve;
            Ke = tb::warp_profile(T, TB_PROFILE_EXP, 0.0, el, kMaxGal, ae, ve);
            tb::shape_basis(s.shape_type, s.sa0, s.sa1, s.sa2, G, re);
            tb::pixel_factor(im.cd_inv, G, M00, M01, M11);
            if (el < Ke) {
                a = ae * (1.0 - f);
                V00 = ve * M00;
                V01 = ve * M01;
                V11 = ve * M11;
            }
        }
        if (Kd < 0 || Ke < 0 || Kd + Ke > kMaxGal) flag = 2;
        else Kg = Kd + Ke;
    } else {
        double ab, vb;
        const int Kb = tb::warp_profile(T, s.profile, s.sersic_n, lane, kMaxGal, ab, vb);
        // Sersic components sorted by variance (sersic.py:338-341)
        const int rank = s.profile == TB_PROFILE_SERSIC ? tb::variance_rank(vb, Kb, lane) : lane;
        double G[4], re, M00, M01, M11;
        tb::shape_basis(s.shape_type, s.sa0, s.sa1, s.sa2, G, re);
        tb::pixel_factor(im.cd_inv, G, M00, M01, M11);
        if (Kb < 0) {
            flag = 2;
        } else {
            Kg = Kb;
            if (lane < Kb) {
                a = ab;
                V00 = vb * M00;
                V01 = vb * M01;
                V11 = vb * M11;
                slot = rank;
            }
        }
    }
    const int K = Kg * Kp;
    if (flag == 0 && K > stride) flag = 2;
    const int c0 = i * stride;
    if (flag == 0 && lane < Kg) {
        // MixtureOfGaussians.convolve (mixture_profiles.py:158-172): PSF
        // component p (outer) x galaxy component k (inner)
        const double mx = point ? 0.0 : s.px, my = point ? 0.0 : s.py;
        for (int p = 0; p < Kp; p++) {
            const int pc = im.psf_c0 + p;
            const int c = c0 + p * Kg + slot;
            camp[c] = a * pamp[pc];
            cmean[2 * c] = mx + pmean[2 * pc];
            cmean[2 * c + 1] = my + pmean[2 * pc + 1];
            cvar[4 * c] = V00 + pvar[4 * pc];
            cvar[4 * c + 1] = V01 + pvar[4 * pc + 1];
            cvar[4 * c + 2] = V01 + pvar[4 * pc + 2];
            cvar[4 * c + 3] = V11 + pvar[4 * pc + 3];
        }
    }
    if (lane == 0) {
        tb_scene_item it;
        it.x0 = x0;
        it.y0 = y0;
        it.w = flag == 0 ? x1 - x0 : 0;
        it.h = flag == 0 ? y1 - y0 : 0;
        it.c0 = c0;
        it.K = flag == 0 ? K : 0;
        it.image = s.image;
        it.flag = flag;
        it.fx = point ? s.px : 0.0;
        it.fy = point ? s.py : 0.0;
        it.scale = (float)s.counts;
        it.floor = -50.0f;   // c_gauss_2d_grid: Mahalanobis^2 >= 100 is skipped
        items[i] = it;
    }
}

// ---------------------------------------------------------------------------
// 2. binning
// ---------------------------------------------------------------------------

__device__ __forceinline__ bool item_tiles(const tb_scene_item& it, const tb_scene_image& im,
                                           int tile_h, int& tx0, int& tx1, int& ty0, int& ty1) {
    if (it.flag != 0 || it.w <= 0 || it.h <= 0 || it.K <= 0) return false;
    tx0 = it.x0 / TB_MOG_TILE;
    tx1 = (it.x0 + it.w - 1) / TB_MOG_TILE;
    ty0 = it.y0 / tile_h;
    ty1 = (it.y0 + it.h - 1) / tile_h;
    return true;
}

// One warp per item, its lanes over the tiles the item's rectangle touches
// (a thread per item waited for up to 81 returning atomics in turn: 23 us for
// 150 items, 46 us for 20,000; now 3 and 9).  The count pass fills `counts`,
// the fill pass takes list positions from the end of each tile's range by
// counting it down (the render sorts each tile's items).
constexpr int kBinThreads = 256;

template <bool kFill>
__global__ void __launch_bounds__(kBinThreads)
scene_bin_kernel(const tb_scene_item* __restrict__ items, int n_items,
                 const tb_scene_image* __restrict__ images, int n_images, int64_t n_tiles,
                 int tile_h, int32_t* __restrict__ counts, const int32_t* __restrict__ offsets,
                 int32_t* __restrict__ list, int64_t max_pairs, tb_status* st) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * (kBinThreads / 32) + (threadIdx.x >> 5);
    if (i >= n_items) return;
    const tb_scene_item it = items[i];
    if (it.image < 0 || it.image >= n_images) {
        if (!kFill && it.flag == 0 && lane == 0) tb::report(st, TB_STATUS_BAD_ITEM, i, -1);
        return;
    }
    const tb_scene_image im = images[it.image];
    int tx0, tx1, ty0, ty1;
    if (!item_tiles(it, im, tile_h, tx0, tx1, ty0, ty1)) return;
    const int tiles_x = (im.W + TB_MOG_TILE - 1) / TB_MOG_TILE;
    const int nx = tx1 - tx0 + 1, n = nx * (ty1 - ty0 + 1);
    for (int q = lane; q < n; q += 32) {
        const int64_t t = im.tile0 + (int64_t)(ty0 + q / nx) * tiles_x + tx0 + q % nx;
        if (t < 0 || t >= n_tiles) {
            if (!kFill) tb::report(st, TB_STATUS_BAD_ITEM, i, -2);
            continue;
        }
        if (kFill) {
            const int64_t at = (int64_t)offsets[t] + atomicSub(&counts[t], 1) - 1;
            if (at < max_pairs) list[at] = i;
            else tb::report(st, TB_STATUS_BAD_ITEM, i, -3);
        } else {
            atomicAdd(&counts[t], 1);
        }
    }
}

// Exclusive scan of counts[0..n) into offsets[0..n] in three passes:
// per-block scans (1024 values per block), a scan of the block totals, and
// the block offsets added back.
constexpr int kScanThreads = 1024;

__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_tot, int& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < (int)(blockDim.x >> 5) ? warp_tot[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        warp_tot[lane] = w;   // inclusive over warps
    }
    __syncthreads();
    total = warp_tot[(blockDim.x >> 5) - 1];
    const int before = warp > 0 ? warp_tot[warp - 1] : 0;
    __syncthreads();
    return before + x - v;
}

__global__ void __launch_bounds__(kScanThreads)
scan_blocks_kernel(const int32_t* __restrict__ counts, int64_t n, int32_t* __restrict__ offsets,
                   int32_t* __restrict__ bsum) {
    // (one block: the whole scan, its total included)
    __shared__ int warp_tot[32];
    const int64_t i = (int64_t)blockIdx.x * kScanThreads + threadIdx.x;
    const int v = i < n ? counts[i] : 0;
    int total;
    const int ex = block_exclusive_scan(v, warp_tot, total);
    if (i < n) offsets[i] = ex;
    if (threadIdx.x == 0) {
        bsum[blockIdx.x] = total;
        if (gridDim.x == 1) offsets[n] = total;
    }
}

__global__ void __launch_bounds__(kScanThreads)
scan_sums_kernel(int32_t* __restrict__ bsum, int nb, int32_t* __restrict__ offsets, int64_t n) {
    __shared__ int warp_tot[32];
    int carry = 0;
    for (int b0 = 0; b0 < nb; b0 += kScanThreads) {
        const int b = b0 + threadIdx.x;
        const int v = b < nb ? bsum[b] : 0;
        int total;
        const int ex = block_exclusive_scan(v, warp_tot, total);
        if (b < nb) bsum[b] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) offsets[n] = carry;
}

__global__ void __launch_bounds__(kScanThreads)
scan_add_kernel(int32_t* __restrict__ offsets, int64_t n, const int32_t* __restrict__ bsum) {
    const int64_t i = (int64_t)blockIdx.x * kScanThreads + threadIdx.x;
    if (i < n) offsets[i] += bsum[blockIdx.x];
}

// ---------------------------------------------------------------------------
// 3. render
// ---------------------------------------------------------------------------

using tb::f32x2;
using tb::pack;
using tb::unpack;
using tb::fma2;
using tb::mul2;
using tb::add2;

// A staged component: exponent qxx dx^2 + qxy dx dy + qyy dy^2 (log2 units),
// its tile-relative centre as the nearest pixel plus a fraction (the centre
// as one FP32 number was the largest error of the render: half an ulp of a
// coordinate up to 64), Q = 2^(2 qyy), the amplitude s, the floor 2^fl, the
// source it belongs to and the source's rectangle in the tile.
struct __align__(16) SceneC {
    float qxx[2], qxy[2];     // twice each: packed operands
    float Q[2], s[2];
    float ix, fx, iy, fy;
    float qyy, thr;
    int src;
    uint32_t rect;            // x0 | x1 << 6 | y0 << 12 | y1 << 19, kInner, kDirect
};
constexpr uint32_t kInner = 1u << 30;    // no pixel of the rectangle is below the floor
constexpr uint32_t kDirect = 1u << 31;   // every pixel's exponential by itself

// Largest |qyy| of a component whose rows are chained (R rows of a thread).
template <int R>
constexpr float kMaxCurve = R > 2 ? 0.75f : 1.0f;

// Largest exponent of a component (a dx^2 + b dx dy + c dy^2, concave) over
// the box [x0, x1] x [y0, y1] about its centre.
__device__ __forceinline__ float max_exponent(float a, float b, float c, float x0, float x1,
                                              float y0, float y1) {
    if (x0 <= 0.f && x1 >= 0.f && y0 <= 0.f && y1 >= 0.f) return 0.f;
    auto e = [&](float x, float y) { return fmaf(x, fmaf(a, x, b * y), c * y * y); };
    const float ky = __fdividef(-0.5f * b, c), kx = __fdividef(-0.5f * b, a);
    float m = e(x0, fminf(fmaxf(ky * x0, y0), y1));
    m = fmaxf(m, e(x1, fminf(fmaxf(ky * x1, y0), y1)));
    m = fmaxf(m, e(fminf(fmaxf(kx * y0, x0), x1), y0));
    return fmaxf(m, e(fminf(fmaxf(kx * y1, x0), x1), y1));
}

// Persistent over tiles of 32 x TH pixels; a thread holds CP pairs of adjacent
// columns of R consecutive rows.
//
// Bound: issue slots and ex2.  Down a column the exponential follows
//   E(y + 1) = E(y) R(y), R(y + 1) = R(y) Q, Q = 2^(2 qyy),
// so eight pixels take four ex2 (E and R of the first row in two columns) and
// five packed multiplies instead of eight ex2 and their exponents.  Three
// steps from an anchor add about 3 ulp; with the centre split into pixel and
// fraction the result is nearer to FP64 than eight separate ex2 from a
// rounded centre.  A first row so far out that E flushes to zero (2^-126) must
// have no later row above the floor (2^-72.1 of the component's peak): with
// four rows that holds up to |qyy| = 0.79 (sqrt(126) - 3 sqrt(|qyy|) >=
// sqrt(72.1)), so components above 0.75 (variances below 0.96 px^2; with two
// rows 1 and 0.72) take every pixel's ex2.  Exponents below the floor count as 0 (c_gauss_2d_grid skips Mahalanobis^2
// >= 100), tested only where the component reaches it inside the rectangle.
template <int TH, int CP, int R>
__global__ void __launch_bounds__(16 * TH / (CP * R), (CP == 1 ? 1024 : 768) / (16 * TH / (CP * R)))
scene_render_kernel(const tb_scene_item* __restrict__ items, int n_items,
                    const tb_scene_image* __restrict__ images, int n_images, int64_t n_tiles,
                    int64_t max_pairs,
                    const double* __restrict__ amp, const double* __restrict__ mean,
                    const double* __restrict__ var, const int32_t* __restrict__ offsets,
                    const int32_t* __restrict__ list, float* __restrict__ out, int mode,
                    int32_t* counter, tb_status* st) {
    constexpr int kThreads = 16 * TH / (CP * R);
    constexpr int kWarps = kThreads / 32;
    constexpr int kWarpRows = 2 * CP * R;      // rows a warp covers, 32 columns wide
    __shared__ SceneC comps[kThreads];
    __shared__ int ids[kCap];
    __shared__ int raw[kCap];
    __shared__ int prefK[kCap + 1];
    __shared__ int64_t slot;
    __shared__ int img_idx;
    __shared__ int warp_count[kWarps];
    __shared__ int warp_tot[32];

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int x0 = 2 * CP * (lane % (16 / CP)), y0 = kWarpRows * warp + R * (lane / (16 / CP));

    // More overlaps than the list holds: the fill dropped some, so no tile
    // list can be trusted (tb_scene_render reports it from the fill pass).
    if ((int64_t)offsets[n_tiles] > max_pairs) return;

    for (;;) {
        const int64_t u = tb::next_unit(counter, &slot);
        if (u >= n_tiles) break;
        if (tid == 0) {
            int lo = 0, hi = n_images - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (images[mid].tile0 <= u) lo = mid; else hi = mid - 1;
            }
            img_idx = lo;
        }
        __syncthreads();
        const tb_scene_image im = images[img_idx];
        const int tiles_x = (im.W + TB_MOG_TILE - 1) / TB_MOG_TILE;
        const int64_t t = u - im.tile0;
        const int ox = (int)(t % tiles_x) * TB_MOG_TILE;
        const int oy = (int)(t / tiles_x) * TH;
        const int tw = min(TB_MOG_TILE, im.W - ox);
        const int th = min(TH, im.H - oy);
        if (tw <= 0 || th <= 0) {   // a tile index beyond its image
            if (tid == 0) tb::report(st, TB_STATUS_BAD_ITEM, img_idx, (int)t);
            continue;
        }

        f32x2 acc[R][CP], part[R][CP];
#pragma unroll
        for (int j = 0; j < R; j++)
#pragma unroll
            for (int p = 0; p < CP; p++) acc[j][p] = part[j][p] = 0ull;

        const int beg = offsets[u];
        const int n = offsets[u + 1] - beg;
        for (int cb = 0; cb < n; cb += kCap) {
            const int m = min(kCap, n - cb);
            for (int q = tid; q < m; q += kThreads) {
                const int v = list[beg + cb + q];
                // an index outside the item table is reported and becomes a
                // distinct negative placeholder with no components
                if (v < 0 || v >= n_items) tb::report(st, TB_STATUS_BAD_ITEM, v, -4);
                raw[q] = (v < 0 || v >= n_items) ? -1 - q : v;
            }
            __syncthreads();
            // rank sort (ids in one tile are distinct): catalog order
            for (int q = tid; q < m; q += kThreads) {
                const int v = raw[q];
                int r = 0;
                for (int z = 0; z < m; z++) r += raw[z] < v;
                ids[r] = v;
            }
            __syncthreads();
            // exclusive prefix of component counts over the sorted items, a
            // few consecutive items per thread
            {
                constexpr int kPer = kCap / kThreads;
                int sum = 0;
                for (int z = 0; z < kPer; z++) {
                    const int q = kPer * tid + z;
                    if (q >= m) break;
                    prefK[q] = sum;
                    sum += ids[q] >= 0 ? items[ids[q]].K : 0;
                }
                int total;
                const int ex = block_exclusive_scan(sum, warp_tot, total);
                for (int z = 0; z < kPer; z++) {
                    const int q = kPer * tid + z;
                    if (q >= m) break;
                    prefK[q] += ex;
                }
                if (tid == 0) prefK[m] = total;
            }
            __syncthreads();
            const int total = prefK[m];

            int cur = -1;
            bool rows = false;          // some row of this warp is in the source's rectangle
            unsigned in_cols = 0u, in_rows = 0u;   // this thread's columns and rows that are
            // the finished source's patch, inside its rectangle
            auto add_part = [&]() {
#pragma unroll
                for (int j = 0; j < R; j++)
#pragma unroll
                    for (int p = 0; p < CP; p++) {
                        const float2 v = unpack(part[j][p]);
                        const unsigned in = (in_rows >> j) & 1u ? in_cols >> (2 * p) : 0u;
                        acc[j][p] = add2(acc[j][p], pack(in & 1u ? v.x : 0.f, in & 2u ? v.y : 0.f));
                        part[j][p] = 0ull;
                    }
            };

            for (int base = 0; base < total; base += kThreads) {
                const int g = base + tid;
                bool keep = false;
                SceneC c;
                if (g < total) {
                    // the item holding global component g: largest q with prefK[q] <= g
                    int lo = 0, hi = m - 1;
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (prefK[mid] <= g) lo = mid; else hi = mid - 1;
                    }
                    const int ii = ids[lo];
                    const tb_scene_item& it = items[ii];
                    const int k = g - prefK[lo];
                    const int ci = it.c0 + k;
                    const int rx0 = max(it.x0 - ox, 0), rx1 = min(it.x0 + it.w - ox, tw);
                    const int ry0 = max(it.y0 - oy, 0), ry1 = min(it.y0 + it.h - oy, th);
                    const double a = amp[ci];
                    const double v0 = var[4 * ci], v3 = var[4 * ci + 3];
                    const double vxy = 0.5 * (var[4 * ci + 1] + var[4 * ci + 2]);
                    const double det = v0 * v3 - vxy * vxy;
                    const double ri = rsqrt(det);
                    const double sc = (double)it.scale * a * (0.5 / TB_PI) * ri;
                    const double f = (-0.5 * TB_LOG2E) * ri * ri;
                    const float fl = (float)((double)it.floor * TB_LOG2E);
                    const double mx = (mean[2 * ci] + it.fx) - (double)ox;
                    const double my = (mean[2 * ci + 1] + it.fy) - (double)oy;
                    const double mxi = rint(mx), myi = rint(my);
                    c.qxx[0] = c.qxx[1] = (float)(v3 * f);
                    c.qxy[0] = c.qxy[1] = (float)(-2.0 * vxy * f);
                    c.qyy = (float)(v0 * f);
                    c.Q[0] = c.Q[1] = exp2f((float)(2.0 * v0 * f));
                    c.s[0] = c.s[1] = (float)sc;
                    c.thr = exp2f(fl);
                    c.ix = (float)mxi;
                    c.fx = (float)(mx - mxi);
                    c.iy = (float)myi;
                    c.fy = (float)(my - myi);
                    c.src = lo;
                    c.rect = (uint32_t)rx0 | ((uint32_t)rx1 << 6) | ((uint32_t)ry0 << 12) |
                             ((uint32_t)ry1 << 19);
                    const bool finite = det > 0.0 && isfinite(sc) && isfinite(f) &&
                                        isfinite(mx) && isfinite(my);
                    if (!finite) {
                        tb::report(st, TB_STATUS_NONFINITE, ii, k);
                    } else if (a != 0.0 && rx0 < rx1 && ry0 < ry1 && v0 > 0.0) {
                        // exponents over the part of the tile inside the
                        // rectangle: all below the floor (with a margin), or none
                        const float bx0 = (float)(rx0 - mx), bx1 = (float)(rx1 - 1 - mx);
                        const float by0 = (float)(ry0 - my), by1 = (float)(ry1 - 1 - my);
                        const float qa = c.qxx[0], qb = c.qxy[0], qc = c.qyy;
                        keep = !(max_exponent(qa, qb, qc, bx0, bx1, by0, by1) < fl - 1.f);
                        auto e = [&](float x, float y) { return fmaf(x, fmaf(qa, x, qb * y), qc * y * y); };
                        const float lowest = fminf(fminf(e(bx0, by0), e(bx1, by0)),
                                                   fminf(e(bx0, by1), e(bx1, by1)));
                        if (lowest > fl + 1.f) c.rect |= kInner;
                        if (!(fabsf(qc) <= kMaxCurve<R>) || fl < -73.f) c.rect |= kDirect;
                    }
                }
                // order-preserving compaction of the kept components
                const unsigned ballot = __ballot_sync(0xffffffffu, keep);
                if (lane == 0) warp_count[warp] = __popc(ballot);
                __syncthreads();
                int wbase = 0, kept = 0;
#pragma unroll
                for (int w = 0; w < kWarps; w++) {
                    wbase += (w < warp) ? warp_count[w] : 0;
                    kept += warp_count[w];
                }
                if (keep) comps[wbase + __popc(ballot & ((1u << lane) - 1u))] = c;
                __syncthreads();

                for (int q = 0; q < kept; q++) {
                    const SceneC& g2 = comps[q];
                    const float4 head = *reinterpret_cast<const float4*>(&g2.qyy);
                    const float qyy = head.x, thr = head.y;
                    const int src = __float_as_int(head.z);
                    const uint32_t rect = __float_as_uint(head.w);
                    if (src != cur) {
                        if (rows) add_part();
                        cur = src;
                        const int rx0 = rect & 63, rx1 = (rect >> 6) & 63;
                        const int ry0 = (rect >> 12) & 127, ry1 = (rect >> 19) & 127;
                        rows = kWarpRows * warp < ry1 && kWarpRows * (warp + 1) > ry0;
                        in_cols = in_rows = 0u;
#pragma unroll
                        for (int i = 0; i < 2 * CP; i++)
                            if (x0 + i >= rx0 && x0 + i < rx1) in_cols |= 1u << i;
#pragma unroll
                        for (int j = 0; j < R; j++)
                            if (y0 + j >= ry0 && y0 + j < ry1) in_rows |= 1u << j;
                    }
                    if (!rows) continue;
                    const ulonglong2 pq = *reinterpret_cast<const ulonglong2*>(g2.qxx);
                    const ulonglong2 ps = *reinterpret_cast<const ulonglong2*>(g2.Q);
                    const float4 ctr = *reinterpret_cast<const float4*>(&g2.ix);
                    const float dx0 = ((float)x0 - ctr.x) - ctr.y;
                    const float dy = ((float)y0 - ctr.z) - ctr.w;
                    f32x2 A[CP], B[CP];
#pragma unroll
                    for (int p = 0; p < CP; p++) {
                        const f32x2 dx = pack(dx0 + (float)(2 * p), dx0 + (float)(2 * p + 1));
                        A[p] = mul2(mul2(pq.x, dx), dx);
                        B[p] = mul2(pq.y, dx);
                    }
                    if (rect & kDirect) {
#pragma unroll
                        for (int p = 0; p < CP; p++) {
                            const float2 a2 = unpack(A[p]), b2 = unpack(B[p]);
#pragma unroll
                            for (int j = 0; j < R; j++) {
                                const float dj = dy + (float)j;
                                const float ea = tb::ex2(fmaf(dj, fmaf(qyy, dj, b2.x), a2.x));
                                const float eb = tb::ex2(fmaf(dj, fmaf(qyy, dj, b2.y), a2.y));
                                part[j][p] = fma2(ps.y, pack(ea >= thr ? ea : 0.f,
                                                             eb >= thr ? eb : 0.f), part[j][p]);
                            }
                        }
                        continue;
                    }
                    // first row: E = 2^(A + dy (B + qyy dy)), R = 2^(B + qyy (2 dy + 1))
                    const float u1 = qyy * dy, u2 = fmaf(2.f, u1, qyy);
                    f32x2 E[CP], F[CP];
#pragma unroll
                    for (int p = 0; p < CP; p++) {
                        const float2 e0 = unpack(fma2(pack(dy, dy), add2(B[p], pack(u1, u1)), A[p]));
                        const float2 r0 = unpack(add2(B[p], pack(u2, u2)));
                        E[p] = pack(tb::ex2(e0.x), tb::ex2(e0.y));
                        // (a ratio above 2^126 starts from E = 0: kept finite)
                        F[p] = pack(tb::ex2(fminf(r0.x, 126.f)), tb::ex2(fminf(r0.y, 126.f)));
                    }
                    if (rect & kInner) {
#pragma unroll
                        for (int j = 0; j < R; j++)
#pragma unroll
                            for (int p = 0; p < CP; p++) {
                                part[j][p] = fma2(ps.y, E[p], part[j][p]);
                                if (j + 1 < R) E[p] = mul2(E[p], F[p]);
                                if (j + 2 < R) F[p] = mul2(F[p], ps.x);
                            }
                    } else {
#pragma unroll
                        for (int j = 0; j < R; j++)
#pragma unroll
                            for (int p = 0; p < CP; p++) {
                                const float2 v = unpack(E[p]);
                                part[j][p] = fma2(ps.y, pack(v.x >= thr ? v.x : 0.f,
                                                             v.y >= thr ? v.y : 0.f), part[j][p]);
                                if (j + 1 < R) E[p] = mul2(E[p], F[p]);
                                if (j + 2 < R) F[p] = mul2(F[p], ps.x);
                            }
                    }
                }
                __syncthreads();   // comps is overwritten by the next pass
            }
            if (rows) add_part();
        }

        const int64_t ldo = im.ldo > 0 ? im.ldo : im.W;
#pragma unroll
        for (int j = 0; j < R; j++) {
            if (y0 + j >= th) continue;
            float* o = out + im.out_off + (int64_t)(oy + y0 + j) * ldo + (ox + x0);
#pragma unroll
            for (int p = 0; p < CP; p++) {
                const float2 v = unpack(acc[j][p]);
                if (x0 + 2 * p < tw) o[2 * p] = mode == TB_MOG_ACCUM ? o[2 * p] + v.x : v.x;
                if (x0 + 2 * p + 1 < tw)
                    o[2 * p + 1] = mode == TB_MOG_ACCUM ? o[2 * p + 1] + v.y : v.y;
            }
        }
    }
}

template <int TH, int CP, int R>
int launch_render(const tb_scene_item* items, int n_items, const tb_scene_image* images,
                  int n_images, int64_t n_tiles, int64_t max_pairs, const double* a, const double* m,
                  const double* v, const int32_t* offsets, const int32_t* list, float* out, int mode,
                  int32_t* counter, tb_status* st, cudaStream_t s) {
    constexpr int kThreads = 16 * TH / (CP * R);
    // the CTAs per SM of the kernel's launch bounds
    const int64_t want = (int64_t)tb::num_sms() * ((CP == 1 ? 1024 : 768) / kThreads);
    const int grid = (int)(n_tiles < want ? n_tiles : want);
    scene_render_kernel<TH, CP, R><<<grid, kThreads, 0, s>>>(
        items, n_items, images, n_images, n_tiles, max_pairs, a, m, v, offsets, list, out, mode,
        counter, st);
    return cudaGetLastError() == cudaSuccess ? TB_OK : TB_ERR_LAUNCH;
}

// Pixels per thread by the number of tiles: sixteen spend the fewest
// instructions per pixel (16,384 tiles: 724 us, against 789 at eight and 1,089
// at four; 2,820 tiles: 178, 179, 218), but a few tiles are rendered sooner by
// more threads each (208 tiles: 70, 62, 57; 550 tiles: 78, 69, 69).
template <int TH, class... Args>
int dispatch_render(int64_t n_tiles, Args... args) {
    const int64_t sms = tb::num_sms();
    if (n_tiles >= 16 * sms) return launch_render<TH, 2, 4>(args...);
    if (n_tiles >= 3 * sms) return launch_render<TH, 1, 4>(args...);
    return launch_render<TH, 1, 2>(args...);
}

// Workspace layout (bytes, each section 256-aligned): the work counter and
// counts[n_tiles] int32 (cleared together), offsets[n_tiles + 1] int32, block
// sums int32, list[max_pairs] int32.
struct Workspace {
    int32_t* counts;
    int32_t* offsets;
    int32_t* bsum;
    int32_t* list;
    int32_t* counter;
    int64_t bytes;
};

inline int64_t align256(int64_t x) { return (x + 255) / 256 * 256; }

Workspace carve(void* base, int64_t n_tiles, int64_t max_pairs) {
    Workspace w;
    const int64_t nb = (n_tiles + kScanThreads - 1) / kScanThreads;
    int64_t o = 0;
    char* b = static_cast<char*>(base);
    w.counter = reinterpret_cast<int32_t*>(b + o);
    w.counts = w.counter + 1;
    o += align256(4 * (n_tiles + 1));
    w.offsets = reinterpret_cast<int32_t*>(b + o);
    o += align256(4 * (n_tiles + 1));
    w.bsum = reinterpret_cast<int32_t*>(b + o);
    o += align256(4 * (nb > 0 ? nb : 1));
    w.list = reinterpret_cast<int32_t*>(b + o);
    o += align256(4 * (max_pairs > 0 ? max_pairs : 1));
    w.bytes = o;
    return w;
}

}  // namespace

extern "C" int tb_scene_prep(const tb_scene_src* srcs, int32_t n, const tb_scene_image* images,
                             int32_t n_images, const double* psf_amp, const double* psf_mean,
                             const double* psf_var, const tb_profile_tables* tables,
                             tb_scene_item* items, double* comp_amp, double* comp_mean,
                             double* comp_var, int32_t comp_stride, void* stream) {
    if (n < 0 || n_images < 0) return TB_ERR_ARG;
    if (n == 0) return TB_OK;
    if (!srcs || !images || !psf_amp || !psf_mean || !psf_var || !tables || !items ||
        !comp_amp || !comp_mean || !comp_var)
        return TB_ERR_ARG;
    if (comp_stride < 1 || comp_stride > TB_MOG_MAX_K) return TB_ERR_SIZE;
    const int per_block = kPrepThreads / 32;
    scene_prep_kernel<<<(n + per_block - 1) / per_block, kPrepThreads, 0,
                        (cudaStream_t)stream>>>(srcs, n, images, n_images, psf_amp, psf_mean,
                                                psf_var, *tables, items, comp_amp, comp_mean,
                                                comp_var, comp_stride);
    return cudaGetLastError() == cudaSuccess ? TB_OK : TB_ERR_LAUNCH;
}

extern "C" int tb_scene_workspace(int64_t n_tiles, int64_t max_pairs, int64_t* bytes) {
    if (n_tiles < 0 || max_pairs < 0 || !bytes) return TB_ERR_ARG;
    if (n_tiles > 0x7ffffffeLL || max_pairs > 0x7fffffffLL) return TB_ERR_SIZE;
    *bytes = carve(nullptr, n_tiles, max_pairs).bytes;
    return TB_OK;
}

extern "C" int tb_scene_render(const tb_scene_item* items, int32_t n_items,
                               const tb_scene_image* images, int32_t n_images, int64_t n_tiles,
                               int32_t tile_h, const double* comp_amp, const double* comp_mean,
                               const double* comp_var, float* out, int32_t mode, void* workspace,
                               int64_t workspace_bytes, int64_t max_pairs, tb_status* status,
                               void* stream) {
    if (n_items < 0 || n_images < 0 || n_tiles < 0 || max_pairs < 0) return TB_ERR_ARG;
    if (mode != TB_MOG_STORE && mode != TB_MOG_ACCUM) return TB_ERR_ARG;
    if (tile_h != 16 && tile_h != 32 && tile_h != 64) return TB_ERR_SIZE;
    if (n_tiles > 0x7ffffffeLL || max_pairs > 0x7fffffffLL) return TB_ERR_SIZE;
    if (n_tiles == 0 || n_images == 0) return TB_OK;
    if (!images || !out || !workspace || (n_items > 0 && (!items || !comp_amp || !comp_mean ||
                                                           !comp_var)))
        return TB_ERR_ARG;
    const Workspace w = carve(workspace, n_tiles, max_pairs);
    if (workspace_bytes < w.bytes) return TB_ERR_SIZE;
    cudaStream_t s = (cudaStream_t)stream;
    if (status && cudaMemsetAsync(status, 0, sizeof(tb_status), s) != cudaSuccess)
        return TB_ERR_LAUNCH;
    if (cudaMemsetAsync(w.counter, 0, 4 * (n_tiles + 1), s) != cudaSuccess) return TB_ERR_LAUNCH;
    const int per_bin = kBinThreads / 32;
    const int nb_items = (n_items + per_bin - 1) / per_bin;
    if (n_items > 0) {
        scene_bin_kernel<false><<<nb_items, kBinThreads, 0, s>>>(
            items, n_items, images, n_images, n_tiles, tile_h, w.counts, nullptr, nullptr,
            max_pairs, status);
    }
    const int nb = (int)((n_tiles + kScanThreads - 1) / kScanThreads);
    scan_blocks_kernel<<<nb, kScanThreads, 0, s>>>(w.counts, n_tiles, w.offsets, w.bsum);
    if (nb > 1) {
        scan_sums_kernel<<<1, kScanThreads, 0, s>>>(w.bsum, nb, w.offsets, n_tiles);
        scan_add_kernel<<<nb, kScanThreads, 0, s>>>(w.offsets, n_tiles, w.bsum);
    }
    if (n_items > 0) {
        scene_bin_kernel<true><<<nb_items, kBinThreads, 0, s>>>(
            items, n_items, images, n_images, n_tiles, tile_h, w.counts, w.offsets, w.list,
            max_pairs, status);
    }
    if (cudaGetLastError() != cudaSuccess) return TB_ERR_LAUNCH;
    auto render = [&](auto... args) {
        return tile_h == 16 ? dispatch_render<16>(n_tiles, args...)
             : tile_h == 32 ? dispatch_render<32>(n_tiles, args...)
                            : dispatch_render<64>(n_tiles, args...);
    };
    return render(items, n_items, images, n_images, n_tiles, max_pairs, comp_amp, comp_mean,
                  comp_var, (const int32_t*)w.offsets, (const int32_t*)w.list, out, mode, w.counter,
                  status, s);
}
