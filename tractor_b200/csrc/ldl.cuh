// LDL^T of a small symmetric positive definite FP64 matrix by one CTA, and
// the triangular solves by one warp (blob_fit.cu's damped steps, lsq.cu's
// least-squares updates).
//
// Bound: the chain of columns.  Four columns at a time: every thread factors
// the 4 x 4 diagonal block itself and finishes one row of the panel, then the
// trailing tiles are updated by FP64 tensor-core products of rank 4 - two
// barriers per four columns and 256 multiply-adds per instruction.
#pragma once

#include "tb_common.cuh"

namespace tb {

__device__ __forceinline__ void mma884(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// 1 / d by Newton's iteration r <- r + r (1 - d r) from the hardware's
// 20-bit estimate (twice: past FP64's precision): a shorter chain than an
// IEEE division, and the refinement step covers its last bit.  For a d that is a
// positive normal number (a `pivot`).
__device__ __forceinline__ double reciprocal(double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    r = fma(r, fma(-d, r, 1.0), r);
    return fma(r, fma(-d, r, 1.0), r);
}

__device__ __forceinline__ bool pivot(double d) {
    return d >= 2.2250738585072014e-308 && isfinite(d);
}

// Factor storage: packed lower triangle by columns, padded to a multiple of
// 8 rows (identity): element (i, j) at L[packed_col(j, n) + i], n the padded
// size.
__host__ __device__ constexpr int packed_col(int j, int n) { return j * (2 * n - j - 1) / 2; }
__host__ __device__ constexpr int packed_size(int n) { return n * (n + 1) / 2; }

// Factors in place, right-looking: column k is left as d_k (diagonal) and
// c_ik = d_k l_ik below it, after subtracting c_ik c_jk / d_k from the trailing
// columns; rdg = 1 / d.  n a multiple of 8.  All kThreads threads of the CTA
// call it, after a barrier behind the fill.  0, or 1 + the first column whose
// pivot is not a positive finite normal number (the same in every thread).
template <int kThreads>
__device__ int ldl_factor(double* L, double* rdg, int n) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto col = [&](int j) { return L + packed_col(j, n); };
    for (int k0 = 0; k0 < n; k0 += 4) {
        const double *c0 = col(k0), *c1 = col(k0 + 1), *c2k = col(k0 + 2), *c3 = col(k0 + 3);
        // the 4 x 4 diagonal block, the same in every thread
        const double a10 = c0[k0 + 1], a20 = c0[k0 + 2], a30 = c0[k0 + 3];
        const double d0 = c0[k0], r0 = reciprocal(d0);
        const double d1 = c1[k0 + 1] - a10 * a10 * r0, r1 = reciprocal(d1);
        const double a21 = c1[k0 + 2] - a20 * a10 * r0, a31 = c1[k0 + 3] - a30 * a10 * r0;
        const double d2 = c2k[k0 + 2] - a20 * a20 * r0 - a21 * a21 * r1,
                     r2 = reciprocal(d2);
        const double a32 = c2k[k0 + 3] - a30 * a20 * r0 - a31 * a21 * r1;
        const double d3 = c3[k0 + 3] - a30 * a30 * r0 - a31 * a31 * r1 - a32 * a32 * r2;
        const double r3 = reciprocal(d3);
        if (!(pivot(d0) && pivot(d1) && pivot(d2) && pivot(d3)))
            return k0 + (!pivot(d0) ? 1 : !pivot(d1) ? 2 : !pivot(d2) ? 3 : 4);
        // the panel's other rows, one per thread
        const double l10 = a10 * r0, l20 = a20 * r0, l30 = a30 * r0;
        const double l21 = a21 * r1, l31 = a31 * r1, l32 = a32 * r2;
        for (int i = k0 + 4 + tid; i < n; i += kThreads) {
            const double e0 = c0[i];
            const double e1 = c1[i] - e0 * l10;
            const double e2 = c2k[i] - e0 * l20 - e1 * l21;
            const double e3 = c3[i] - e0 * l30 - e1 * l31 - e2 * l32;
            col(k0 + 1)[i] = e1;
            col(k0 + 2)[i] = e2;
            col(k0 + 3)[i] = e3;
        }
        __syncthreads();   // the panel's rows are complete, the diagonal block is read
        if (tid == 0) {
            col(k0 + 1)[k0 + 1] = d1;
            col(k0 + 1)[k0 + 2] = a21;
            col(k0 + 1)[k0 + 3] = a31;
            col(k0 + 2)[k0 + 2] = d2;
            col(k0 + 2)[k0 + 3] = a32;
            col(k0 + 3)[k0 + 3] = d3;
            rdg[k0] = r0;
            rdg[k0 + 1] = r1;
            rdg[k0 + 2] = r2;
            rdg[k0 + 3] = r3;
        }
        // trailing 8 x 8 tiles: row lane / 4, columns 2 (lane % 4) + {0, 1}
        const int base = (k0 + 4) / 8 * 8, T = (n - base) / 8;
        const int q = lane & 3;
        const double rq = -(q == 0 ? r0 : q == 1 ? r1 : q == 2 ? r2 : r3);
        const double* ck = col(k0 + q);
        int tj = 0, ti = warp;
        for (int e = warp; e < T * (T + 1) / 2; e += 3 * (kThreads / 32)) {
            // three tiles' loads before the first product
            double *p0[3], *p1[3], fa[3], fb[3], c[3][2];
            bool on0[3], on1[3];
#pragma unroll
            for (int t = 0; t < 3; t++) {
                on0[t] = on1[t] = e + t * (kThreads / 32) < T * (T + 1) / 2;
                fa[t] = fb[t] = c[t][0] = c[t][1] = 0.0;
                if (!on0[t]) continue;
                while (ti >= T) {   // the lower triangle's tile columns in turn
                    tj++;
                    ti += tj - T;
                }
                const int i = base + 8 * ti + (lane >> 2), j = base + 8 * tj + 2 * q;
                const int jb = base + 8 * tj + (lane >> 2);
                p0[t] = col(j) + i;
                p1[t] = col(j + 1) + i;
                // rows and columns above the trailing part (first tile only)
                // belong to the panel
                on0[t] = j >= k0 + 4 && i >= j;
                on1[t] = j + 1 >= k0 + 4 && i >= j + 1;
                if (i >= k0 + 4) fa[t] = ck[i];
                if (jb >= k0 + 4) fb[t] = ck[jb] * rq;
                if (on0[t]) c[t][0] = *p0[t];
                if (on1[t]) c[t][1] = *p1[t];
                ti += kThreads / 32;
            }
#pragma unroll
            for (int t = 0; t < 3; t++) mma884(c[t], fa[t], fb[t]);
#pragma unroll
            for (int t = 0; t < 3; t++) {
                if (on0[t]) *p0[t] = c[t][0];
                if (on1[t]) *p1[t] = c[t][1];
            }
        }
        __syncthreads();
    }
    return 0;
}

// y <- (L D L^T)^-1 y by the calling warp.
__device__ inline void ldl_solve(const double* L, const double* rdg, double* y, int n) {
    const int lane = threadIdx.x & 31;
    auto col = [&](int j) { return L + packed_col(j, n); };
    // L z = y, w = D^-1 z, L^T x = w in place in y, four columns at a
    // time: every lane solves the 4 x 4 triangle, then the lanes
    // update the remaining rows; l_ik = c_ik / d_k
    for (int k = 0; k < n; k += 4) {
        const double *c0 = col(k), *c1 = col(k + 1), *c2k = col(k + 2), *c3 = col(k + 3);
        const double z0 = y[k] * rdg[k];
        const double z1 = (y[k + 1] - c0[k + 1] * z0) * rdg[k + 1];
        const double z2 = (y[k + 2] - c0[k + 2] * z0 - c1[k + 2] * z1) * rdg[k + 2];
        const double z3 = (y[k + 3] - c0[k + 3] * z0 - c1[k + 3] * z1 -
                           c2k[k + 3] * z2) * rdg[k + 3];
        for (int i = k + 4 + lane; i < n; i += 32)
            y[i] -= (c0[i] * z0 + c1[i] * z1) + (c2k[i] * z2 + c3[i] * z3);
        __syncwarp();   // the triangle's rows are read
        if (lane < 4) y[k + lane] = lane == 0 ? z0 : lane == 1 ? z1 : lane == 2 ? z2 : z3;
        __syncwarp();
    }
    for (int k = n - 4; k >= 0; k -= 4) {
        const double *c0 = col(k), *c1 = col(k + 1), *c2k = col(k + 2);
        const double x3 = y[k + 3];
        const double x2 = y[k + 2] - c2k[k + 3] * rdg[k + 2] * x3;
        const double x1 = y[k + 1] - (c1[k + 2] * x2 + c1[k + 3] * x3) * rdg[k + 1];
        const double x0 = y[k] - (c0[k + 1] * x1 + c0[k + 2] * x2 + c0[k + 3] * x3) * rdg[k];
        for (int j = lane; j < k; j += 32) {
            const double* cj = col(j) + k;
            y[j] -= ((cj[0] * x0 + cj[1] * x1) + (cj[2] * x2 + cj[3] * x3)) * rdg[j];
        }
        __syncwarp();
        if (lane < 3) y[k + lane] = lane == 0 ? x0 : lane == 1 ? x1 : x2;
        __syncwarp();
    }
}

}  // namespace tb
