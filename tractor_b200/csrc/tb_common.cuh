// Shared device helpers for the tractor_b200 kernels (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "tractor_b200.h"

#define TB_LOG2E 1.4426950408889634
#define TB_PI 3.14159265358979323846

namespace tb {

// 2^e in FP64 for |e| < 1000 by the table-driven scheme of Tang (ACM TOMS
// 15(2), 1989): n = rint(16 e), r = e - n / 16 exactly (|r| <= 1/32),
// 2^e = 2^(n div 16) T[n mod 16] 2^r with T[j] = 2^(j / 16) and a polynomial
// of degree 6 for 2^r; relative error below 4e-16.  Ten FP64 operations.  The
// 16 table entries lie in 16 different pairs of shared-memory banks, so the
// lookups of a warp never conflict.
constexpr int kExpTab = 16;

__device__ __forceinline__ void exp2_tab_init(double* tab) {
    if (threadIdx.x < kExpTab) tab[threadIdx.x] = exp2((double)threadIdx.x / kExpTab);
}

// (2^r - 1) / r interpolated at the six Chebyshev nodes of |r| <= 1/32 (2^r to
// 1.5e-17; the Taylor sum of that degree is off by 4.5e-16 there).
__device__ __forceinline__ double exp2_poly(double r) {
    double p = 1.5403723980749256e-04;
    p = fma(p, r, 1.3333781576784268e-03);
    p = fma(p, r, 9.6181291069195370e-03);
    p = fma(p, r, 5.5504108656639302e-02);
    p = fma(p, r, 2.4022650695910075e-01);
    return fma(p, r, 6.9314718055994573e-01);
}

__device__ __forceinline__ double exp2_tab(double e, const double* tab) {
    const double magic = 6755399441055744.0;   // 1.5 x 2^52: rounds to an integer in the low word
    const double t = fma(e, (double)kExpTab, magic);
    const unsigned n = __double2loint(t);
    const double r = fma(t - magic, -1.0 / kExpTab, e);
    const double T = tab[n & (kExpTab - 1)];
    const double y = fma(T * r, exp2_poly(r), T);
    return __hiloint2double((int)(__double2hiint(y) + ((n & ~15u) << 16)), __double2loint(y));
}

// The same with the table's entries in two parts (tab[j] = (T[j], 2^(j/16) -
// T[j])), so that only 2^e's own rounding is left of their error: relative error
// below 1.3e-16 where e itself is exact.  One operation more.
static __device__ const double2 kExp2Parts[kExpTab] = {
    {1.0, 0.0},
    {1.0442737824274138, 8.5518897055379649e-17},
    {1.0905077326652577, -3.0467820798124711e-17},
    {1.1387886347566916, 8.9128126760254078e-17},
    {1.189207115002721, 3.9820152314656461e-17},
    {1.241857812073484, 4.6580275918369368e-17},
    {1.2968395546510096, 2.5382502794888315e-17},
    {1.3542555469368927, 7.7009483798029895e-17},
    {1.4142135623730951, -9.6672933134529135e-17},
    {1.4768261459394993, -3.4839945568927958e-17},
    {1.5422108254079407, 7.9498348096976209e-17},
    {1.6104903319492543, 2.4707192569797888e-17},
    {1.681792830507429, 8.1990100205814965e-17},
    {1.7562521603732995, 2.9601406954488733e-17},
    {1.8340080864093424, 3.2831072242456272e-17},
    {1.9152065613971474, -1.0619946056195963e-16},
};

__device__ __forceinline__ void exp2_tab_init(double2* tab) {
    if (threadIdx.x < kExpTab) tab[threadIdx.x] = kExp2Parts[threadIdx.x];
}

__device__ __forceinline__ double exp2_tab(double e, const double2* tab) {
    const double magic = 6755399441055744.0;
    const double t = fma(e, (double)kExpTab, magic);
    const unsigned n = __double2loint(t);
    const double r = fma(t - magic, -1.0 / kExpTab, e);
    const double2 T = tab[n & (kExpTab - 1)];
    const double y = T.x + fma(T.x * r, exp2_poly(r), T.y);
    return __hiloint2double((int)(__double2hiint(y) + ((n & ~15u) << 16)), __double2loint(y));
}

// 2^x on the SFU (MUFU.EX2), flushing denormal results to zero.
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Records the first failure of a launch in a device status word.
__device__ __forceinline__ void report(tb_status* st, int code, int item, int detail) {
    if (st == nullptr) return;
    if (atomicCAS(&st->code, 0, code) == 0) {
        st->item = item;
        st->detail = detail;
    }
    atomicAdd(&st->count, 1);
}

// Dynamic work distribution for persistent kernels: thread 0 takes the next
// unit from a global counter and broadcasts it through shared memory.
__device__ __forceinline__ int64_t next_unit(int32_t* counter, int64_t* slot) {
    __syncthreads();
    if (threadIdx.x == 0) *slot = (int64_t)atomicAdd(counter, 1);
    __syncthreads();
    return *slot;
}

inline int num_sms() {
    int n = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 148;
}

}  // namespace tb
