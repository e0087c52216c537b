/* Enough of CUDA's device language for a host compiler to run the FP64 form's
 * headers as they are: round-to-nearest intrinsics on IEEE doubles (build with
 * -ffp-contract=off).  A quotient's rounding constant (1.5 * 2^52) must leave the
 * sum in [2^52, 2^53), where it rounds to an integer: otherwise shim_bad counts. */
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __restrict__ __restrict

static long shim_bad;

struct ulonglong2 { unsigned long long x, y; };
typedef void* cudaStream_t;
struct dim3_shim { unsigned x, y, z; };
static dim3_shim threadIdx, blockIdx;

static inline double __longlong_as_double(long long v) { double d; memcpy(&d, &v, 8); return d; }
static inline long long __double_as_longlong(double d) { long long v; memcpy(&v, &d, 8); return v; }
static inline double __hiloint2double(int hi, int lo)
{
    return __longlong_as_double((long long)(((unsigned long long)(unsigned)hi << 32) | (unsigned)lo));
}
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __fma_rn(double a, double b, double c)
{
    const double r = fma(a, b, c);
    if (c == 6755399441055744.0 && !(r >= 4503599627370496.0 && r < 9007199254740992.0)) shim_bad++;
    return r;
}
template <class T>
static inline T __ldg(const T* p) { return *p; }
static inline unsigned __brev(unsigned v)
{
    unsigned r = 0;
    for (int i = 0; i < 32; i++) r |= ((v >> i) & 1u) << (31 - i);
    return r;
}
static inline void __syncthreads() {}
