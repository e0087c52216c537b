// BigFloat linear kernels: windowed add/subtract (uadd/usub, BigFloat.cpp:
// 184-287), multiply by a 32-bit word (BigFloat.cpp:156-183), leading-zero
// strip and magnitude compare (BigFloat.cpp:123-147).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace pic {

// A magnitude as the reference stores it: words T[0..L) at exponent exp.
struct WordView {
    const uint32_t* T;
    int64_t exp;
    int64_t L;
};

// z[0..TL) = a(bot + c) +/- b(bot + c) with carries/borrows (the one out of word
// TL-1 is dropped).
void lin_addsub(uint32_t* z, size_t TL, const WordView& a, const WordView& b, int64_t bot, bool sub,
                cudaStream_t s);
// BigFloat's operations, on the library's stream; each waits for its result.
// z[0..TL) = a + b over the window, z[TL] = the carry out, which is returned.
uint32_t lin_add(uint32_t* z, size_t TL, const WordView& a, const WordView& b, int64_t bot);
// z[0..TL) = |a| - |b| over the window when |a| > |b|, else |b| - |a| (order 1,
// -1: known to the caller; 0: compared on the device).  Returns 1 + the index of
// the highest nonzero word of z; *order tells which of the two (1 or -1) where
// there is one.
size_t lin_diff(uint32_t* z, size_t TL, const WordView& a, const WordView& b, int64_t bot, int* order);
// z[0..L] = a[0..L) * x (z has L+1 words); returns z[L], which may be 0.
uint32_t lin_mul_u32(uint32_t* z, const uint32_t* a, size_t L, uint32_t x);
// p[0] = lo, and p[1] = hi when two are set (no host copy).
void lin_set(uint32_t* p, uint32_t lo, uint32_t hi, int n, cudaStream_t s);
// 1 + index of the highest nonzero word (0 if none).  Synchronises.
size_t lin_top_nonzero(const uint32_t* z, size_t n, cudaStream_t s);
// The comparison of |a| and |b| that needs no words: 1, -1, or 0 when their
// highest words are at one magnitude.
inline int lin_mag_order(const WordView& a, const WordView& b)
{
    const int64_t ma = a.exp + a.L, mb = b.exp + b.L;
    return ma > mb ? 1 : (ma < mb ? -1 : 0);
}
// Sign of |a| - |b| over aligned magnitudes.  Synchronises.
int lin_ucmp(const WordView& a, const WordView& b, cudaStream_t s);

}  // namespace pic
