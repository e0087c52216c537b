// Device code shared by the pass kernels: the prime of a batch item, the
// shared-memory swizzles, reading pieces from source words, the butterflies of
// both product forms, the register rounds of one group and their plans.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fp64mod.cuh"
#include "ntt.cuh"

namespace pic {

// Constant-index selection keeps the prime's fields in registers (a dynamic
// index into the kernel's parameter array would spill the array to local memory).
__device__ __forceinline__ PrimeDev pick_prime(const NttBatch& B, int tr)
{
    return tr < B.per_prime ? B.prime[0] : (tr < 2 * B.per_prime ? B.prime[1] : B.prime[2]);
}

#ifndef PIC_NTT_SWIZZLE
#define PIC_NTT_SWIZZLE 1
#endif
// Row layout swizzle: XOR bits 4..7 of an element's index into bits 0..3, a
// bijection on every row that spreads the small-stride rounds over all
// shared-memory banks.
__device__ __forceinline__ int swz(int e)
{
#if PIC_NTT_SWIZZLE
    return e ^ ((e >> 4) & 15);
#else
    return e;
#endif
}

struct LazyPrime {
    uint64_t p, p4;
    uint32_t c;  // p = c * 2^32 + 1
};

__device__ __forceinline__ LazyPrime lazy_prime(const PrimeDev& P)
{
    LazyPrime L;
    L.p = P.p;
    L.p4 = 4 * P.p;
    L.c = (uint32_t)(P.p >> 32);
    return L;
}

// Piece j of batch item tr from the item's child slot (SplitSrc), reduced to
// [0, 4p) (a 64-bit piece is below 9p for the lazy primes).
struct SrcRow {
    const uint32_t* x;
    uint32_t n;
};

__device__ __forceinline__ SrcRow src_row(const NttBatch& B, int tr)
{
    const size_t c = B.src.c0 + (size_t)(tr % B.per_prime);
    SrcRow r;
    r.x = B.src.words + c * (size_t)B.src.cap;
    r.n = B.src.len != nullptr ? B.src.len[c] : B.src.n;
    return r;
}

__device__ __forceinline__ uint64_t src_piece_raw(const NttBatch& B, const SrcRow& r, size_t j)
{
    const size_t wi = 2 * (B.src.first + j);
    uint64_t v = 0;
    if (wi < r.n) {
        v = __ldg(r.x + wi);
        if (wi + 1 < r.n) v |= (uint64_t)__ldg(r.x + wi + 1) << 32;
    }
    return v;
}

__device__ __forceinline__ uint64_t src_piece(const NttBatch& B, const SrcRow& r, size_t j, uint64_t p4)
{
    return piece_to_lazy(src_piece_raw(B, r, j), p4);
}

// Forward (DIF): operands and results in [0, 4p).
__device__ __forceinline__ void fbfly_dif(uint64_t& a, uint64_t& b, const ulonglong2 t, const LazyPrime& L)
{
    uint64_t x = a + b;
    x = x >= L.p4 ? x - L.p4 : x;
    b = shoup_approx32(a + L.p4 - b, t.x, t.y, L.c);
    a = x;
}

__device__ __forceinline__ void fbfly_unit_dif(uint64_t& a, uint64_t& b, const LazyPrime& L)
{
    uint64_t x = a + b;
    x = x >= L.p4 ? x - L.p4 : x;
    uint64_t y = a + L.p4 - b;
    y = y >= L.p4 ? y - L.p4 : y;
    a = x;
    b = y;
}

// Inverse (DIT): operands and results in [0, 8p).
__device__ __forceinline__ void fbfly_dit(uint64_t& a, uint64_t& b, const ulonglong2 t, const LazyPrime& L)
{
    const uint64_t u = shoup_approx32(b, t.x, t.y, L.c);
    const uint64_t x = a >= L.p4 ? a - L.p4 : a;
    a = x + u;
    b = x + L.p4 - u;
}

__device__ __forceinline__ void fbfly_unit_dit(uint64_t& a, uint64_t& b, const LazyPrime& L)
{
    const uint64_t x = a >= L.p4 ? a - L.p4 : a;
    const uint64_t y = b >= L.p4 ? b - L.p4 : b;
    a = x + y;
    b = x + L.p4 - y;
}

// Arithmetic of the fast passes.  ArithInt: lazy Shoup butterflies on 64-bit
// residues (lazy primes).  ArithDbl: FP64 butterflies (FP64 primes, values
// stored as the bits of doubles; a product with a twiddle lands below p).
// An FP64 forward sum grows only along the path that has met no product since
// the round began, so reduce_sum / reduce_unit name the few outputs of a
// round's last level that need a reduction (three FP64 instructions each).
// Radix-2 .. radix-8 rounds take and return |x| <= 2 p: inside a radix-8 round
// the values stay below 2^3 2 p = 16 p, and of its sums only outputs 0 (16 p)
// and 4 (4 p) are reduced, the others are sums of two products.  Radix-16
// rounds take and return |x| <= p, all sums reduced, again 16 p inside;
// 16 p < 2^51 for primes below 2^47.
// With the shorter product of dmul_w this took a product of 1,048,573 by
// 400,009 words from 186.4 to 179.8 us, one of 2^24-word operands from 4.03
// to 3.97 ms (the passes are bound by shared-memory traffic, not by FP64).
// FP64 inverse butterflies add at most p per level and never reduce: a pass
// of L levels over inputs below X ends below 2 X + (L - 1) p (15 p for a
// 13-level row pass over the merges' T1 +- T2, below 1.5 p).
struct ArithInt {
    using T = uint64_t;
    using Tw = ulonglong2;  // twiddle table entry: Shoup pair (w, w')
    using Ctx = LazyPrime;
    static __device__ __forceinline__ Ctx ctx(const PrimeDev& P) { return lazy_prime(P); }
    static __device__ __forceinline__ T ld(uint64_t v) { return v; }
    static __device__ __forceinline__ uint64_t st(T v) { return v; }
    template <bool RED>
    static __device__ __forceinline__ void dif(T& a, T& b, const ulonglong2 t, const Ctx& L) { fbfly_dif(a, b, t, L); }
    template <bool RED>
    static __device__ __forceinline__ void dif_unit(T& a, T& b, const Ctx& L) { fbfly_unit_dif(a, b, L); }
    static constexpr bool reduce_sum(int, int) { return false; }  // its butterflies keep [0, 4p) by themselves
    static constexpr bool reduce_unit(int, int) { return false; }
    static __device__ __forceinline__ void dit(T& a, T& b, const ulonglong2 t, const Ctx& L) { fbfly_dit(a, b, t, L); }
    static __device__ __forceinline__ void dit_unit(T& a, T& b, const Ctx& L) { fbfly_unit_dit(a, b, L); }
    // v * w (pass twiddle) into [0, 4p) from any 64-bit v
    static __device__ __forceinline__ T twiddle(T v, const ulonglong2 t, const Ctx& L)
    {
        return shoup_approx32(v, t.x, t.y, L.c);
    }
    // piece j of the item's child words, as a residue
    static __device__ __forceinline__ T piece(const NttBatch& B, const SrcRow& r, size_t j, const Ctx& L)
    {
        return src_piece(B, r, j, L.p4);
    }
};

struct ArithDbl {
    using T = double;
    using Tw = double;  // twiddle table entry: w; the companion is formed per use (dmul_w)
    struct Ctx {
        double p, pinv;
    };
    static __device__ __forceinline__ Ctx ctx(const PrimeDev& P) { return Ctx{P.pd, P.pinv}; }
    static __device__ __forceinline__ T ld(uint64_t v) { return dbits(v); }
    static __device__ __forceinline__ uint64_t st(T v) { return dstore(v); }
    // last level of a radix-2^B round: whether the sum at even output m, or
    // with unit twiddles both outputs at m and m + 1, must be reduced
    static constexpr bool reduce_sum(int B, int m) { return B == 4 || (m & 3) == 0; }
    static constexpr bool reduce_unit(int B, int m) { return reduce_sum(B, m); }
    template <bool RED>
    static __device__ __forceinline__ void dif(T& a, T& b, const Tw t, const Ctx& L)
    {
        const double s = __dadd_rn(a, b), d = __dadd_rn(a, -b);
        b = dmul_w(d, t, L.p, L.pinv);
        a = RED ? dreduce(s, L.p, L.pinv) : s;
    }
    template <bool RED>
    static __device__ __forceinline__ void dif_unit(T& a, T& b, const Ctx& L)
    {
        const double s = __dadd_rn(a, b), d = __dadd_rn(a, -b);
        a = RED ? dreduce(s, L.p, L.pinv) : s;
        b = RED ? dreduce(d, L.p, L.pinv) : d;
    }
    static __device__ __forceinline__ void dit(T& a, T& b, const Tw t, const Ctx& L)
    {
        const double u = dmul_w(b, t, L.p, L.pinv);
        b = __dadd_rn(a, -u);
        a = __dadd_rn(a, u);
    }
    static __device__ __forceinline__ void dit_unit(T& a, T& b, const Ctx&)
    {
        const double s = __dadd_rn(a, b);
        b = __dadd_rn(a, -b);
        a = s;
    }
    static __device__ __forceinline__ T twiddle(T v, const Tw t, const Ctx& L) { return dmul_w(v, t, L.p, L.pinv); }
    static __device__ __forceinline__ T piece(const NttBatch& B, const SrcRow& r, size_t j, const Ctx& L)
    {
        return dpiece56(src_piece56_raw(r.x, r.n, B.src.first + j), L.p, L.pinv);
    }
};

// The B levels of one group (elements base + j + m 2^LST, m < 2^B) with the
// per-level inner tables: the twiddle of butterfly u at group level l is
// root_(2^(B-l+LST))^(j + u 2^LST), pair 2^(B-l+LST-1) - 1 + j + u 2^LST, so
// lanes with consecutive j read consecutive pairs.
template <int B, bool INV, int LST, class A>
__device__ __forceinline__ void group_fast(typename A::T (&x)[1 << B], int j, const typename A::Ctx& L,
                                           const typename A::Tw* __restrict__ tw)
{
    static_assert(B + LST <= 13, "sub-block larger than the inner table");
    if (!INV) {
#pragma unroll
        for (int l = 0; l < B; l++) {
            const int hm = 1 << (B - 1 - l);
            if (l == B - 1 && LST == 0) {
#pragma unroll
                for (int m = 0; m < (1 << B); m += 2) {
                    if (A::reduce_unit(B, m)) A::template dif_unit<true>(x[m], x[m + 1], L);
                    else A::template dif_unit<false>(x[m], x[m + 1], L);
                }
                continue;
            }
#pragma unroll
            for (int m = 0; m < (1 << B); m++) {
                if (m & hm) continue;
                const int u = m & (hm - 1);
                const typename A::Tw t = __ldg(tw + ((1 << (B - l + LST - 1)) - 1) + j + (u << LST));
                if (l == B - 1 && A::reduce_sum(B, m)) A::template dif<true>(x[m], x[m + hm], t, L);
                else A::template dif<false>(x[m], x[m + hm], t, L);
            }
        }
    } else {
#pragma unroll
        for (int l = B - 1; l >= 0; l--) {
            const int hm = 1 << (B - 1 - l);
            if (l == B - 1 && LST == 0) {
#pragma unroll
                for (int m = 0; m < (1 << B); m += 2) A::dit_unit(x[m], x[m + 1], L);
                continue;
            }
#pragma unroll
            for (int m = 0; m < (1 << B); m++) {
                if (m & hm) continue;
                const int u = m & (hm - 1);
                A::dit(x[m], x[m + hm], __ldg(tw + ((1 << (B - l + LST - 1)) - 1) + j + (u << LST)), L);
            }
        }
    }
}

// Radix-2^RB rounds of a 2^LOGN transform (plus one smaller round when RB
// does not divide LOGN, at the smallest stride); forward rounds run from the
// largest stride down, inverse rounds the other way.
template <int LOGN, int RB = 3>
struct RoundPlan {
    static constexpr int NF = LOGN / RB, REM = LOGN % RB, NR = NF + (REM ? 1 : 0);
    template <int RR>
    struct At {
        static constexpr int B = RR < NF ? RB : REM;
        static constexpr int LB = LOGN - RB * RR;  // log2 sub-block size
        static constexpr int LST = LB - B;         // log2 stride inside a group
    };
};

// Radix-8 rounds with the remainder first (the largest stride).
template <int LC>
struct ColPlan {
    static constexpr int REM = LC % 3, NR = LC / 3 + (REM ? 1 : 0);
    template <int R>
    struct At {
        static constexpr int B = (R == 0 && REM) ? REM : 3;
        static constexpr int LB = R == 0 ? LC : LC - (REM ? REM : 3) - 3 * (R - 1);  // log2 sub-block
        static constexpr int LST = LB - B;                                           // log2 stride
    };
};

// Shared-memory place of element (row << LW) + column: half a warp that holds
// several rows eight apart falls in different banks.  Linear, like place().
template <int LW>
__host__ __device__ constexpr int col_place(int e)
{
    return LW == 2 ? e ^ (((e >> 5) & 3) << 2) : (LW == 3 ? e ^ (((e >> 6) & 1) << 3) : e);
}

// Place of element base + m (disjoint bits) from pb = col_place(base).
template <int LW>
__host__ __device__ constexpr int col_at(int pb, int m)
{
    return (pb ^ (col_place<LW>(m) & 15)) + (col_place<LW>(m) & ~15);
}

constexpr int brev3(int i, int bits) { return bits == 3 ? ((i & 1) << 2 | (i & 2) | i >> 2) : (bits == 2 ? ((i & 1) << 1 | i >> 1) : i); }

// Root of unity w_(2^lM)^e in Montgomery form from the two-level tables.
template <bool INV>
__device__ __forceinline__ uint64_t outer_root(const PrimeDev& P, uint64_t e, int lM)
{
    const uint64_t E = e << (P.K - lM);
    const uint64_t lo = E & ((1ull << P.S) - 1), hi = E >> P.S;
    const uint64_t* tl = INV ? P.olo_inv : P.olo_fwd;
    const uint64_t* th = INV ? P.ohi_inv : P.ohi_fwd;
    return mont_mul(__ldg(th + hi), __ldg(tl + lo), P.p, P.pinv_neg);
}

}  // namespace pic
