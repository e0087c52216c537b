// The FP64 form's CRT on the device: three residues -> a coefficient as three
// digits to base 2^56, the base its place is a power of, so that neighbouring
// coefficients add digit by digit; eight digit sums -> 14 words, with the carries
// inside a CTA resolved.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "carry.cuh"
#include "fp64mod.cuh"

namespace pic {

struct CrtDConsts {
    double p[3], pinv[3];
    double sw[3], swp[3];  // N^-1 mod p_q and its companion
    double i01, i01p;      // p0^-1 mod p1
    double i012, i012p;    // (p0 p1)^-1 mod p2
    double q012, q012p;    // p1^-1 mod p2 = p0 (p0 p1)^-1 mod p2
    double off[3];         // 2^140 mod p_q when every coefficient gets the offset 2^140, else 0; off[0] - 2 p0
    uint32_t c0, c01, cc;  // p_q = c_q 2^32 + 1: c0, c0 + c1 and c0 c1
};

// The constants at product length 2^k; offset: every coefficient gets 2^140.
CrtDConsts make_crtd(int k, bool offset);

// A residue |x| < 2^51 as an integer.
__device__ __forceinline__ int64_t dto_i64(double x)
{
    return __double_as_longlong(__dadd_rn(x, kDblRound)) - 0x4338000000000000ll;
}

constexpr uint64_t kMask56 = ((uint64_t)1 << 56) - 1;

// Garner's CRT on three FP64 residues (|y| < 2^51): x = r0 + p0 (v1 + p1 v2)
// with r_q = y_q N^-1 (+ offset) mod p_q, as digits x = d0 + d1 2^56 + d2 2^112
// (x < 2^141, d2 < 2^29).  r0 and v1 are taken at or below zero (no comparisons):
// x - r0 and (x - r0) / p0 - v1 are then nonnegative and far below the primes'
// products, so v2, the only digit brought into [0, p2), is the true one.  With
// p_q = c_q 2^32 + 1 the sum is (r0 + v1 + v2) + (c0 v1 + (c0 + c1) v2) 2^32 +
// c0 c1 v2 2^64: products by 15-, 16- and 30-bit numbers.
__device__ __forceinline__ void crt3d(const CrtDConsts& C, double y0, double y1, double y2, uint64_t& d0, uint64_t& d1,
                                      uint32_t& d2)
{
    const double r0 = __dadd_rn(dmul_tw(y0, C.sw[0], C.swp[0], C.p[0]), C.off[0]);  // (-2.75 p0, -0.25 p0]
    const double r1 = __dadd_rn(dmul_tw(y1, C.sw[1], C.swp[1], C.p[1]), C.off[1]);
    const double r2 = __dadd_rn(dmul_tw(y2, C.sw[2], C.swp[2], C.p[2]), C.off[2]);
    const double v1 = __dadd_rn(dmul_tw(__dadd_rn(r1, -r0), C.i01, C.i01p, C.p[1]), -C.p[1]);  // (-1.75, -0.25] p1
    const double a = dmul_tw(__dadd_rn(r2, -r0), C.i012, C.i012p, C.p[2]);
    const double b = dmul_tw(v1, C.q012, C.q012p, C.p[2]);
    const double v2 = dcanon(dreduce(__dadd_rn(a, -b), C.p[2], C.pinv[2]), C.p[2]);
    const int64_t V1 = dto_i64(v1), V2 = dto_i64(v2);
    const int64_t A = dto_i64(r0) + V1 + V2;                                          // |A| < 2^50
    const int64_t B = V1 * (int64_t)C.c0 + V2 * (int64_t)C.c01;                       // in (-2^63, 2^63)
    const uint64_t lo = (uint64_t)(uint32_t)V2 * C.cc, hi = (uint64_t)(V2 >> 32) * C.cc + (lo >> 32);  // c0 c1 v2
    const uint64_t D = (hi << 32) | (uint32_t)lo;                                     // its low 64 bits
    // digits, the parts' signs carried upwards
    const int64_t t0 = A + (int64_t)(((uint64_t)B & 0xffffffu) << 32);
    d0 = (uint64_t)t0 & kMask56;
    const int64_t t1 = (t0 >> 56) + (B >> 24) + (int64_t)((D << 8) & kMask56);
    d1 = (uint64_t)t1 & kMask56;
    d2 = (uint32_t)((t1 >> 56) + (int64_t)(hi >> 16));
}

// A CTA's coefficients' digits in shared memory, the i-th at crt_slot(i).  All
// threads take coefficients in turn, so the residues are read coalesced and no
// thread waits for a neighbour; the groups are then assembled from shared
// memory, whose padding keeps threads eight coefficients apart in different
// banks.
__host__ __device__ constexpr int crt_slot(int i) { return i + (i >> 3); }

template <int XS>
struct CrtDigits {
    uint64_t d0[XS], d1[XS];
    uint32_t d2[XS];
};

// Coefficients at[i], i < n: index(i) names the i-th (negative or past the last
// one: zero), res(j, y0, y1, y2) gives its residues, ahead of their use;
// fix(j, y0, y1, y2) may change them when they have arrived.
template <int XS, class Index, class Res, class Fix>
__device__ __forceinline__ void crt_coefs(CrtDigits<XS>& X, int n, const CrtDConsts& C, const Index& index,
                                          const Res& res, const Fix& fix)
{
    // the next coefficient's residues are on the way while one is converted
    double n0 = 0, n1 = 0, n2 = 0;
    int64_t nj = (int)threadIdx.x < n ? index((int)threadIdx.x) : -1;
    if (nj >= 0) res(nj, n0, n1, n2);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double y0 = n0, y1 = n1, y2 = n2;
        const int64_t j = nj;
        nj = i + (int)blockDim.x < n ? index(i + (int)blockDim.x) : -1;
        if (nj >= 0) res(nj, n0, n1, n2);
        uint64_t d0 = 0, d1 = 0;
        uint32_t d2 = 0;
        if (j >= 0) {
            fix(j, y0, y1, y2);
            crt3d(C, y0, y1, y2, d0, d1, d2);
        }
        const int at = crt_slot(i);
        X.d0[at] = d0;
        X.d1[at] = d1;
        X.d2[at] = d2;
    }
}

// The eight base-2^56 digits of a group whose first coefficient is the CTA's
// i-th (i >= 3: the three before it are in place), the carries of the digit sums
// (at most 2) added in, with one carry out of each (bit 56) still to pass on.
template <int XS>
__device__ __forceinline__ void crt_group(const CrtDigits<XS>& X, int i, uint64_t (&t)[8])
{
    uint64_t a1 = X.d1[crt_slot(i - 2)];
    uint32_t a2 = X.d2[crt_slot(i - 3)], b2 = X.d2[crt_slot(i - 2)];
    uint64_t below = X.d0[crt_slot(i - 1)] + a1 + a2;  // the digit sum before the group
    a1 = X.d1[crt_slot(i - 1)];
    a2 = b2;
    b2 = X.d2[crt_slot(i - 1)];
#pragma unroll
    for (int u = 0; u < 8; u++) {
        const int at = crt_slot(i + u);
        const uint64_t sum = X.d0[at] + a1 + a2;
        t[u] = (sum & kMask56) + (below >> 56);
        below = sum;
        if (u < 7) {
            a1 = X.d1[at];
            a2 = b2;
            b2 = X.d2[at];
        }
    }
}

// Digits -> words W[14 threadIdx.x ..] in shared memory (which may be where the
// digits came from: every thread has read them before any writes), the carries
// of the whole CTA resolved in thread order; thread 0 writes the CTA's (G, P).
// A thread with `end` set drops its carry out (the last of a product).  Ends
// with a barrier; the caller copies the words out in runs, whole sectors at a
// time, where a thread's own 14 words would go to L2 in four-byte pieces.
__device__ __forceinline__ void digits_to_words(uint64_t (&t)[8], bool any, bool end, uint32_t* W, uint32_t* agg_slot)
{
    uint32_t gp = kGPIdentity;
    if (any) {
        uint64_t c = 0, all = kMask56;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const uint64_t v = t[u] + c;
            c = v >> 56;
            t[u] = v & kMask56;
            all &= t[u];
        }
        gp = end ? 0u : (uint32_t)c | ((uint32_t)(all == kMask56) << 1);
    }
    uint32_t total;
    const uint32_t cin = block_gp_scan(gp, &total) & 1u;
    if (threadIdx.x == 0) *agg_slot = total;
    if (any) {
        if (cin) {
            uint64_t c = 1;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const uint64_t v = t[u] + c;
                c = v >> 56;
                t[u] = v & kMask56;
            }
        }
        uint32_t* w = W + 14 * threadIdx.x;
#pragma unroll
        for (int i = 0; i < 14; i++) {
            const int bit = 32 * i, u = bit / 56, r = bit % 56;
            uint64_t v = t[u] >> r;
            if (r > 24 && u + 1 < 8) v |= t[u + 1] << (56 - r);
            w[i] = (uint32_t)v;
        }
    }
    __syncthreads();
}

}  // namespace pic
