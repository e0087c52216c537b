// The FP64 form's CRT on the device: three residues -> a coefficient of three
// limbs, a group of eight coefficients at 56-bit offsets -> seven limbs, limb
// digits -> words with the carries inside a CTA resolved.
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
    double off[3];         // 2^140 mod p_q when every coefficient gets the offset 2^140, else 0
    uint64_t p0, p01_lo, p01_hi;
};

// The constants at product length 2^k; offset: every coefficient gets 2^140.
CrtDConsts make_crtd(int k, bool offset);

// Shared tail of both conversions: limb digits (T = D_i + C_(i-1)) -> words
// with in-block carry resolution; writes the CTA's (G, P).
template <int NL>
__device__ __forceinline__ void limbs_to_words(const uint64_t (&dig)[NL], const uint32_t (&gen)[NL],
                                               size_t first_limb, uint32_t* z, size_t zw, uint32_t* agg_slot)
{
    uint32_t gp = kGPIdentity;
#pragma unroll
    for (int u = 0; u < NL; u++) {
        const size_t w = 2 * (first_limb + u);
        const uint32_t lo = (uint32_t)dig[u], hi = (uint32_t)(dig[u] >> 32);
        if (w < zw) gp = gp_combine(gp, (uint32_t)(lo == 0xffffffffu) << 1);
        if (w + 1 < zw) gp = gp_combine(gp, gen[u] | ((uint32_t)(hi == 0xffffffffu) << 1));
    }
    uint32_t total;
    uint32_t cin = block_gp_scan(gp, &total) & 1u;
#pragma unroll
    for (int u = 0; u < NL; u++) {
        const size_t w = 2 * (first_limb + u);
        const uint32_t lo = (uint32_t)dig[u], hi = (uint32_t)(dig[u] >> 32);
        if (w < zw) z[w] = lo + cin;
        cin = (uint32_t)(lo == 0xffffffffu) & cin;
        if (w + 1 < zw) z[w + 1] = hi + cin;
        cin = gen[u] | ((uint32_t)(hi == 0xffffffffu) & cin);
    }
    if (threadIdx.x == 0) *agg_slot = total;
}

__device__ __forceinline__ void add128(uint64_t& lo, uint64_t& hi, uint64_t v)
{
    lo += v;
    hi += (lo < v);
}

// x in (-p, 2p) -> [0, p)
__device__ __forceinline__ double dcanon2(double x, double p)
{
    x = x < 0.0 ? __dadd_rn(x, p) : x;
    return x >= p ? __dadd_rn(x, -p) : x;
}

// Garner's CRT on three FP64 residues (|y| < 2^51): x = r0 + p0 (v1 + p1 v2)
// with r_q = y_q N^-1 (+ offset) mod p_q, as three 64-bit limbs (x < 2^141).
__device__ __forceinline__ void crt3d(const CrtDConsts& C, double y0, double y1, double y2, uint64_t& l0,
                                      uint64_t& l1, uint64_t& l2)
{
    // r1 and r2 only enter products, as any representatives
    const double r0 = dcanon2(__dadd_rn(dmul_tw(y0, C.sw[0], C.swp[0], C.p[0]), C.off[0]), C.p[0]);
    const double r1 = __dadd_rn(dmul_tw(y1, C.sw[1], C.swp[1], C.p[1]), C.off[1]);
    const double r2 = __dadd_rn(dmul_tw(y2, C.sw[2], C.swp[2], C.p[2]), C.off[2]);
    const double v1 = dcanon(dmul_tw(__dadd_rn(r1, -r0), C.i01, C.i01p, C.p[1]), C.p[1]);
    const double a = dmul_tw(__dadd_rn(r2, -r0), C.i012, C.i012p, C.p[2]);
    const double b = dmul_tw(v1, C.q012, C.q012p, C.p[2]);
    const double v2 = dcanon(dreduce(__dadd_rn(a, -b), C.p[2], C.pinv[2]), C.p[2]);
    const uint64_t R0 = dto_u64(r0), V1 = dto_u64(v1), V2 = dto_u64(v2);
    const unsigned __int128 lo = (unsigned __int128)R0 + (unsigned __int128)C.p0 * V1 +
                                 (unsigned __int128)C.p01_lo * V2;  // < 2^95 + 2^111
    const unsigned __int128 hi = (lo >> 64) + (unsigned __int128)C.p01_hi * V2;
    l0 = (uint64_t)lo;
    l1 = (uint64_t)hi;
    l2 = (uint64_t)(hi >> 64);
}

// A thread assembles 8 consecutive coefficients (group u: bits 448 u .. 448 u
// + 447 of the product) into the 7 limbs they start; limb L of the group
// collects the windows of the coefficients c = -3 .. 7 that reach it
// (coefficient c at bit 56 c, limb L at bit 64 L), so every shift is a
// compile-time constant and the lanes of a warp never diverge.
// The 64 bits of coefficient x (three limbs, below 2^141) that fall in a limb
// starting s = 56 C - 64 L bits below the coefficient's bit 0.
template <int C, int L>
__device__ __forceinline__ uint64_t coef_win(const uint64_t (&x)[3])
{
    constexpr int s = 56 * C - 64 * L;
    if constexpr (s >= 0) {
        return x[0] << s;
    } else {
        constexpr int r = -s;
        if constexpr (r < 64) return (x[0] >> r) | (x[1] << (64 - r));
        else if constexpr (r == 64) return x[1];
        else if constexpr (r < 128) return (x[1] >> (r - 64)) | (x[2] << (128 - r));
        else if constexpr (r == 128) return x[2];
        else return x[2] >> (r - 128);
    }
}

// Adds coefficient C of a group (limbs x) to the limb sums -1 .. 6.
template <int C, int L = -1>
__device__ __forceinline__ void group_add(const uint64_t (&x)[3], uint64_t (&lo)[8], uint32_t (&hi)[8])
{
    if constexpr (L <= 6) {
        constexpr int s = 56 * C - 64 * L;
        if constexpr (s < 64 && s > -141) {
            const uint64_t v = coef_win<C, L>(x);
            lo[L + 1] += v;
            hi[L + 1] += lo[L + 1] < v;
        }
        group_add<C, L + 1>(x, lo, hi);
    }
}

// A CTA's coefficients as limbs in shared memory: limb w of the i-th at
// X[w XS + crt_slot(i)], the i-th being coefficient j0 + i.  All threads take
// coefficients in turn, so the residues are read coalesced and no thread waits
// for a neighbour; the groups are then assembled from shared memory, whose
// padding keeps threads eight coefficients apart in different banks.
__host__ __device__ constexpr int crt_slot(int i) { return i + (i >> 3); }

// res(j, y0, y1, y2): the residues of coefficient j, 0 <= j < jlim.
template <int XS, class Res>
__device__ __forceinline__ void crt_coefs(uint64_t* X, int64_t j0, int n, int64_t jlim, const CrtDConsts& C,
                                          const Res& res)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int64_t j = j0 + i;
        uint64_t x[3] = {0, 0, 0};
        if (j >= 0 && j < jlim) {
            double y0, y1, y2;
            res(j, y0, y1, y2);
            crt3d(C, y0, y1, y2, x[0], x[1], x[2]);
        }
#pragma unroll
        for (int w = 0; w < 3; w++) X[w * XS + crt_slot(i)] = x[w];
    }
}

template <int XS, int C = -3>
__device__ __forceinline__ void group_sums(const uint64_t* X, int t, uint64_t (&lo)[8], uint32_t (&hi)[8])
{
    if constexpr (C <= 7) {
        const int at = crt_slot(8 * t + C + 3);
        const uint64_t x[3] = {X[at], X[XS + at], X[2 * XS + at]};
        group_add<C>(x, lo, hi);
        group_sums<XS, C + 1>(X, t, lo, hi);
    }
}

// The seven limb digits of the CTA's group t (coefficients i = 8 t .. 8 t + 10,
// the first three being the group before's last) and their carries.
template <int XS>
__device__ __forceinline__ void crt_digits(const uint64_t* X, int t, uint64_t (&dig)[7], uint32_t (&gen)[7])
{
    uint64_t lo[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // limbs -1 .. 6 of the group
    uint32_t hi[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    group_sums<XS>(X, t, lo, hi);
#pragma unroll
    for (int L = 0; L < 7; L++) {
        const uint64_t d = lo[L + 1] + hi[L];
        dig[L] = d;
        gen[L] = d < lo[L + 1];
    }
}

}  // namespace pic
