// The twiddles of the FP64 column passes (cols.cu) and the register round that
// stands beside them.
#pragma once
#include "middle.cuh"

namespace pic {

// Twiddles of one thread's column c: Q^1 .. Q^7 (or fewer rows), and W of a
// group.
template <bool INV, int LC>
struct ColTwiddle {
    static constexpr int BL = LC < 3 ? LC : 3;
    double q[1 << BL];  // q[i] = Q^i, i >= 1
    const double* w;
    const double *lo, *hi;
    int S, esh;
    uint32_t c;
    __device__ __forceinline__ double root(uint64_t e, const Dbl::Ctx& L) const  // root_(2^lblock)^e
    {
        const uint64_t E = e << esh;
        return dmul_w(__ldg(hi + (E >> S)), __ldg(lo + (E & (((uint64_t)1 << S) - 1))), L.p, L.pinv);
    }
    __device__ __forceinline__ void init(const PrimeDev& P, const double* table, int lblock, uint32_t col,
                                         const Dbl::Ctx& L)
    {
        lo = reinterpret_cast<const double*>(INV ? P.slo_inv : P.slo_fwd);
        hi = reinterpret_cast<const double*>(INV ? P.shi_inv : P.shi_fwd);
        S = P.S;
        esh = P.K - lblock;
        c = col;
        w = table != nullptr ? table + col : nullptr;
        q[1] = root((uint64_t)c << (LC - BL), L);
    }
    // made just before the round that uses them, so that they hold no registers
    // in the others
    __device__ __forceinline__ void powers(const Dbl::Ctx& L)
    {
        if constexpr (BL >= 2) {
            q[2] = dmul_w(q[1], q[1], L.p, L.pinv);
            q[3] = dmul_w(q[2], q[1], L.p, L.pinv);
        }
        if constexpr (BL >= 3) {
            q[4] = dmul_w(q[2], q[2], L.p, L.pinv);
            q[5] = dmul_w(q[3], q[2], L.p, L.pinv);
            q[6] = dmul_w(q[3], q[3], L.p, L.pinv);
            q[7] = dmul_w(q[4], q[3], L.p, L.pinv);
        }
    }
    // W of group g (rows 8 g ..): loaded early by the caller
    __device__ __forceinline__ double group(int g, int lM, const Dbl::Ctx& L) const
    {
        if constexpr (LC <= 3) return 1.0;
        if (w != nullptr) return __ldg(w + ((size_t)g << lM));
        return root((uint64_t)c * (__brev((unsigned)g) >> (32 - (LC > 3 ? LC - 3 : 1))), L);
    }
    // |result| <= p: where neither W nor a power of Q multiplies a point (row 0 of a
    // pass of at most three bits) it is reduced instead, as it may be a sum of eight
    // pieces (4 p, where a row accepts 2 p) or what a row left (up to 15.75 p, to
    // which the inverse butterflies add 7 p: past 2^51).  Three FP64 instructions on
    // one point in two to eight.
    __device__ __forceinline__ double apply(double v, int i, double wg, const Dbl::Ctx& L) const
    {
        const int r = brev3(i, BL);
        if (LC > 3) v = dmul_w(v, wg, L.p, L.pinv);
        if (r) return dmul_w(v, q[r], L.p, L.pinv);
        return LC > 3 ? v : dreduce(v, L.p, L.pinv);
    }
    // The round beside the twiddles, forward: its smallest-stride butterflies, then
    // the twiddles of rows i < 2^BL of group g.
    __device__ __forceinline__ void forward_tail(double (&x)[1 << BL], const GroupTw<BL, 0>& t, double wg,
                                                 const Dbl::Ctx& L) const
    {
        fwd_tail<BL>(x, t, L);
#pragma unroll
        for (int i = 0; i < (1 << BL); i++) x[i] = apply(x[i], i, wg, L);
    }
    // Inverse: the twiddles, then the butterflies.
    __device__ __forceinline__ void inverse_head(double (&x)[1 << BL], const GroupTw<BL, 0>& t, double wg,
                                                 const Dbl::Ctx& L) const
    {
#pragma unroll
        for (int i = 0; i < (1 << BL); i++) x[i] = apply(x[i], i, wg, L);
        inv_head<BL, (LC > 10)>(x, t, L);
    }
};

}  // namespace pic
