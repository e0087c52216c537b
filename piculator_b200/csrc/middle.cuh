// Rows of the FP64 form in shared memory: the register rounds of a forward row
// pass of several operands and of an inverse one of several results, shared by
// the fused middle passes (middle.cu) and the short products (small.cu).
#pragma once
#include "passes.cuh"

namespace pic {

using Dbl = ArithDbl;

// The twiddles of one group (see group_fast): level l, butterfly u at
// (2^B - 2^(B-l)) + u.  The unit level of LST 0 is not loaded.
template <int B, int LST>
struct GroupTw {
    double w[(1 << B) - 1];
    __device__ __forceinline__ void load(const double* __restrict__ tw, int j)
    {
#pragma unroll
        for (int l = 0; l < B; l++) {
            if (l == B - 1 && LST == 0) continue;
#pragma unroll
            for (int u = 0; u < (1 << (B - 1 - l)); u++)
                w[(1 << B) - (1 << (B - l)) + u] = __ldg(tw + ((1 << (B - l + LST - 1)) - 1) + j + (u << LST));
        }
    }
    __device__ __forceinline__ double at(int l, int u) const { return w[(1 << B) - (1 << (B - l)) + u]; }
};

template <int B, int LST>
__device__ __forceinline__ void fwd_group(double (&x)[1 << B], const GroupTw<B, LST>& t, const Dbl::Ctx& L)
{
#pragma unroll
    for (int l = 0; l < B; l++) {
        const int hm = 1 << (B - 1 - l);
#pragma unroll
        for (int m = 0; m < (1 << B); m++) {
            if (m & hm) continue;
            if (l == B - 1 && LST == 0) {
                if (Dbl::reduce_unit(B, m)) Dbl::dif_unit<true>(x[m], x[m + hm], L);
                else Dbl::dif_unit<false>(x[m], x[m + hm], L);
            } else {
                if (l == B - 1 && Dbl::reduce_sum(B, m)) Dbl::dif<true>(x[m], x[m + hm], t.at(l, m & (hm - 1)), L);
                else Dbl::dif<false>(x[m], x[m + hm], t.at(l, m & (hm - 1)), L);
            }
        }
    }
}

template <int B, int LST>
__device__ __forceinline__ void inv_group(double (&x)[1 << B], const GroupTw<B, LST>& t, const Dbl::Ctx& L)
{
#pragma unroll
    for (int l = B - 1; l >= 0; l--) {
        const int hm = 1 << (B - 1 - l);
#pragma unroll
        for (int m = 0; m < (1 << B); m++) {
            if (m & hm) continue;
            if (l == B - 1 && LST == 0) Dbl::dit_unit(x[m], x[m + hm], L);
            else Dbl::dit(x[m], x[m + hm], t.at(l, m & (hm - 1)), L);
        }
    }
}

// The same for the smallest-stride round, where t.at(l, u) = root_(2^(B - l))^u,
// so u = 0 needs no product and the unit level none.  Forward: |x| <= 2 p gives
// |x| <= 16 p (8 p for B = 2), unreduced, for a product that follows at once.
template <int B>
__device__ __forceinline__ void fwd_tail(double (&x)[1 << B], const GroupTw<B, 0>& t, const Dbl::Ctx& L)
{
#pragma unroll
    for (int l = 0; l < B; l++) {
        const int hm = 1 << (B - 1 - l);
#pragma unroll
        for (int m = 0; m < (1 << B); m++) {
            if (m & hm) continue;
            if ((m & (hm - 1)) == 0) Dbl::dif_unit<false>(x[m], x[m + hm], L);
            else Dbl::dif<false>(x[m], x[m + hm], t.at(l, m & (hm - 1)), L);
        }
    }
}

// Inverse: |x| <= X gives |x| <= 2^B X, or 2^(B - 1) X + p with the products of
// the last level's u = 0 kept (KEEP: the levels after it add up to p each and
// must end below 15.75 p).
template <int B, bool KEEP>
__device__ __forceinline__ void inv_head(double (&x)[1 << B], const GroupTw<B, 0>& t, const Dbl::Ctx& L)
{
#pragma unroll
    for (int l = B - 1; l >= 0; l--) {
        const int hm = 1 << (B - 1 - l);
#pragma unroll
        for (int m = 0; m < (1 << B); m++) {
            if (m & hm) continue;
            if ((m & (hm - 1)) == 0 && !(KEEP && l == 0)) Dbl::dit_unit(x[m], x[m + hm], L);
            else Dbl::dit(x[m], x[m + hm], t.at(l, m & (hm - 1)), L);
        }
    }
}

// The last forward round of a row, for pointwise products: of two factors one is
// reduced (|x| <= p / 2 + 1) and the other left at up to 16 p, a product of at
// most 8 p^2 and below 0.75 p after its reduction.
template <int B, bool RED>
__device__ __forceinline__ void fwd_last(double (&x)[1 << B], const GroupTw<B, 0>& t, const Dbl::Ctx& L)
{
    fwd_tail<B>(x, t, L);
    if constexpr (RED) {
#pragma unroll
        for (int m = 0; m < (1 << B); m++) x[m] = dreduce(x[m], L.p, L.pinv);
    }
}

// The first inverse round of a 2^LR row whose points are below X = 0.75 TERMS p
// (a sum of TERMS products): at most 4 X, the LR - 2 levels (or LR - 1, of 2 X)
// after it p each, and the row ends below 15.75 p.
template <int B, int LR, int TERMS>
__device__ __forceinline__ void inv_first(double (&x)[1 << B], const GroupTw<B, 0>& t, const Dbl::Ctx& L)
{
    if constexpr (B == 1 || 4 * 0.75 * TERMS + (LR - 2) > 15.75) inv_group<B, 0>(x, t, L);
    else inv_head<B, B == 3>(x, t, L);
}

// Shared-memory place of a row's element e: bits 4, 5, 6 of e are XORed into
// bits 0, (1 and 2), 3.  The map is linear, so the place of base + (m << LST)
// (disjoint bits) is place(base) ^ place(m << LST), the latter a constant.
// Half a warp's 16 elements then fall in 16 different bank pairs in every round
// of 11-bit rows (strides 2^8, 2^5, 2^2, 1).
__host__ __device__ constexpr int place(int e)
{
    return e ^ ((e >> 4) & 1) ^ (((e >> 5) & 1) * 6) ^ (((e >> 6) & 1) << 3);
}

// The place of element base + m (disjoint bits) from pb = place(base): only the
// low four bits of place(m) need the XOR, the others are zero in pb and become
// the access's constant offset.
__host__ __device__ constexpr int place_at(int pb, int m) { return (pb ^ (place(m) & 15)) + (place(m) & ~15); }

// Rounds of a 2^LR row: radix 8, the remainder last (smallest stride).
template <int LR, int R>
using Round = typename RoundPlan<LR, 3>::template At<R>;

// A CTA's shape: 2^LT rows of 2^LR points of each operand, one thread per
// radix-8 group of one operand.
template <int LR, int LT>
struct MiddleShape {
    static constexpr int TOT = 1 << (LR + LT);  // points of one operand in the CTA
    static constexpr int NT = TOT >> 3;
    static constexpr int NR = RoundPlan<LR, 3>::NR;
};

// Forward rounds 0 .. NR - 2 of every operand: in(a, t, e) reads operand a's
// element e of the CTA's row t.
template <int LR, int LT, int NOP, int R, class In>
__device__ __forceinline__ void forward_rounds(double* __restrict__ s, const Dbl::Ctx& L,
                                               const double* __restrict__ tw, int nop, const In& in)
{
    using Sh = MiddleShape<LR, LT>;
    if constexpr (R + 1 < Sh::NR) {
        using At = Round<LR, R>;
        constexpr int B = At::B, LB = At::LB, LST = At::LST, LG = LR - B;
        static_assert(B == 3, "full rounds come first");
        const int g = threadIdx.x;
        const int t = g >> LG, gi = g & ((1 << LG) - 1);
        const int j = gi & ((1 << LST) - 1);
        const int base = ((gi >> LST) << LB) + j;
        const int pb = (t << LR) + place(base);
        GroupTw<B, LST> w;
        w.load(tw, j);
#pragma unroll 2
        for (int a = 0; a < nop; a++) {
            double x[8];
            double* sa = s + a * Sh::TOT;
#pragma unroll
            for (int m = 0; m < 8; m++) {
                if constexpr (R == 0) x[m] = in(a, t, base + (m << LST));
                else x[m] = sa[place_at(pb, m << LST)];
            }
            fwd_group<B, LST>(x, w, L);
#pragma unroll
            for (int m = 0; m < 8; m++) sa[place_at(pb, m << LST)] = x[m];
        }
        __syncthreads();
        forward_rounds<LR, LT, NOP, R + 1>(s, L, tw, nop, in);
    }
}

// Inverse rounds R .. 0 of the results in rows act(i), i < nout; out(i, t, e, v)
// writes result i's element e of the CTA's row t.
template <int LR, int LT, int R, class Act, class Out>
__device__ __forceinline__ void inverse_rounds(double* __restrict__ s, const Dbl::Ctx& L,
                                               const double* __restrict__ tw, int nout, const Act& act, const Out& out)
{
    using Sh = MiddleShape<LR, LT>;
    using At = Round<LR, R>;
    constexpr int B = At::B, LB = At::LB, LST = At::LST, LG = LR - B;
    const int g = threadIdx.x;
    const int t = g >> LG, gi = g & ((1 << LG) - 1);
    const int j = gi & ((1 << LST) - 1);
    const int base = ((gi >> LST) << LB) + j;
    const int pb = (t << LR) + place(base);
    GroupTw<B, LST> w;
    w.load(tw, j);
    __syncthreads();
#pragma unroll 2
    for (int i = 0; i < nout; i++) {
        double x[8];
        double* sa = s + act(i) * Sh::TOT;
#pragma unroll
        for (int m = 0; m < 8; m++) x[m] = sa[place_at(pb, m << LST)];
        inv_group<B, LST>(x, w, L);
#pragma unroll
        for (int m = 0; m < 8; m++) {
            if constexpr (R == 0) out(i, t, base + (m << LST), x[m]);
            else sa[place_at(pb, m << LST)] = x[m];
        }
    }
    if constexpr (R > 0) inverse_rounds<LR, LT, R - 1>(s, L, tw, nout, act, out);
}

}  // namespace pic
