// Natural-order NTTs modulo the reference's 63-bit primes (NTT.h).
//
// The general passes run any prime and geometry with run-time rounds, move the
// order apart (a scattered 16 bytes a point) and scale apart.  Here the rounds
// are compile-time, the row pass also does the bit reversal, and the inverse's
// factor 2^-k rides on the last pass's twiddles.  DIF output r 2^lr + j stands
// for frequency brev(j) 2^(k - lr) + brev(r), so a CTA that takes the four rows
// whose brev(r) are 4 c .. 4 c + 3 writes (forward) or reads (inverse) runs of
// four words, a whole sector: the price is a second buffer of 2^k words.
// Values stay in [0, p): below 2^63 there is no room for lazy residues, and a
// butterfly is about 35 integer instructions, which is what bounds the passes.
// 2^22 points, forward: 96 us of columns, 76 of rows and 42 of reversal with the
// general passes; 67 and 49 here.  The NTT.h flow on operands of 1,048,571 and
// 1,000,003 words 753 -> 426 us (with the 16-bit conversion of mul.cu).
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "modarith.cuh"
#include "passes.cuh"

namespace pic {

constexpr int kNatThreads = 256;
constexpr int kNatRowBits = 11;
constexpr int kNatRows = 4;                              // rows per CTA
constexpr int kNatStride = (1 << kNatRowBits) + 8;       // words between them: other banks

// The levels of a group at stride 2^LST with the per-level Shoup tables (see
// group_fast); the unit level of LST 0 has no product.
template <int B, bool INV, int LST>
__device__ __forceinline__ void nat_group(uint64_t (&x)[1 << B], const ulonglong2 (&w)[(1 << B) - 1], uint64_t p)
{
    if (!INV) {
#pragma unroll
        for (int l = 0; l < B; l++) {
            const int hm = 1 << (B - 1 - l);
#pragma unroll
            for (int m = 0; m < (1 << B); m++) {
                if (m & hm) continue;
                const uint64_t a = x[m], b = x[m + hm];
                x[m] = add_mod(a, b, p);
                if (l == B - 1 && LST == 0) {
                    x[m + hm] = sub_mod(a, b, p);
                } else {
                    const ulonglong2 t = w[(1 << B) - (1 << (B - l)) + (m & (hm - 1))];
                    x[m + hm] = shoup_mul(a + (p - b), t.x, t.y, p);  // below 2 p < 2^64
                }
            }
        }
    } else {
#pragma unroll
        for (int l = B - 1; l >= 0; l--) {
            const int hm = 1 << (B - 1 - l);
#pragma unroll
            for (int m = 0; m < (1 << B); m++) {
                if (m & hm) continue;
                const uint64_t a = x[m];
                uint64_t b = x[m + hm];
                if (!(l == B - 1 && LST == 0)) {
                    const ulonglong2 t = w[(1 << B) - (1 << (B - l)) + (m & (hm - 1))];
                    b = shoup_mul(b, t.x, t.y, p);
                }
                x[m] = add_mod(a, b, p);
                x[m + hm] = sub_mod(a, b, p);
            }
        }
    }
}

template <int B, int LST>
__device__ __forceinline__ void nat_twiddles(ulonglong2 (&w)[(1 << B) - 1], const ulonglong2* __restrict__ tw, int j)
{
#pragma unroll
    for (int l = 0; l < B; l++) {
        if (l == B - 1 && LST == 0) continue;
#pragma unroll
        for (int u = 0; u < (1 << (B - 1 - l)); u++)
            w[(1 << B) - (1 << (B - l)) + u] = __ldg(tw + ((1 << (B - l + LST - 1)) - 1) + j + (u << LST));
    }
}

// Column pass over blocks of 2^lblock points, src -> dst (may be the same): a
// CTA takes 2^LW columns of 2^LC rows.  The smallest-stride round, radix 8 or
// the only one, stands beside the twiddle W(g, c) Q(c)^brev3(i) of row 8 g + i
// (see cols.cu), in Montgomery form; scale (Montgomery, 0: none) multiplies
// every point too.
template <bool INV, int LC, int LW>
__global__ void __launch_bounds__(kNatThreads, 3) nat_cols_kernel(const uint64_t* src, uint64_t* dst, PrimeDev P,
                                                                  int lblock, int lpre, uint64_t scale)
{
    using Plan = ColPlan<LC>;
    constexpr int NR = Plan::NR, TOT = 1 << (LC + LW), WMASK = (1 << LW) - 1, BL = LC < 3 ? LC : 3;
    extern __shared__ uint64_t nsm[];
    const int lM = lblock - LC, ltiles = lM - LW;
    const size_t ob = blockIdx.x >> ltiles;
    const uint32_t c0 = (uint32_t)((blockIdx.x & (((size_t)1 << ltiles) - 1)) << LW);
    const int w = threadIdx.x & WMASK;
    const uint64_t c = c0 + w;
    const size_t at = (ob << lblock) + c;
    const uint64_t p = P.p, pn = P.pinv_neg;
    const ulonglong2* __restrict__ tw = reinterpret_cast<const ulonglong2*>(INV ? P.lvl_inv : P.lvl_fwd);
    auto round = [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        using At = typename Plan::template At<R>;
        constexpr int B = At::B, LB = At::LB, LST = At::LST, E = 1 << B;
        constexpr int G = TOT >> B;
        constexpr bool FIRST = INV ? R == NR - 1 : R == 0, LAST = INV ? R == 0 : R == NR - 1;
        constexpr bool TAIL = R == NR - 1;
        uint64_t q[TAIL ? (1 << BL) : 2];  // Q^i
        if constexpr (TAIL) {
            q[1] = outer_root<INV>(P, c << (LC - BL), lblock);
#pragma unroll
            for (int i = 2; i < (1 << BL); i++) q[i] = mont_mul(q[i - 1], q[1], p, pn);
        }
#pragma unroll 1
        for (int g = threadIdx.x; g < G; g += kNatThreads) {
            const int gi = g >> LW, j = gi & ((1 << LST) - 1);
            const int r0 = ((gi >> LST) << LB) + j;
            const int pb = col_place<LW>((r0 << LW) + w);
            uint64_t x[E];
            uint64_t wg = 0;
            if constexpr (TAIL) {
                wg = scale;
                if constexpr (LC > 3) {
                    wg = outer_root<INV>(P, c * (__brev((unsigned)gi) >> (32 - (LC - 3))), lblock);
                    if (scale) wg = mont_mul(wg, scale, p, pn);
                }
            }
            if constexpr (FIRST) {
                const uint64_t* s = src + at + ((size_t)r0 << lM);
                const size_t step = (size_t)1 << (LST + lM);
#pragma unroll
                for (int m = 0; m < E; m++, s += step) x[m] = *s;
            } else {
#pragma unroll
                for (int m = 0; m < E; m++) x[m] = nsm[col_at<LW>(pb, m << (LST + LW))];
            }
            ulonglong2 t[E - 1];
            nat_twiddles<B, LST>(t, tw, j);
            auto twiddle = [&]() {
#pragma unroll
                for (int m = 0; m < E; m++) {
                    const int r = brev3(m, BL);
                    if (LC > 3 || wg) x[m] = mont_mul(x[m], wg, p, pn);
                    if (r) x[m] = mont_mul(x[m], q[r], p, pn);
                }
            };
            if constexpr (TAIL && INV) twiddle();
            nat_group<B, INV, LST>(x, t, p);
            if constexpr (TAIL && !INV) twiddle();
            if constexpr (LAST) {
                uint64_t* d = dst + at + ((size_t)r0 << lM);
                const size_t step = (size_t)1 << (LST + lM);
#pragma unroll
                for (int m = 0; m < E; m++, d += step) *d = x[m];
            } else {
#pragma unroll
                for (int m = 0; m < E; m++) nsm[col_at<LW>(pb, m << (LST + LW))] = x[m];
            }
        }
        if constexpr (!LAST) __syncthreads();
    };
    if constexpr (!INV) {
        round(std::integral_constant<int, 0>{});
        if constexpr (NR > 1) round(std::integral_constant<int, 1>{});
        if constexpr (NR > 2) round(std::integral_constant<int, 2>{});
        if constexpr (NR > 3) round(std::integral_constant<int, 3>{});
    } else {
        if constexpr (NR > 3) round(std::integral_constant<int, 3>{});
        if constexpr (NR > 2) round(std::integral_constant<int, 2>{});
        if constexpr (NR > 1) round(std::integral_constant<int, 1>{});
        round(std::integral_constant<int, 0>{});
    }
}

// Row pass with the bit reversal: forward reads rows of src in place and writes
// dst in natural order, inverse the other way round.  CTA c takes the rows r
// with brev(r) = 4 c + t, t < 4.
template <bool INV>
__global__ void __launch_bounds__(kNatThreads, 3) nat_rows_kernel(const uint64_t* __restrict__ src,
                                                                  uint64_t* __restrict__ dst, PrimeDev P, int k)
{
    constexpr int LR = kNatRowBits, NR = RoundPlan<LR, 3>::NR;
    extern __shared__ uint64_t nsm[];
    const int lrow = k - LR;
    const uint32_t f0 = blockIdx.x * kNatRows;
    const uint64_t p = P.p;
    const ulonglong2* __restrict__ tw = reinterpret_cast<const ulonglong2*>(INV ? P.lvl_inv : P.lvl_fwd);
    auto row = [&](int t) { return (size_t)(__brev(f0 + t) >> (32 - lrow)) << LR; };
    auto natural = [&](int t, int e) {
        return ((size_t)(__brev((unsigned)e) >> (32 - LR)) << lrow) + f0 + t;
    };
    if constexpr (INV) {
        for (int i = threadIdx.x; i < (kNatRows << LR); i += kNatThreads) {
            const int t = i & (kNatRows - 1), e = i >> 2;
            nsm[t * kNatStride + swz(e)] = src[natural(t, e)];
        }
        __syncthreads();
    }
    auto round = [&](auto rc) {
        constexpr int RR = INV ? NR - 1 - decltype(rc)::value : decltype(rc)::value;
        using At = typename RoundPlan<LR, 3>::template At<RR>;
        constexpr int B = At::B, LB = At::LB, LST = At::LST, E = 1 << B, G = 1 << (LR - B);
        constexpr bool FIRST = decltype(rc)::value == 0, LAST = decltype(rc)::value == NR - 1;
        for (int g = threadIdx.x; g < G; g += kNatThreads) {
            const int j = g & ((1 << LST) - 1), base = ((g >> LST) << LB) + j;
            ulonglong2 w[E - 1];
            nat_twiddles<B, LST>(w, tw, j);
#pragma unroll 1
            for (int t = 0; t < kNatRows; t++) {
                uint64_t x[E];
                uint64_t* s = nsm + t * kNatStride;
#pragma unroll
                for (int m = 0; m < E; m++) {
                    const int e = base + (m << LST);
                    x[m] = !INV && FIRST ? src[row(t) + e] : s[swz(e)];
                }
                nat_group<B, INV, LST>(x, w, p);
#pragma unroll
                for (int m = 0; m < E; m++) {
                    const int e = base + (m << LST);
                    if (INV && LAST) dst[row(t) + e] = x[m];
                    else s[swz(e)] = x[m];
                }
            }
        }
        if constexpr (!(INV && LAST)) __syncthreads();
    };
    static_assert(NR == 4, "11-bit rows");
    round(std::integral_constant<int, 0>{});
    round(std::integral_constant<int, 1>{});
    round(std::integral_constant<int, 2>{});
    round(std::integral_constant<int, 3>{});
    if constexpr (!INV) {
        for (int i = threadIdx.x; i < (kNatRows << LR); i += kNatThreads) {
            const int t = i & (kNatRows - 1), e = i >> 2;
            dst[natural(t, e)] = nsm[t * kNatStride + swz(e)];
        }
    }
}

template <bool INV, int LC, int LW>
static void launch_nat_cols(const uint64_t* src, uint64_t* dst, const PrimeDev& P, int k, int lpre, uint64_t scale,
                            cudaStream_t s)
{
    const int lblock = k - lpre;
    const size_t grid = (size_t)1 << (lblock - LC - LW + lpre);
    const size_t smem = ColPlan<LC>::NR > 1 ? sizeof(uint64_t) << (LC + LW) : 0;
    auto kern = nat_cols_kernel<INV, LC, LW>;
    if (smem > 48 * 1024) PIC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<(unsigned)grid, kNatThreads, smem, s>>>(src, dst, P, lblock, lpre, scale);
    PIC_CHECK_LAUNCH();
    count_launch();
}

template <bool INV>
static void nat_cols(const uint64_t* src, uint64_t* dst, const PrimeDev& P, int k, int lpre, int lc, uint64_t scale,
                     cudaStream_t s)
{
    ProfScope ps(KC_NTT_COLS, 16.0 * (double)((size_t)1 << k), s);
    switch (lc) {
    case 2: launch_nat_cols<INV, 2, 8>(src, dst, P, k, lpre, scale, s); break;
    case 3: launch_nat_cols<INV, 3, 8>(src, dst, P, k, lpre, scale, s); break;
    case 4: launch_nat_cols<INV, 4, 7>(src, dst, P, k, lpre, scale, s); break;
    case 5: launch_nat_cols<INV, 5, 6>(src, dst, P, k, lpre, scale, s); break;
    case 6: launch_nat_cols<INV, 6, 5>(src, dst, P, k, lpre, scale, s); break;
    case 7: launch_nat_cols<INV, 7, 4>(src, dst, P, k, lpre, scale, s); break;
    case 8: launch_nat_cols<INV, 8, 4>(src, dst, P, k, lpre, scale, s); break;
    case 9: launch_nat_cols<INV, 9, 3>(src, dst, P, k, lpre, scale, s); break;
    case 10: launch_nat_cols<INV, 10, 2>(src, dst, P, k, lpre, scale, s); break;
    case 11: launch_nat_cols<INV, 11, 2>(src, dst, P, k, lpre, scale, s); break;
    default: throw Error(PIC_ERR_INVALID, "column pass outside its kernels' shapes");
    }
}

template <bool INV>
static void nat_rows(const uint64_t* src, uint64_t* dst, const PrimeDev& P, int k, cudaStream_t s)
{
    ProfScope ps(KC_NTT_ROWS, 16.0 * (double)((size_t)1 << k), s);
    const size_t smem = sizeof(uint64_t) * kNatRows * kNatStride;
    PIC_CUDA(cudaFuncSetAttribute(nat_rows_kernel<INV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    nat_rows_kernel<INV><<<(unsigned)(((size_t)1 << (k - kNatRowBits)) / kNatRows), kNatThreads, smem, s>>>(src, dst,
                                                                                                           P, k);
    PIC_CHECK_LAUNCH();
    count_launch();
}

bool ntt_natural(uint64_t* T, int k, const PrimeDev& P, bool inverse, cudaStream_t s)
{
    if (k < kNatRowBits + 2 || P.lvl_fwd == nullptr || P.fp64 || P.K < k) return false;
    cudaStreamCaptureStatus cst = cudaStreamCaptureStatusNone;
    PIC_CUDA(cudaStreamIsCapturing(s, &cst));
    if (cst != cudaStreamCaptureStatusNone) return false;
    const size_t bytes = sizeof(uint64_t) << k;
    if (bytes > ((size_t)1 << 30) && bytes > device_available_bytes() / 2) return false;
    DevBuf<uint64_t> tmp;
    try {
        tmp = DevBuf<uint64_t>((size_t)1 << k, s);
    } catch (const Error&) {
        return false;
    }
    // column passes of at most 11 bits, balanced; the last block is the row
    const int rest = k - kNatRowBits, ncol = (rest + 10) / 11;
    std::vector<int> bits;
    for (int i = 0, left = rest; i < ncol; i++) {
        bits.push_back((left + ncol - i - 1) / (ncol - i));
        left -= bits.back();
    }
    if (!inverse) {
        int lpre = 0;
        for (int i = 0; i < ncol; i++) {
            nat_cols<false>(i == 0 ? T : tmp.get(), tmp.get(), P, k, lpre, bits[i], 0, s);
            lpre += bits[i];
        }
        nat_rows<false>(tmp.get(), T, P, k, s);
    } else {
        const uint64_t n = (uint64_t)1 << k;
        const uint64_t scale = to_mont(host_powmod(n % P.p, P.p - 2, P.p), P.p);
        nat_rows<true>(T, tmp.get(), P, k, s);
        int lpre = rest;
        for (int i = ncol - 1; i >= 0; i--) {
            lpre -= bits[i];
            nat_cols<true>(tmp.get(), i == 0 ? T : tmp.get(), P, k, lpre, bits[i], i == 0 ? scale : 0, s);
        }
    }
    return true;
}

}  // namespace pic
