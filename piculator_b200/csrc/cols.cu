// Column passes of the FP64 product form.
//
// A pass over blocks of 2^lblock points takes a block as 2^LC rows of M =
// 2^(lblock - LC) points: a size-2^LC transform down every column and, after
// it (forward) or before it (inverse), the twiddle root_(2^lblock)^(c k1) of
// column c and frequency k1 = brev(row).  A CTA owns 2^LW columns of one block.
//
//  * The first register round reads global memory, the last one writes it; the
//    rounds between exchange through shared memory.  The remainder round
//    (radix 2 or 4) is the one at the largest stride, so that the round beside
//    the twiddles always has radix 8 (or is the only one): its rows are 8 g + i,
//    whose frequencies are brev(g) + brev3(i) 2^(LC - 3), so the twiddle is
//    W(g, c) Q(c)^brev3(i).  W comes from a table of one entry per eight points
//    (or the two-level outer tables), the powers of Q are made once per thread:
//    one more FP64 product per point instead of a streamed 8-byte table entry.
//    That round's smallest-stride butterflies have twiddles that are constants,
//    one in four of them 1, and nothing after it needs a reduction: the twiddle
//    product takes any |y| < 2^51.  In a pass of at most three bits row 0 meets no
//    twiddle; it alone is reduced, in both directions (cols.cuh).
//  * The first forward pass reads its points from the operand's words.  The
//    rows of one thread are a multiple of four pieces apart, hence a whole
//    number of words: one shift and one word address serve all of them.
//
// Bound by instruction issue and latency together (FP64 pipe 50 - 60 %, 2.6
// instructions per clock, 32 warps; three CTAs per SM without the few spills of
// four ran the 1e9-digit computation in 1.44 s instead of 1.36).  Against the
// passes before (a streamed twiddle per point, pieces extracted one by one, a
// 7-bit pass from words 143 us on 2^23 points x 3 primes, here 128; 3-bit ones
// 94 and 71): pi to 1e9 digits 1.49 -> 1.36 s, 2^24-word operands 3.32 -> 2.96
// ms, 1,048,573 x 400,009 words 143 -> 122 us of kernels.
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>

#include "cols.cuh"
#include "common.cuh"
#include "middle.cuh"

namespace pic {

constexpr int kColThreads = 256;

struct ColTables {
    const double* w[3];  // per prime: W(g, c) at g M + c, or null
};

struct ColArgs {
    NttBatch b;
    ColTables t;
    int lblock;  // log2 points of a block
    int lpre;    // log2 blocks of a transform
};

// The pieces of rows r0 + m 2^LST (m < 2^B) of a column from the operand's
// words: word address wi of row r0, `step` words between the rows, bit offset
// sh of every piece in its first word.
template <int B>
__device__ __forceinline__ void load_pieces(double (&x)[1 << B], const uint32_t* __restrict__ words, uint32_t n,
                                            size_t wi, size_t step, int sh, const Dbl::Ctx& L)
{
    constexpr int E = 1 << B;
    uint32_t w0[E], w1[E], w2[E];
    if (wi + (E - 1) * step + 2 < n) {  // every word there: no test per word
        const uint32_t* p = words + wi;
#pragma unroll
        for (int m = 0; m < E; m++, p += step) {
            w0[m] = __ldg(p);
            w1[m] = __ldg(p + 1);
            w2[m] = __ldg(p + 2);
        }
    } else {
#pragma unroll
        for (int m = 0; m < E; m++) {
            const size_t a = wi + m * step;
            w0[m] = a < n ? __ldg(words + a) : 0u;
            w1[m] = a + 1 < n ? __ldg(words + a + 1) : 0u;
            w2[m] = a + 2 < n ? __ldg(words + a + 2) : 0u;
        }
    }
#pragma unroll
    for (int m = 0; m < E; m++) {
        const uint32_t lo = __funnelshift_r(w0[m], w1[m], sh), hi = __funnelshift_r(w1[m], w2[m], sh);
        x[m] = dpiece28(__funnelshift_l(lo, hi, 4) & 0x0fffffffu, lo & 0x0fffffffu, L.p, L.pinv);
    }
}

template <bool INV, int LC, int LW, bool SRC>
__global__ void __launch_bounds__(kColThreads, 4) cols56_kernel(const __grid_constant__ ColArgs A)
{
    using Plan = ColPlan<LC>;
    constexpr int NR = Plan::NR, TOT = 1 << (LC + LW), WMASK = (1 << LW) - 1;
    extern __shared__ double cs[];
    const int lM = A.lblock - LC, ltiles = lM - LW;
    const size_t cta = blockIdx.x;
    const int tr = (int)(cta >> (ltiles + A.lpre));
    const size_t rem = cta & (((size_t)1 << (ltiles + A.lpre)) - 1);
    const size_t ob = rem >> ltiles;
    const uint32_t c0 = (uint32_t)((rem & (((size_t)1 << ltiles) - 1)) << LW);
    const int pq = tr < A.b.per_prime ? 0 : (tr < 2 * A.b.per_prime ? 1 : 2);
    const PrimeDev& P = pq == 0 ? A.b.prime[0] : (pq == 1 ? A.b.prime[1] : A.b.prime[2]);
    const Dbl::Ctx L = Dbl::ctx(P);
    const double* __restrict__ tw = reinterpret_cast<const double*>(INV ? P.lvl_inv : P.lvl_fwd);
    const int w = threadIdx.x & WMASK;  // the thread's column in every round
    uint64_t* __restrict__ col = A.b.data + (size_t)tr * A.b.stride + (ob << A.lblock) + c0 + w;
    ColTwiddle<INV, LC> T;
    T.init(P, pq == 0 ? A.t.w[0] : (pq == 1 ? A.t.w[1] : A.t.w[2]), A.lblock, c0 + w, L);
    // source words: bit 56 (first + row M + c0 + w)
    const uint32_t* words = nullptr;
    uint32_t n = 0;
    size_t wi0 = 0;
    int sh = 0;
    if constexpr (SRC) {
        const SrcRow sr = src_row(A.b, tr);
        words = sr.x;
        n = sr.n;
        const size_t bit = 56 * (A.b.src.first + c0 + w);
        wi0 = bit >> 5;
        sh = (int)(bit & 31);
    }

    // one round of every group of the thread; R counts from the largest stride
    auto round = [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        using At = typename Plan::template At<R>;
        constexpr int B = At::B, LB = At::LB, LST = At::LST, E = 1 << B;
        constexpr int G = TOT >> B;
        constexpr bool FIRST = INV ? R == NR - 1 : R == 0, LAST = INV ? R == 0 : R == NR - 1;
        constexpr bool TAIL = R == NR - 1;  // smallest stride: beside the twiddles
        GroupTw<B, LST> t;
        if constexpr (LST == 0) t.load(tw, 0);
        if constexpr (TAIL) T.powers(L);
#pragma unroll 1
        for (int g = threadIdx.x; g < G; g += kColThreads) {
            const int gi = g >> LW, j = gi & ((1 << LST) - 1);
            const int r0 = ((gi >> LST) << LB) + j;
            const int pb = col_place<LW>((r0 << LW) + w);
            double x[E];
            double wg = 1.0;
            if constexpr (TAIL) wg = T.group(gi, lM, L);
            if constexpr (FIRST && SRC) {
                // 7 words per four pieces; M is a multiple of four
                load_pieces<B>(x, words, n, wi0 + (((size_t)r0 << lM) >> 2) * 7, ((size_t)7 << (LST + lM)) >> 2, sh,
                               L);
            } else if constexpr (FIRST) {
                const uint64_t* p = col + ((size_t)r0 << lM);
                const size_t step = (size_t)1 << (LST + lM);
#pragma unroll
                for (int m = 0; m < E; m++, p += step) x[m] = dbits(*p);
            } else {
#pragma unroll
                for (int m = 0; m < E; m++) x[m] = cs[col_at<LW>(pb, m << (LST + LW))];
            }
            if constexpr (LST > 0) t.load(tw, j);
            if constexpr (!INV) {
                if constexpr (TAIL) {
                    T.forward_tail(x, t, wg, L);
                } else {
                    fwd_group<B, LST>(x, t, L);
                }
            } else {
                if constexpr (TAIL) {
                    T.inverse_head(x, t, wg, L);
                } else {
                    inv_group<B, LST>(x, t, L);
                }
            }
            if constexpr (LAST) {
                uint64_t* p = col + ((size_t)r0 << lM);
                const size_t step = (size_t)1 << (LST + lM);
#pragma unroll
                for (int m = 0; m < E; m++, p += step) *p = dstore(x[m]);
            } else {
#pragma unroll
                for (int m = 0; m < E; m++) cs[col_at<LW>(pb, m << (LST + LW))] = x[m];
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

// ---- tables of W ----------------------------------------------------------------
// Entry g M + c = root_(2^lblock)^(c brev_(LC - 3)(g)), 2^(lblock - 3) entries:
// built on the device on first use per (device, prime, direction, lblock, LC),
// kept for the process; never built while the stream is being captured.  A table
// enters the cache only when its build kernel has finished.
__global__ void col_table_kernel(double* __restrict__ out, PrimeDev P, int inv, int lblock, int lc)
{
    const int lM = lblock - lc;
    const size_t n = (size_t)1 << (lblock - 3);
    const double* dlo = reinterpret_cast<const double*>(inv ? P.slo_inv : P.slo_fwd);
    const double* dhi = reinterpret_cast<const double*>(inv ? P.shi_inv : P.shi_fwd);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint64_t g = i >> lM, c = i & (((size_t)1 << lM) - 1);
        const uint64_t E = (c * (__brev((unsigned)g) >> (32 - (lc - 3)))) << (P.K - lblock);
        out[i] = dmul_w(__ldg(dhi + (E >> P.S)), __ldg(dlo + (E & (((uint64_t)1 << P.S) - 1))), P.pd, P.pinv);
    }
}

static std::mutex g_col_lock;
static std::map<std::tuple<int, uint64_t, int, int, int>, double*> g_col_tables;

static const double* col_table(const PrimeDev& P, bool inv, int lblock, int lc, cudaStream_t s)
{
    if (lc <= 3 || lblock > 24 || lblock > ntt_dbl_pass_bits()) return nullptr;
    int dev = 0;
    PIC_CUDA(cudaGetDevice(&dev));
    const auto key = std::make_tuple(dev, P.p, inv ? 1 : 0, lblock, lc);
    std::lock_guard<std::mutex> g(g_col_lock);
    auto it = g_col_tables.find(key);
    if (it != g_col_tables.end()) return it->second;
    cudaStreamCaptureStatus cst = cudaStreamCaptureStatusNone;
    PIC_CUDA(cudaStreamIsCapturing(s, &cst));
    if (cst != cudaStreamCaptureStatusNone) return nullptr;
    void* d = nullptr;
    const size_t n = (size_t)1 << (lblock - 3);
    if (raw_dev_alloc(&d, sizeof(double) * n) != cudaSuccess) return nullptr;  // the two-level tables instead
    col_table_kernel<<<grid_for(n, 256), 256, 0, s>>>(static_cast<double*>(d), P, inv ? 1 : 0, lblock, lc);
    PIC_CHECK_LAUNCH();
    count_launch();
    PIC_CUDA(cudaStreamSynchronize(s));
    g_col_tables[key] = static_cast<double*>(d);
    return g_col_tables[key];
}

template <bool INV, int LC, int LW, bool SRC>
static void launch_cols56(const ColArgs& A, cudaStream_t s)
{
    const size_t grid = (size_t)A.b.count << (A.lblock - LC - LW + A.lpre);
    PIC_REQUIRE(grid <= 0x7fffffffu, PIC_ERR_INVALID, "column pass grid too large");
    const size_t smem = ColPlan<LC>::NR > 1 ? sizeof(double) << (LC + LW) : 0;
    auto kern = cols56_kernel<INV, LC, LW, SRC>;
    if (smem > 48 * 1024) PIC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<(unsigned)grid, kColThreads, smem, s>>>(A);
    PIC_CHECK_LAUNCH();
    count_launch();
}

template <int LC, int LW>
static void cols56_dir(bool inv, const ColArgs& A, cudaStream_t s)
{
    if (inv) launch_cols56<true, LC, LW, false>(A, s);
    else if (A.b.src.words != nullptr) launch_cols56<false, LC, LW, true>(A, s);
    else launch_cols56<false, LC, LW, false>(A, s);
}

// Tile widths: 2^11 .. 2^13 points (every thread at least one group, at most 64
// KB), short columns as wide as it takes (64 columns of 2^2 or 2^3 rows gave a
// quarter of the threads work: the merge level of 2^13 points took 169 ms of
// the 1e9 run instead of 46).
void ntt_cols56(bool inv, const NttBatch& b, int k, int lpre, int lc, int lw, cudaStream_t s)
{
    ColArgs A;
    A.b = b;
    A.lblock = k - lpre;
    A.lpre = lpre;
    const int lM = A.lblock - lc;
    PIC_REQUIRE(lM >= 8, PIC_ERR_INVALID, "FP64 column pass narrower than its tiles");
    bool all = true;
    for (int q = 0; q < 3; q++) {
        A.t.w[q] = q * b.per_prime < b.count ? col_table(b.prime[q], inv, A.lblock, lc, s) : nullptr;
        if (q * b.per_prime < b.count && A.t.w[q] == nullptr) all = false;
    }
    if (!all) A.t = ColTables{};  // one form for every prime of the launch
    const int lo = std::max(2, 11 - lc), hi = std::max(2, 13 - lc);
    lw = std::min(std::max(lw, lo), hi);
#define PIC_COLS56(C, W) case (C) * 16 + (W): cols56_dir<C, W>(inv, A, s); return
    switch (lc <= 3 ? lc * 16 + 8 : (lc == 4 ? 4 * 16 + 7 : (lc == 5 ? 5 * 16 + 6 : lc * 16 + std::min(lw, 6)))) {
    PIC_COLS56(1, 8);
    PIC_COLS56(2, 8);
    PIC_COLS56(3, 8);
    PIC_COLS56(4, 7);
    PIC_COLS56(5, 6);
    PIC_COLS56(6, 5);
    PIC_COLS56(6, 6);
    PIC_COLS56(7, 4);
    PIC_COLS56(7, 5);
    PIC_COLS56(7, 6);
    PIC_COLS56(8, 3);
    PIC_COLS56(8, 4);
    PIC_COLS56(8, 5);
    PIC_COLS56(9, 2);
    PIC_COLS56(9, 3);
    PIC_COLS56(9, 4);
    PIC_COLS56(10, 2);
    PIC_COLS56(10, 3);
    PIC_COLS56(11, 2);
    default: throw Error(PIC_ERR_INVALID, "FP64 column pass outside its kernels' shapes");
    }
#undef PIC_COLS56
}

}  // namespace pic
