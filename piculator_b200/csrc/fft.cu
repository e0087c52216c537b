// FP64 FFT engine (see fft.cuh) and the FFT product with its rounding check.
#include <math.h>

#include <mutex>
#include <vector>

#include "carry.cuh"
#include "common.cuh"
#include "fft.cuh"
#include "mul.cuh"
#include "ntt.cuh"
#include "passes.cuh"

namespace pic {

static constexpr int kFftInnerBits = 13;  // in-CTA sub-transforms up to 2^13 points
static constexpr int kFftK = 30;          // outer twiddle order 2^30
static constexpr int kFftS = 15;          // outer split e = hi * 2^15 + lo

struct FftTables {
    double2* inner = nullptr;  // exp(+2 pi i j / 2^13), j < 2^12
    double2* lvl = nullptr;    // the same by level: exp(+2 pi i e / 2^m), e < 2^(m-1), at 2^(m-1) - 1 + e
    double2* olo = nullptr;    // exp(+2 pi i j / 2^30), j < 2^15
    double2* ohi = nullptr;    // exp(+2 pi i j 2^15 / 2^30), j < 2^15
};

static std::once_flag g_fft_once;
static FftTables g_fft;

static double2* upload2(const std::vector<double2>& v)
{
    double2* d = nullptr;
    PIC_CUDA(raw_dev_alloc((void**)&d, v.size() * sizeof(double2)));
    PIC_CUDA(cudaMemcpy(d, v.data(), v.size() * sizeof(double2), cudaMemcpyHostToDevice));
    return d;
}

// Table entries are cos/sin of 2 pi j / 2^m evaluated directly per entry, as
// fft_ensure_table does (FFT.cpp:45-56), never by recurrence.
static const FftTables& fft_tables()
{
    std::call_once(g_fft_once, [] {
        const double two_pi = 6.283185307179586476925286766559;
        std::vector<double2> in((size_t)1 << (kFftInnerBits - 1));
        for (size_t j = 0; j < in.size(); j++) {
            const double a = two_pi * (double)j / (double)(1 << kFftInnerBits);
            in[j] = make_double2(cos(a), sin(a));
        }
        std::vector<double2> lo((size_t)1 << kFftS), hi((size_t)1 << (kFftK - kFftS));
        for (size_t j = 0; j < lo.size(); j++) {
            const double a = two_pi * (double)j / (double)(1u << kFftK);
            lo[j] = make_double2(cos(a), sin(a));
        }
        for (size_t j = 0; j < hi.size(); j++) {
            const double a = two_pi * (double)j / (double)(1u << (kFftK - kFftS));
            hi[j] = make_double2(cos(a), sin(a));
        }
        std::vector<double2> lv((size_t)1 << kFftInnerBits);
        for (int m = 1; m <= kFftInnerBits; m++)
            for (size_t e = 0; e < ((size_t)1 << (m - 1)); e++)
                lv[((size_t)1 << (m - 1)) - 1 + e] = in[e << (kFftInnerBits - m)];
        g_fft.inner = upload2(in);
        g_fft.lvl = upload2(lv);
        g_fft.olo = upload2(lo);
        g_fft.ohi = upload2(hi);
    });
    return g_fft;
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b)  // a * conj(b)
{
    return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

template <int B, bool INV>
__device__ __forceinline__ void fft_group(double2 (&x)[1 << B], int j, int lst, const double2* __restrict__ tw)
{
    if (!INV) {
#pragma unroll
        for (int l = 0; l < B; l++) {
            const int hm = 1 << (B - 1 - l);
            const int shift = kFftInnerBits - (B - l) - lst;
#pragma unroll
            for (int m = 0; m < (1 << B); m++) {
                if (m & hm) continue;
                const int t = j + ((m & (hm - 1)) << lst);
                const double2 w = __ldg(tw + (t << shift));
                const double2 a = x[m], b = x[m + hm];
                x[m] = cadd(a, b);
                x[m + hm] = cmul(csub(a, b), w);
            }
        }
    } else {
#pragma unroll
        for (int l = B - 1; l >= 0; l--) {
            const int hm = 1 << (B - 1 - l);
            const int shift = kFftInnerBits - (B - l) - lst;
#pragma unroll
            for (int m = 0; m < (1 << B); m++) {
                if (m & hm) continue;
                const int t = j + ((m & (hm - 1)) << lst);
                const double2 w = __ldg(tw + (t << shift));
                const double2 a = x[m], b = cmulc(x[m + hm], w);
                x[m] = cadd(a, b);
                x[m + hm] = csub(a, b);
            }
        }
    }
}

template <int B, bool INV>
__device__ __forceinline__ void fft_run_group(double2* ptr, int base, int j, int lst, int es, const double2* tw)
{
    double2 x[1 << B];
#pragma unroll
    for (int m = 0; m < (1 << B); m++) x[m] = ptr[(size_t)(base + (m << lst)) * es];
    fft_group<B, INV>(x, j, lst, tw);
#pragma unroll
    for (int m = 0; m < (1 << B); m++) ptr[(size_t)(base + (m << lst)) * es] = x[m];
}

template <bool INV>
__device__ void cta_fft(double2* s, int logn, int nt, int es, int ts, bool tr_fast, const double2* tw)
{
    const int nfull = logn / 3, rem = logn % 3;
    const int nr = nfull + (rem ? 1 : 0);
    for (int ri = 0; ri < nr; ri++) {
        const int r = INV ? (nr - 1 - ri) : ri;
        const int b = (r < nfull) ? 3 : rem;
        const int lB = logn - 3 * r;
        const int lst = lB - b;
        const int lgpt = logn - b;
        const int G = nt << lgpt;
        for (int g = threadIdx.x; g < G; g += blockDim.x) {
            int tr, gi;
            if (tr_fast) {
                tr = g % nt;
                gi = g / nt;
            } else {
                tr = g >> lgpt;
                gi = g & ((1 << lgpt) - 1);
            }
            const int sb = gi >> lst, j = gi & ((1 << lst) - 1);
            const int base = (sb << lB) + j;
            double2* ptr = s + (size_t)tr * ts;
            if (b == 3) fft_run_group<3, INV>(ptr, base, j, lst, es, tw);
            else if (b == 2) fft_run_group<2, INV>(ptr, base, j, lst, es, tw);
            else fft_run_group<1, INV>(ptr, base, j, lst, es, tw);
        }
        __syncthreads();
    }
}

__device__ __forceinline__ double2 fft_outer_root(const double2* lo, const double2* hi, uint64_t e, int lM)
{
    const uint64_t E = e << (kFftK - lM);
    return cmul(__ldg(hi + (E >> kFftS)), __ldg(lo + (E & ((1u << kFftS) - 1))));
}

template <bool INV>
__global__ void __launch_bounds__(512) fft_rows_kernel(FftBatch B, int k, int lr, int rpc, const double2* tw)
{
    extern __shared__ double2 fsm[];
    const int n = 1 << lr;
    const size_t rows_per_tr = (size_t)1 << (k - lr);
    const size_t row0 = (size_t)blockIdx.x * rpc;
    for (int idx = threadIdx.x; idx < rpc * n; idx += blockDim.x) {
        const size_t row = row0 + idx / n;
        const size_t tr = row / rows_per_tr, rr = row % rows_per_tr;
        fsm[idx] = B.data[tr * B.stride + (rr << lr) + idx % n];
    }
    __syncthreads();
    cta_fft<INV>(fsm, lr, rpc, 1, n, false, tw);
    for (int idx = threadIdx.x; idx < rpc * n; idx += blockDim.x) {
        const size_t row = row0 + idx / n;
        const size_t tr = row / rows_per_tr, rr = row % rows_per_tr;
        B.data[tr * B.stride + (rr << lr) + idx % n] = fsm[idx];
    }
}

// ---- passes with compile-time rounds (transforms longer than one CTA's) --------
// The butterflies, twiddle values and their order are those of the general
// kernels above, which serve the single-pass lengths; here the strides fold away,
// consecutive lanes read consecutive twiddles, the first round reads and the
// last writes global memory, and the shared-memory places keep eight lanes' 16
// bytes in different banks.  Bound by latency (three CTAs
// per SM, 64 - 84 registers) while the data stays in L2: forward passes of 2^20
// points 28.9 us (rows) and 27.8 (columns) before, 12.2 and 15.4 here; the FFT.h
// flow at 2^20 245 -> 148 us.

// Bits 3, 4, 5 of a row's element XORed into bits 0, 1, 2 (rounds at strides
// 2^8, 2^5, 2^2, 1 of 11-bit rows).
__host__ __device__ constexpr int fft_place(int e) { return e ^ ((e >> 3) & 7); }
// A column tile's (row << LW) + column, 2^LW >= 4: rows eight apart.
template <int LW>
__host__ __device__ constexpr int fft_col_place(int e)
{
    return LW == 2 ? e ^ (((e >> 5) & 1) << 2) : e;
}

template <int B, bool INV, int LST>
__device__ __forceinline__ void fft_levels(double2 (&x)[1 << B], int j, const double2* __restrict__ lvl)
{
#pragma unroll
    for (int q = 0; q < B; q++) {
        const int l = INV ? B - 1 - q : q;
        const int hm = 1 << (B - 1 - l);
#pragma unroll
        for (int m = 0; m < (1 << B); m++) {
            if (m & hm) continue;
            const double2 w = __ldg(lvl + ((1 << (B - l + LST - 1)) - 1) + j + ((m & (hm - 1)) << LST));
            if (!INV) {
                const double2 a = x[m], b = x[m + hm];
                x[m] = cadd(a, b);
                x[m + hm] = cmul(csub(a, b), w);
            } else {
                const double2 a = x[m], b = cmulc(x[m + hm], w);
                x[m] = cadd(a, b);
                x[m + hm] = csub(a, b);
            }
        }
    }
}

constexpr int kFftThreads = 256;
constexpr int kFftRowBits = 11;

template <bool INV>
__global__ void __launch_bounds__(kFftThreads, 3) fft_rows_fast_kernel(FftBatch B, int k,
                                                                       const double2* __restrict__ lvl)
{
    constexpr int LR = kFftRowBits, NR = RoundPlan<LR, 3>::NR;
    extern __shared__ double2 fsm[];
    const int lrow = k - LR;
    double2* row = B.data + (blockIdx.x >> lrow) * B.stride + ((blockIdx.x & (((size_t)1 << lrow) - 1)) << LR);
    auto round = [&](auto rc) {
        constexpr int RR = INV ? NR - 1 - decltype(rc)::value : decltype(rc)::value;
        using At = typename RoundPlan<LR, 3>::template At<RR>;
        constexpr int Bb = At::B, LB = At::LB, LST = At::LST, E = 1 << Bb, G = 1 << (LR - Bb);
        constexpr bool FIRST = decltype(rc)::value == 0, LAST = decltype(rc)::value == NR - 1;
#pragma unroll 1
        for (int g = threadIdx.x; g < G; g += kFftThreads) {
            const int j = g & ((1 << LST) - 1), base = ((g >> LST) << LB) + j;
            double2 x[E];
#pragma unroll
            for (int m = 0; m < E; m++) {
                const int e = base + (m << LST);
                x[m] = FIRST ? row[e] : fsm[fft_place(e)];
            }
            fft_levels<Bb, INV, LST>(x, j, lvl);
#pragma unroll
            for (int m = 0; m < E; m++) {
                const int e = base + (m << LST);
                if (LAST) row[e] = x[m];
                else fsm[fft_place(e)] = x[m];
            }
        }
        if constexpr (!LAST) __syncthreads();
    };
    static_assert(NR == 4, "11-bit rows");
    round(std::integral_constant<int, 0>{});
    round(std::integral_constant<int, 1>{});
    round(std::integral_constant<int, 2>{});
    round(std::integral_constant<int, 3>{});
}

template <bool INV, int LC, int LW>
__global__ void __launch_bounds__(kFftThreads, 3)
    fft_cols_fast_kernel(FftBatch B, int k, int lpre, const double2* __restrict__ lvl, const double2* __restrict__ olo,
                         const double2* __restrict__ ohi)
{
    using Plan = RoundPlan<LC, 3>;
    constexpr int NR = Plan::NR, WMASK = (1 << LW) - 1;
    extern __shared__ double2 fsm[];
    const int lblock = k - lpre, lM = lblock - LC, ltiles = lM - LW;
    const size_t cta = blockIdx.x;
    const size_t tr = cta >> (ltiles + lpre), rem = cta & (((size_t)1 << (ltiles + lpre)) - 1);
    const size_t ob = rem >> ltiles;
    const int w = threadIdx.x & WMASK;
    const uint64_t c = ((rem & (((size_t)1 << ltiles) - 1)) << LW) + w;
    double2* col = B.data + tr * B.stride + (ob << lblock) + c;
    auto root = [&](int r) { return fft_outer_root(olo, ohi, c * (__brev((unsigned)r) >> (32 - LC)), lblock); };
    auto round = [&](auto rc) {
        constexpr int RR = INV ? NR - 1 - decltype(rc)::value : decltype(rc)::value;
        using At = typename Plan::template At<RR>;
        constexpr int Bb = At::B, LB = At::LB, LST = At::LST, E = 1 << Bb, G = 1 << (LC - Bb + LW);
        constexpr bool FIRST = decltype(rc)::value == 0, LAST = decltype(rc)::value == NR - 1;
#pragma unroll 1
        for (int g = threadIdx.x; g < G; g += kFftThreads) {
            const int gi = g >> LW, j = gi & ((1 << LST) - 1), r0 = ((gi >> LST) << LB) + j;
            double2 x[E];
#pragma unroll
            for (int m = 0; m < E; m++) {
                const int r = r0 + (m << LST);
                if (FIRST) {
                    x[m] = col[(size_t)r << lM];
                    if (INV) x[m] = cmulc(x[m], root(r));
                } else {
                    x[m] = fsm[fft_col_place<LW>((r << LW) + w)];
                }
            }
            fft_levels<Bb, INV, LST>(x, j, lvl);
#pragma unroll
            for (int m = 0; m < E; m++) {
                const int r = r0 + (m << LST);
                if (LAST) col[(size_t)r << lM] = INV ? x[m] : cmul(x[m], root(r));
                else fsm[fft_col_place<LW>((r << LW) + w)] = x[m];
            }
        }
        if constexpr (!LAST) __syncthreads();
    };
    round(std::integral_constant<int, 0>{});
    if constexpr (NR > 1) round(std::integral_constant<int, 1>{});
    if constexpr (NR > 2) round(std::integral_constant<int, 2>{});
}

static void fft_rows_fast(bool inv, const FftBatch& b, int k, cudaStream_t s)
{
    const size_t grid = (size_t)b.count << (k - kFftRowBits);
    const size_t smem = sizeof(double2) << kFftRowBits;
    if (inv) fft_rows_fast_kernel<true><<<(unsigned)grid, kFftThreads, smem, s>>>(b, k, fft_tables().lvl);
    else fft_rows_fast_kernel<false><<<(unsigned)grid, kFftThreads, smem, s>>>(b, k, fft_tables().lvl);
}

// 2^11-point tiles: a group of every round per thread.
template <int LC>
static void fft_cols_fast(bool inv, const FftBatch& b, int k, int lpre, cudaStream_t s)
{
    constexpr int LW = 11 - LC > 8 ? 8 : 11 - LC;
    const FftTables& T = fft_tables();
    const size_t grid = (size_t)b.count << (k - LC - LW);
    const size_t smem = RoundPlan<LC, 3>::NR > 1 ? sizeof(double2) << (LC + LW) : 0;
    if (inv) fft_cols_fast_kernel<true, LC, LW><<<(unsigned)grid, kFftThreads, smem, s>>>(b, k, lpre, T.lvl, T.olo, T.ohi);
    else fft_cols_fast_kernel<false, LC, LW><<<(unsigned)grid, kFftThreads, smem, s>>>(b, k, lpre, T.lvl, T.olo, T.ohi);
}

static std::vector<int> fft_pass_bits(int k)
{
    std::vector<int> bits;
    if (k <= kFftInnerBits) {
        bits.push_back(k);
        return bits;
    }
    const int row = kFftRowBits, colmax = 9;  // 16-byte points: half the NTT's tile
    int rest = k - row;
    const int ncol = (rest + colmax - 1) / colmax;
    for (int i = 0; i < ncol; i++) {
        const int b = rest / (ncol - i) + ((rest % (ncol - i)) ? 1 : 0);
        bits.push_back(b);
        rest -= b;
    }
    bits.push_back(row);
    return bits;
}

static void fft_launch_rows(bool inv, const FftBatch& b, int k, int lr, cudaStream_t s)
{
    const FftTables& T = fft_tables();
    const int n = 1 << lr;
    int rpc = 1;
    if (lr == k) {
        rpc = (1 << 10) / n;
        if (rpc < 1) rpc = 1;
        while (rpc > 1 && (b.count % rpc)) rpc >>= 1;
    }
    const size_t grid = ((size_t)b.count << (k - lr)) / rpc;
    ProfScope ps(KC_FFT_ROWS, 32.0 * (double)b.count * (double)((size_t)1 << k), s);
    if (lr < k) {
        fft_rows_fast(inv, b, k, s);
        PIC_CHECK_LAUNCH();
        count_launch();
        return;
    }
    constexpr size_t kFftRowSmem = sizeof(double2) << kFftInnerBits;  // the longest single pass
    const size_t smem = (size_t)rpc * n * sizeof(double2);
    int threads = (rpc * n) / 8;
    if (threads < 32) threads = 32;
    if (threads > 512) threads = 512;
    if (inv) {
        allow_smem(fft_rows_kernel<true>, smem, kFftRowSmem);
        fft_rows_kernel<true><<<(unsigned)grid, threads, smem, s>>>(b, k, lr, rpc, T.inner);
    } else {
        allow_smem(fft_rows_kernel<false>, smem, kFftRowSmem);
        fft_rows_kernel<false><<<(unsigned)grid, threads, smem, s>>>(b, k, lr, rpc, T.inner);
    }
    PIC_CHECK_LAUNCH();
    count_launch();
}

static void fft_launch_cols(bool inv, const FftBatch& b, int k, int lpre, int lc, cudaStream_t s)
{
    ProfScope ps(KC_FFT_COLS, 32.0 * (double)b.count * (double)((size_t)1 << k), s);
    switch (lc) {
    case 3: fft_cols_fast<3>(inv, b, k, lpre, s); break;
    case 4: fft_cols_fast<4>(inv, b, k, lpre, s); break;
    case 5: fft_cols_fast<5>(inv, b, k, lpre, s); break;
    case 6: fft_cols_fast<6>(inv, b, k, lpre, s); break;
    case 7: fft_cols_fast<7>(inv, b, k, lpre, s); break;
    case 8: fft_cols_fast<8>(inv, b, k, lpre, s); break;
    case 9: fft_cols_fast<9>(inv, b, k, lpre, s); break;
    default: throw Error(PIC_ERR_INVALID, "FFT column pass outside its kernels' shapes");
    }
    PIC_CHECK_LAUNCH();
    count_launch();
}

void fft_forward_dif(const FftBatch& b, int k, cudaStream_t s)
{
    PIC_REQUIRE(k >= 1 && k <= kFftK, PIC_ERR_INVALID, "FFT length out of range");
    const std::vector<int> bits = fft_pass_bits(k);
    int lpre = 0;
    for (size_t i = 0; i + 1 < bits.size(); i++) {
        fft_launch_cols(false, b, k, lpre, bits[i], s);
        lpre += bits[i];
    }
    fft_launch_rows(false, b, k, bits.back(), s);
}

void fft_inverse_dit(const FftBatch& b, int k, cudaStream_t s)
{
    PIC_REQUIRE(k >= 1 && k <= kFftK, PIC_ERR_INVALID, "FFT length out of range");
    const std::vector<int> bits = fft_pass_bits(k);
    fft_launch_rows(true, b, k, bits.back(), s);
    int lpre = k - bits.back();
    for (int i = (int)bits.size() - 2; i >= 0; i--) {
        lpre -= bits[i];
        fft_launch_cols(true, b, k, lpre, bits[i], s);
    }
}

__global__ void fft_pointwise_kernel(double2* T, const double2* A, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        T[i] = cmul(T[i], A[i]);
}

void fft_pointwise(double2* T, const double2* A, size_t n, cudaStream_t s)
{
    fft_pointwise_kernel<<<grid_for(n, 256), 256, 0, s>>>(T, A, n);
    PIC_CHECK_LAUNCH();
    count_launch();
}

// Worst-case rounding error of a length-2^k FFT convolution of b-bit pieces,
// after C. Percival, "Rapid multiplication modulo the sum and difference of
// highly composite numbers" (Math. Comp. 72, 2003), Theorem 5.1:
//   err <= N X Y [ (1+e)^(3k) (1+e sqrt5)^(3k+1) (1+beta)^(3k) - 1 ]
// with X = Y = 2^b - 1, e = 2^-53 and beta the twiddle error (2.5 e here: each
// outer twiddle is the rounded product of two rounded table entries).
double fft_error_bound(int k, int bits)
{
    const double e = ldexp(1.0, -53), beta = 2.5 * e;
    const double X = ldexp(1.0, bits) - 1.0;
    const double lg = 3.0 * k * log1p(e) + (3.0 * k + 1) * log1p(e * sqrt(5.0)) + 3.0 * k * log1p(beta);
    return ldexp(1.0, k) * X * X * expm1(lg);
}

int fft_piece_bits(int k)
{
    for (int b = 16; b >= 8; b--)
        if (fft_error_bound(k, b) < 0.25) return b;
    return 0;
}

__global__ void fft_split_kernel(double2* T, size_t N, const uint32_t* A, size_t AL, int bits)
{
    const uint32_t mask = (1u << bits) - 1u;
    const size_t nbits = AL * 32;
    for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < N; j += (size_t)gridDim.x * blockDim.x) {
        double v = 0;
        const size_t b0 = j * (size_t)bits;
        if (b0 < nbits) {
            const size_t w = b0 >> 5;
            const int r = (int)(b0 & 31);
            uint64_t x = A[w];
            if (w + 1 < AL) x |= (uint64_t)A[w + 1] << 32;
            v = (double)((uint32_t)(x >> r) & mask);
        }
        T[j] = make_double2(v, 0.0);
    }
}

void fft_split(double2* T, int k, const uint32_t* A, size_t AL, int bits, cudaStream_t s)
{
    const size_t N = (size_t)1 << k;
    fft_split_kernel<<<grid_for(N, 256), 256, 0, s>>>(T, N, A, AL, bits);
    PIC_CHECK_LAUNCH();
    count_launch();
}

bool mul_fft(uint32_t* z, const uint32_t* a, size_t na, const uint32_t* b, size_t nb, cudaStream_t s,
             double* max_err)
{
    const size_t zw = na + nb;
    int k = 1, bits = 0;
    for (k = 1; k <= kFftK; k++) {
        const int bb = fft_piece_bits(k);
        if (bb == 0) break;
        if (((size_t)1 << k) * (size_t)bb >= 32 * zw) {
            bits = bb;
            break;
        }
    }
    PIC_REQUIRE(bits != 0, PIC_ERR_LENGTH, "product too long for a provably exact FP64 FFT");
    const size_t N = (size_t)1 << k;
    const bool square = (a == b && na == nb);
    DevBuf<double2> A(N, s), B(square ? 0 : N, s);
    fft_split(A.get(), k, a, na, bits, s);
    fft_forward_dif(FftBatch{A.get(), N, 1}, k, s);
    if (!square) {
        fft_split(B.get(), k, b, nb, bits, s);
        fft_forward_dif(FftBatch{B.get(), N, 1}, k, s);
    }
    fft_pointwise(A.get(), square ? A.get() : B.get(), N, s);
    fft_inverse_dit(FftBatch{A.get(), N, 1}, k, s);
    const size_t ncoef = (32 * zw + bits - 1) / bits;
    const double err = fft_coef_to_words(A.get(), ncoef < N ? ncoef : N, 1.0 / (double)N, bits, z, zw, s);
    fft_note_max_err(err);
    if (max_err) *max_err = err;
    return err <= 0.25;
}

}  // namespace pic
