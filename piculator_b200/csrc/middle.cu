// Fused middle passes of the FP64 product form (see ntt.cuh).
//
// A product needs, after the column passes, the forward row pass of each
// operand, a pointwise product and the inverse row pass of each result.  Rows
// are contiguous and the three steps keep a row's points in place, so one CTA
// takes the same row of every operand through all of them in shared memory:
// the row passes' own HBM traffic (16 B a point and pass) and the pointwise
// kernel's (80 B per parent point of a merge) become one read of the operands
// and one write of the results, 72 B per parent point of a merge instead of 224.
// The last forward round, the pointwise product and the first inverse round
// work on the same groups of points, so they run in registers without an
// exchange between them.  A thread takes the same group of every operand, so a
// round's twiddles are loaded once for all of them.
//
// Merges of a pi computation at 1e9 digits (binary splitting, one B200): a
// level of 2^17-point transforms 64.4 -> 54.5 ms, of 2^12 points 55.8 -> 38.6,
// the whole computation 1.73 -> 1.49 s, against the same passes launched
// apart.  What is left in the kernel is FP64 work (about 415 instructions per
// parent point and prime: 6 forward and 3 inverse rows of 11 levels; 16 more with
// the products by one and a reduction of every last sum: the merges' middle
// passes 409 ms for 401, a whole computation 1.2005 s for 1.1945) with two
// CTAs of 256 threads per SM, the rows' 96 KB of shared memory being the limit.
// One product (two operands, 24 B a point instead of 72): 2^24-word operands
// 4.00 -> 3.32 ms, 1,048,573 x 400,009 words 186 -> 146 us, 4096 words 82 -> 45
// us (the operands' pieces are read by the first pass, 16 launches -> 8).
#include <algorithm>

#include "common.cuh"
#include "middle.cuh"

namespace pic {

struct MergeMiddleDev {
    uint64_t* arr[3];  // P, Q, R
    SplitSrc src[3];
    size_t stride;
    uint32_t np;
    uint32_t blocks;  // CTAs per prime
    const uint8_t* sgn;
    int need_r;
    PrimeDev prime[3];
};

// Operand rows of a merge in shared memory: PL, PR, QL, QR, RL, RR.
template <int LR, int LT, bool SRC>
__global__ void __launch_bounds__(MiddleShape<LR, LT>::NT, MiddleShape<LR, LT>::NT > 256 ? 1 : 2)
    merge_middle_kernel(const __grid_constant__ MergeMiddleDev M, int lrow)
{
    using Sh = MiddleShape<LR, LT>;
    constexpr int TOT = Sh::TOT;
    extern __shared__ double ms[];
    const uint32_t q = blockIdx.x / M.blocks, cb = blockIdx.x - q * M.blocks;
    const PrimeDev& P = q == 0 ? M.prime[0] : (q == 1 ? M.prime[1] : M.prime[2]);
    const Dbl::Ctx L = Dbl::ctx(P);
    const double* __restrict__ tf = reinterpret_cast<const double*>(P.lvl_fwd);
    const double* __restrict__ ti = reinterpret_cast<const double*>(P.lvl_inv);
    const size_t row0 = (size_t)cb << LT;  // (parent, row) pairs, 2^lrow rows a parent
    const size_t nrows = (size_t)M.np << lrow;
    const size_t rmask = ((size_t)1 << lrow) - 1;
    // element e of operand a's row t: child 2 i + (a & 1) of array a / 2
    auto off = [&](int a, int t, int e) {
        const size_t row = row0 + t;
        const size_t item = (size_t)q * 2 * M.np + 2 * (row >> lrow) + (a & 1);
        return item * M.stride + ((row & rmask) << LR) + e;
    };
    auto pick = [&](int a) { return a < 2 ? M.arr[0] : (a < 4 ? M.arr[1] : M.arr[2]); };
    auto in = [&](int a, int t, int e) -> double {
        if (LT > 0 && row0 + t >= nrows) return 0.0;
        if constexpr (SRC) {  // lrow == 0: the row is child c of the source
            const SplitSrc& S = a < 2 ? M.src[0] : (a < 4 ? M.src[1] : M.src[2]);
            const size_t c = S.c0 + 2 * (row0 + t) + (a & 1);
            const uint32_t n = __ldg(S.len + c);
            return dpiece56(src_piece56_raw(S.words + c * (size_t)S.cap, n, S.first + e), L.p, L.pinv);
        } else {
            return dbits(pick(a)[off(a, t, e)]);
        }
    };
    auto put = [&](int a, int t, int e, double v) {
        if (LT == 0 || row0 + t < nrows) pick(a)[off(a, t, e)] = dstore(v);
    };
    const int nop = M.need_r ? 6 : 5;
    forward_rounds<LR, LT, 6, 0>(ms, L, tf, nop, in);
    // last forward round, pointwise products, first inverse round
    {
        using At = Round<LR, Sh::NR - 1>;
        constexpr int B = At::B, LST = At::LST, LG = LR - B, E = 1 << B;
        static_assert(LST == 0, "the last round has stride 1");
        constexpr int G = 1 << (LT + LG);
        GroupTw<B, 0> wf, wi;
        wf.load(tf, 0);
        wi.load(ti, 0);
#pragma unroll 1
        for (int g = threadIdx.x; g < G; g += Sh::NT) {
            const int t = g >> LG;
            const int pb = (t << LR) + place((g & ((1 << LG) - 1)) << B);
            const int base = (g & ((1 << LG) - 1)) << B;
            auto load = [&](int a, double(&x)[E]) {  // NR 1: the only round
#pragma unroll
                for (int m = 0; m < E; m++) x[m] = Sh::NR == 1 ? in(a, t, base + m) : ms[a * TOT + place_at(pb, m)];
                if (a == 3 || a == 4) fwd_last<B, true>(x, wf, L);  // QR and RL, in two products each
                else fwd_last<B, false>(x, wf, L);
            };
            auto store = [&](int a, double(&x)[E]) {
                inv_first<B, LR, 2>(x, wi, L);
#pragma unroll
                for (int m = 0; m < E; m++) {
                    if constexpr (Sh::NR == 1) put(a, t, base + m, x[m]);
                    else ms[a * TOT + place_at(pb, m)] = x[m];
                }
            };
            double qr[E], rl[E], x[E], y[E];
            load(3, qr);
            load(4, rl);
            load(0, x);
            load(1, y);
#pragma unroll
            for (int m = 0; m < E; m++) {
                x[m] = dmul_mod(x[m], qr[m], L.p, L.pinv);
                y[m] = dmul_mod(y[m], rl[m], L.p, L.pinv);
            }
            if (M.sgn != nullptr) {
                const size_t row = row0 + t;
                const size_t i = LT > 0 && row >= nrows ? 0 : row >> lrow;
                const bool same = (M.sgn[2 * i] != 0) == (M.sgn[2 * i + 1] != 0);
#pragma unroll
                for (int m = 0; m < E; m++) x[m] = __dadd_rn(x[m], same ? y[m] : -y[m]);
            } else {
                store(1, y);
            }
            store(0, x);
            load(2, x);
#pragma unroll
            for (int m = 0; m < E; m++) x[m] = dmul_mod(x[m], qr[m], L.p, L.pinv);
            store(2, x);
            if (M.need_r) {
                load(5, y);
#pragma unroll
                for (int m = 0; m < E; m++) y[m] = dmul_mod(y[m], rl[m], L.p, L.pinv);
                store(4, y);
            }
        }
    }
    // results in rows 0 (T1 or V), 2 (Q), 4 (R), 1 (T2)
    const int apart = M.sgn == nullptr;
    const int nout = 2 + (M.need_r ? 1 : 0) + apart;
    auto act = [&](int i) { return i == nout - 1 && apart ? 1 : 2 * i; };
    auto out = [&](int i, int t, int e, double v) { put(act(i), t, e, v); };
    if constexpr (Sh::NR > 1) inverse_rounds<LR, LT, Sh::NR - 2>(ms, L, ti, nout, act, out);
}

int middle_row_bits(int k) { return k <= 12 ? k : 11; }

template <int LR, bool SRC>
static void launch_merge_middle(const MergeMiddle& m, int k, cudaStream_t s)
{
    constexpr int LT = LR < 11 ? 11 - LR : 0;
    using Sh = MiddleShape<LR, LT>;
    MergeMiddleDev d;
    d.arr[0] = m.P;
    d.arr[1] = m.Q;
    d.arr[2] = m.R;
    d.src[0] = m.sP;
    d.src[1] = m.sQ;
    d.src[2] = m.sR;
    d.stride = m.stride;
    d.np = (uint32_t)m.np;
    d.sgn = m.sgn;
    d.need_r = m.need_r ? 1 : 0;
    for (int q = 0; q < 3; q++) d.prime[q] = dbl_prime_tables(kDblPrimes[q]).dev;
    const size_t rows = m.np << (k - LR);
    const size_t blocks = (rows + ((size_t)1 << LT) - 1) >> LT;
    PIC_REQUIRE(3 * blocks <= 0x7fffffffu, PIC_ERR_INVALID, "merge grid too large");
    d.blocks = (uint32_t)blocks;
    const size_t smem = sizeof(double) * 6 * Sh::TOT;
    auto kern = merge_middle_kernel<LR, LT, SRC>;
    PIC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<(unsigned)(3 * blocks), Sh::NT, smem, s>>>(d, k - LR);
    PIC_CHECK_LAUNCH();
    count_launch();
}

void ntt_merge_middle(const MergeMiddle& m, int k, cudaStream_t s)
{
    // 6 rows read and 3 (or 4) written per row of a parent
    ProfScope ps(KC_NTT_MIDDLE, 3.0 * (double)m.np * (double)((size_t)1 << k) * 72.0, s);
    const int lr = middle_row_bits(k);
    if (lr < k) {
        launch_merge_middle<11, false>(m, k, s);
        return;
    }
    switch (lr) {
    case 2: launch_merge_middle<2, true>(m, k, s); break;
    case 3: launch_merge_middle<3, true>(m, k, s); break;
    case 4: launch_merge_middle<4, true>(m, k, s); break;
    case 5: launch_merge_middle<5, true>(m, k, s); break;
    case 6: launch_merge_middle<6, true>(m, k, s); break;
    case 7: launch_merge_middle<7, true>(m, k, s); break;
    case 8: launch_merge_middle<8, true>(m, k, s); break;
    case 9: launch_merge_middle<9, true>(m, k, s); break;
    case 10: launch_merge_middle<10, true>(m, k, s); break;
    case 11: launch_merge_middle<11, true>(m, k, s); break;
    case 12: launch_merge_middle<12, true>(m, k, s); break;
    default: throw Error(PIC_ERR_INVALID, "merge transform too short");
    }
}

// ---- one product -----------------------------------------------------------------
struct ProductMiddleDev {
    uint64_t* out;
    const uint64_t *a, *b;
    uint64_t* spec;
    size_t out_stride, a_stride, b_stride, spec_stride;
    SplitSrc sa, sb;
    uint32_t blocks;  // CTAs per prime
    int square, spec_ready;
    PrimeDev prime[3];
};

// Operand rows in shared memory: a, b (one row in a square, or with a spectrum
// read in place of the other operand).  Three CTAs of 256 threads per SM: the
// register budget of four (64) spills.
template <int LR, int LT, bool SRC>
__global__ void __launch_bounds__(MiddleShape<LR, LT>::NT, MiddleShape<LR, LT>::NT > 256 ? 1 : 3)
    product_middle_kernel(const __grid_constant__ ProductMiddleDev M, int lrow)
{
    using Sh = MiddleShape<LR, LT>;
    constexpr int TOT = Sh::TOT;
    static_assert(Sh::NR > 1, "rows of at least two rounds");
    extern __shared__ double ms[];
    const uint32_t q = blockIdx.x / M.blocks, cb = blockIdx.x - q * M.blocks;
    const PrimeDev& P = q == 0 ? M.prime[0] : (q == 1 ? M.prime[1] : M.prime[2]);
    const Dbl::Ctx L = Dbl::ctx(P);
    const double* __restrict__ tf = reinterpret_cast<const double*>(P.lvl_fwd);
    const double* __restrict__ ti = reinterpret_cast<const double*>(P.lvl_inv);
    const size_t row0 = (size_t)cb << LT, nrows = (size_t)1 << lrow;
    // rows to transform: a (unless it is a square of a ready spectrum), then b
    const bool need_a = !(M.square && M.spec_ready), need_b = !M.square && !M.spec_ready;
    const int nop = (need_a ? 1 : 0) + (need_b ? 1 : 0);
    auto in = [&](int i, int t, int e) -> double {
        if (LT > 0 && row0 + t >= nrows) return 0.0;
        if constexpr (SRC) {
            const SplitSrc& S = i == 0 ? M.sa : M.sb;
            return dpiece56(src_piece56_raw(S.words, S.n, S.first + e), L.p, L.pinv);
        } else {
            return dbits((i == 0 ? M.a + q * M.a_stride : M.b + q * M.b_stride)[((row0 + t) << LR) + e]);
        }
    };
    forward_rounds<LR, LT, 2, 0>(ms, L, tf, nop, in);
    {
        using At = Round<LR, Sh::NR - 1>;
        constexpr int B = At::B, LG = LR - B, E = 1 << B;
        constexpr int G = 1 << (LT + LG);
        GroupTw<B, 0> wf, wi;
        wf.load(tf, 0);
        wi.load(ti, 0);
#pragma unroll 1
        for (int g = threadIdx.x; g < G; g += Sh::NT) {
            const int t = g >> LG;
            const int base = (g & ((1 << LG) - 1)) << B;
            const int pb = (t << LR) + place(base);
            const bool live = LT == 0 || row0 + t < nrows;
            uint64_t* sp = M.spec + q * M.spec_stride + ((row0 + t) << LR) + base;
            double x[E], y[E];
            auto load = [&](int i, double(&v)[E]) {
#pragma unroll
                for (int m = 0; m < E; m++) v[m] = ms[i * TOT + place_at(pb, m)];
                if (i == 1 || M.square) fwd_last<B, true>(v, wf, L);
                else fwd_last<B, false>(v, wf, L);
            };
            if (need_a) load(0, x);
            if (need_b) load(1, y);
            if (M.spec != nullptr && live) {
                double(&h)[E] = M.square ? x : y;
#pragma unroll
                for (int m = 0; m < E; m++) {
                    if (M.spec_ready) h[m] = dbits(sp[m]);
                    else sp[m] = dstore(h[m]);
                }
            }
#pragma unroll
            for (int m = 0; m < E; m++) x[m] = dmul_mod(x[m], M.square ? x[m] : y[m], L.p, L.pinv);
            inv_first<B, LR, 1>(x, wi, L);
#pragma unroll
            for (int m = 0; m < E; m++) ms[place_at(pb, m)] = x[m];
        }
    }
    auto act = [](int) { return 0; };
    auto out = [&](int, int t, int e, double v) {
        if (LT == 0 || row0 + t < nrows) M.out[q * M.out_stride + ((row0 + t) << LR) + e] = dstore(v);
    };
    inverse_rounds<LR, LT, Sh::NR - 2>(ms, L, ti, 1, act, out);
}

template <int LR, bool SRC>
static void launch_product_middle(const ProductMiddle& m, int k, cudaStream_t s)
{
    constexpr int LT = LR < 11 ? 11 - LR : 0;
    using Sh = MiddleShape<LR, LT>;
    ProductMiddleDev d;
    d.out = m.out;
    d.a = m.a;
    d.b = m.b;
    d.spec = m.spec;
    d.out_stride = m.out_stride;
    d.a_stride = m.a_stride;
    d.b_stride = m.b_stride;
    d.spec_stride = (size_t)1 << k;
    d.sa = m.sa;
    d.sb = m.sb;
    d.square = m.square ? 1 : 0;
    d.spec_ready = m.spec_ready ? 1 : 0;
    for (int q = 0; q < 3; q++) d.prime[q] = dbl_prime_tables(kDblPrimes[q]).dev;
    const size_t rows = (size_t)1 << (k - LR);
    d.blocks = (uint32_t)((rows + ((size_t)1 << LT) - 1) >> LT);
    const size_t smem = sizeof(double) * 2 * Sh::TOT;
    auto kern = product_middle_kernel<LR, LT, SRC>;
    if (smem > 48 * 1024) PIC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<3 * d.blocks, Sh::NT, smem, s>>>(d, k - LR);
    PIC_CHECK_LAUNCH();
    count_launch();
}

void ntt_product_middle(const ProductMiddle& m, int k, cudaStream_t s)
{
    // two rows read, one written
    ProfScope ps(KC_NTT_MIDDLE, 3.0 * (double)((size_t)1 << k) * 24.0, s);
    const int lr = middle_row_bits(k);
    if (lr < k) {
        launch_product_middle<11, false>(m, k, s);
        return;
    }
    switch (lr) {
    case 4: launch_product_middle<4, true>(m, k, s); break;
    case 5: launch_product_middle<5, true>(m, k, s); break;
    case 6: launch_product_middle<6, true>(m, k, s); break;
    case 7: launch_product_middle<7, true>(m, k, s); break;
    case 8: launch_product_middle<8, true>(m, k, s); break;
    case 9: launch_product_middle<9, true>(m, k, s); break;
    case 10: launch_product_middle<10, true>(m, k, s); break;
    case 11: launch_product_middle<11, true>(m, k, s); break;
    case 12: launch_product_middle<12, true>(m, k, s); break;
    default: throw Error(PIC_ERR_INVALID, "product transform too short");
    }
}

}  // namespace pic
