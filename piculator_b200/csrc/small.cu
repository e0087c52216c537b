// Short products of the FP64 form in one launch (PIC_MUL_NTT3D with at most 2^13
// coefficients, and the batches of such products).
//
// A cluster of three CTAs multiplies two operands, one CTA per prime: it reads
// the operands' pieces, transforms both in shared memory, multiplies and
// transforms back (middle.cuh), all without leaving the SM; then each CTA
// takes a third of the product's words, reads the other two primes' residues
// through distributed shared memory for the CRT and passes its carry on the
// same way.  A product of this length is bound by latency: as separate
// launches (forward, product and inverse of a main and a tail transform,
// fix-up, CRT, carries) one of 4096-word operands took 45 us, here 33; in a
// batch the residues' HBM traffic goes too (8192 products of 1 .. 8192 words:
// 1.29 ms with the integer form's bins, now 0.95).  About 13 us of the 33 are
// the FP64 work of one prime on one SM, the rest launch, barriers and exchanges.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "crt56.cuh"
#include "middle.cuh"
#include "mul.cuh"

namespace cg = cooperative_groups;

namespace pic {

struct SmallArgs {
    const DevDesc* d;     // null: the product(s) below
    const uint32_t* idx;  // product i is d[idx[i]]
    DevDesc one;
    size_t zs, as;  // without d: product i is one.z + i zs = (one.a + i as) one.b
    MailRef mail;  // the product's top word
    CrtDConsts C;
    PrimeDev prime[3];
};

template <int LR>
struct SmallShape {
    static constexpr int TOT = 1 << LR;
    static constexpr int PER = (TOT / 8 + 3) / 3;                // groups per CTA, at most
    static constexpr int XS = (crt_slot(8 * PER + 3) + 1) & ~1;  // digit slots
    static constexpr size_t SMEM = 8 * (size_t)TOT + std::max(8 * (size_t)TOT, sizeof(CrtDigits<XS>));
};

// Operand rows a, b; afterwards row 0 holds the residues and b's place the
// coefficients' limbs.  64 registers a thread, so that a batch keeps 32 warps
// on an SM (2^12 coefficients: 320 us of the batch above, 427 with 16 warps and
// no spills).
template <int LR>
__global__ void __cluster_dims__(3, 1, 1) __launch_bounds__(MiddleShape<LR, 0>::NT, 1024 / MiddleShape<LR, 0>::NT)
    product_small_kernel(const __grid_constant__ SmallArgs M)
{
    using Sh = MiddleShape<LR, 0>;
    constexpr int TOT = Sh::TOT, NT = Sh::NT;
    extern __shared__ double ms[];
    __shared__ uint32_t s_total;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t q = blockIdx.x % 3, item = blockIdx.x / 3;
    const PrimeDev& P = q == 0 ? M.prime[0] : (q == 1 ? M.prime[1] : M.prime[2]);
    const Dbl::Ctx L = Dbl::ctx(P);
    const double* __restrict__ tf = reinterpret_cast<const double*>(P.lvl_fwd);
    const double* __restrict__ ti = reinterpret_cast<const double*>(P.lvl_inv);
    DevDesc D = M.one;
    if (M.d != nullptr) {
        D = M.d[M.idx[item]];
    } else {
        D.z += item * M.zs;
        D.a += item * M.as;
    }
    const bool square = D.a == D.b && D.na == D.nb;
    auto in = [&](int i, int, int e) -> double {
        return dpiece56(src_piece56_raw(i == 0 ? D.a : D.b, i == 0 ? D.na : D.nb, e), L.p, L.pinv);
    };
    forward_rounds<LR, 0, 2, 0>(ms, L, tf, square ? 1 : 2, in);
    {
        using At = Round<LR, Sh::NR - 1>;
        constexpr int B = At::B, E = 1 << B, G = TOT >> B;
        GroupTw<B, 0> wf, wi;
        wf.load(tf, 0);
        wi.load(ti, 0);
#pragma unroll 1
        for (int g = threadIdx.x; g < G; g += NT) {
            const int pb = place(g << B);
            double x[E], y[E];
            auto load = [&](int i, double(&v)[E]) {
#pragma unroll
                for (int m = 0; m < E; m++) v[m] = ms[i * TOT + place_at(pb, m)];
                if (i == 1 || square) fwd_last<B, true>(v, wf, L);
                else fwd_last<B, false>(v, wf, L);
            };
            load(0, x);
            if (!square) load(1, y);
#pragma unroll
            for (int m = 0; m < E; m++) x[m] = dmul_mod(x[m], square ? x[m] : y[m], L.p, L.pinv);
            inv_first<B, LR, 1>(x, wi, L);
#pragma unroll
            for (int m = 0; m < E; m++) ms[place_at(pb, m)] = x[m];
        }
    }
    auto act = [](int) { return 0; };
    auto out = [&](int, int, int e, double v) { ms[place(e)] = v; };
    inverse_rounds<LR, 0, Sh::NR - 2>(ms, L, ti, 1, act, out);
    cluster.sync();
    // words: 14 per group of 8 coefficients, a third of the groups per CTA
    const double* Y[3];
#pragma unroll
    for (int r = 0; r < 3; r++) Y[r] = cluster.map_shared_rank(ms, r);
    const uint32_t zw = D.na + D.nb;
    const int ncoef = (int)((32 * (size_t)D.na + 55) / 56 + (32 * (size_t)D.nb + 55) / 56 - 1);
    const int jlim = min(ncoef, (int)((32 * (size_t)zw + 55) / 56));
    const int groups = (int)((zw + 13) / 14), per = (groups + 2) / 3;
    const int u = (int)q * per + (int)threadIdx.x;
    const bool mine = (int)threadIdx.x < per && u < groups;
    using Digits = CrtDigits<SmallShape<LR>::XS>;
    Digits& X = *reinterpret_cast<Digits*>(ms + TOT);  // b's place and some more
    const int j0 = 8 * (int)q * per - 3;
    crt_coefs(X, 8 * per + 3, M.C, [&](int i) { return j0 + i < jlim ? (int64_t)(j0 + i) : (int64_t)-1; },
              [&](int64_t j, double& y0, double& y1, double& y2) {
                  const int at = place((int)j);
                  y0 = Y[0][at];
                  y1 = Y[1][at];
                  y2 = Y[2][at];
              },
              [](int64_t, double&, double&, double&) {});
    __syncthreads();
    uint64_t t[8];
    if (mine) crt_group(X, 8 * (int)threadIdx.x + 3, t);
    const size_t wb = 14 * (size_t)q * per, we = min((size_t)zw, wb + 14 * (size_t)per);
    uint32_t* W = reinterpret_cast<uint32_t*>(ms + TOT);
    digits_to_words(t, mine, false, W, &s_total);
    for (size_t i = wb + threadIdx.x; i < we; i += NT) D.z[i] = W[i - wb];
    cluster.sync();
    uint32_t cin = 0;
    for (uint32_t r = 0; r < q; r++) {
        const uint32_t gp = *cluster.map_shared_rank(&s_total, r);
        cin = (gp & 1u) | ((gp >> 1) & cin);
    }
    if (cin) chunk_ripple(D.z, wb, we, false);
    if (M.mail.slot != nullptr && wb < zw && zw <= we) {
        __syncthreads();
        if (threadIdx.x == 0) mail_post(M.mail, D.z[zw - 1]);
    }
    cluster.sync();  // the others may still read this CTA's total
}

template <int LR>
static void launch_small(const SmallArgs& m, size_t count, cudaStream_t s)
{
    using Sh = MiddleShape<LR, 0>;
    const size_t smem = SmallShape<LR>::SMEM;
    auto kern = product_small_kernel<LR>;
    if (smem > 48 * 1024)
        PIC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<(unsigned)(3 * count), Sh::NT, smem, s>>>(m);
    PIC_CHECK_LAUNCH();
    count_launch();
}

static void small_products(SmallArgs& m, size_t count, int k, cudaStream_t s)
{
    PIC_REQUIRE(count <= 0x7fffffffu / 3, PIC_ERR_INVALID, "too many products in one launch");
    k = std::max(k, kSmallMinBits);
    m.C = make_crtd(k, false);
    for (int q = 0; q < 3; q++) m.prime[q] = dbl_prime_tables(kDblPrimes[q]).dev;
    ProfScope ps(KC_NTT_MIDDLE, 3.0 * (double)((size_t)count << k) * 24.0, s);
    switch (k) {
    case 8: launch_small<8>(m, count, s); break;
    case 9: launch_small<9>(m, count, s); break;
    case 10: launch_small<10>(m, count, s); break;
    case 11: launch_small<11>(m, count, s); break;
    case 12: launch_small<12>(m, count, s); break;
    case 13: launch_small<13>(m, count, s); break;
    default: throw Error(PIC_ERR_LENGTH, "product too long for one launch");
    }
}

void mul_small(uint32_t* z, const uint32_t* a, size_t na, const uint32_t* b, size_t nb, cudaStream_t s, Mail* mail)
{
    const size_t ncoef = pieces56(na) + pieces56(nb) - 1;
    int k = kSmallMinBits;
    while (((size_t)1 << k) < ncoef) k++;
    SmallArgs m{};
    m.one = DevDesc{z, a, b, (uint32_t)na, (uint32_t)nb};
    if (mail) m.mail = mail->ref();
    small_products(m, 1, k, s);
}

bool mul_small_uniform(uint32_t* z, size_t zs, const uint32_t* a, size_t as, size_t na, const uint32_t* b, size_t nb,
                       size_t count, cudaStream_t s)
{
    if (count == 0) return true;
    const size_t ncoef = pieces56(na) + pieces56(nb) - 1;
    if (mul_auto_mode(na, nb) != PIC_MUL_NTT3D || ncoef > ((size_t)1 << kSmallMaxBits)) return false;
    int k = kSmallMinBits;
    while (((size_t)1 << k) < ncoef) k++;
    SmallArgs m{};
    m.one = DevDesc{z, a, b, (uint32_t)na, (uint32_t)nb};
    m.zs = zs;
    m.as = as;
    count_products(count);
    small_products(m, count, k, s);
    return true;
}

void mul_small_batch(const DevDesc* d, const uint32_t* idx, size_t count, int k, cudaStream_t s)
{
    if (count == 0) return;
    SmallArgs m{};
    m.d = d;
    m.idx = idx;
    small_products(m, count, k, s);
}

}  // namespace pic
