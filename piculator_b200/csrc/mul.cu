// Exact products: piece split, multi-prime NTT convolution, CRT and carry.
#include <math.h>
#include <string.h>

#include <atomic>
#include <utility>

#include "blockmul.cuh"
#include "carry.cuh"
#include "common.cuh"
#include "crt56.cuh"
#include "fp64mod.cuh"
#include "mul.cuh"

namespace pic {

static inline int ceil_log2(size_t n)
{
    int k = 0;
    while (((size_t)1 << k) < n) k++;
    return k;
}

// ---- split -----------------------------------------------------------------
// Three-prime form: piece j = a[2j] | a[2j+1] << 32, reduced mod each prime.
__global__ void split3_kernel(uint64_t* __restrict__ out, const uint32_t* __restrict__ a, size_t na, size_t N,
                              uint64_t p0, uint64_t p1, uint64_t p2)
{
    const size_t np = (na + 1) / 2;
    for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < N; j += (size_t)gridDim.x * blockDim.x) {
        uint64_t v = 0;
        if (j < np) {
            const uint64_t lo = a[2 * j];
            const uint64_t hi = (2 * j + 1 < na) ? a[2 * j + 1] : 0u;
            v = lo | (hi << 32);
        }
        out[j] = piece_to_strict(v, p0);
        out[N + j] = piece_to_strict(v, p1);
        out[2 * N + j] = piece_to_strict(v, p2);
    }
}

// Pieces first .. first + 2^k - 1 of a (zero past its end) -> residues at
// out + q * stride.
__global__ void split3_off_kernel(uint64_t* __restrict__ out, size_t stride, const uint32_t* __restrict__ a,
                                  size_t na, size_t first, size_t N, uint64_t p0, uint64_t p1, uint64_t p2)
{
    for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < N; j += (size_t)gridDim.x * blockDim.x) {
        const size_t wi = 2 * (first + j);
        uint64_t v = 0;
        if (wi < na) {
            v = a[wi];
            if (wi + 1 < na) v |= (uint64_t)a[wi + 1] << 32;
        }
        out[j] = piece_to_strict(v, p0);
        out[stride + j] = piece_to_strict(v, p1);
        out[2 * stride + j] = piece_to_strict(v, p2);
    }
}

// Reference layout, int_to_ntt NTT.cpp:330-341: two 16-bit points per word.
__global__ void split16_kernel(uint64_t* __restrict__ T, size_t N, const uint32_t* __restrict__ A, size_t AL)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        const size_t w = i >> 1;
        uint64_t v = 0;
        if (w < AL) v = (i & 1) ? (A[w] >> 16) : (A[w] & 0xffffu);
        T[i] = v;
    }
}

// ---- coefficient -> word conversion ----------------------------------------
constexpr int kCvtThreads = 256;
constexpr int kCvtLPT = 2;  // 64-bit limbs per thread
constexpr size_t kCvtLPC = (size_t)kCvtThreads * kCvtLPT;
constexpr size_t kCvtWPC = 2 * kCvtLPC;
// The CRT conversion needs three coefficients below its first limb, so a CTA
// of 256 threads computes 512 coefficients (two per thread, no thread a
// third) and owns the 509 limbs they complete.
constexpr size_t kCrtSlots = (size_t)kCvtThreads * kCvtLPT;
constexpr size_t kCrtLPC = kCrtSlots - 3;
constexpr size_t kCrtWPC = 2 * kCrtLPC;

struct Crt3Consts {
    uint64_t p[3];
    uint32_t c[3];      // p = c 2^32 + 1
    ulonglong2 scale[3];  // N^-1 R^depth mod p_q (Shoup pair): undoes the pointwise R^-1 and the unscaled inverse
    ulonglong2 inv01;     // p0^-1 mod p1
    ulonglong2 p0m2;      // p0 mod p2
    ulonglong2 inv012;    // (p0 p1)^-1 mod p2
    uint64_t p0p1_lo, p0p1_hi;
    uint64_t off[3];      // 2^159 mod p_q when every coefficient gets the offset 2^159, else 0
};

// x * w mod p in [0, p) for a Shoup pair w (product primes c 2^32 + 1).
__device__ __forceinline__ uint64_t crt_mul(uint64_t x, const ulonglong2& w, uint64_t p, uint32_t c)
{
    const uint64_t r = shoup_lazy32(x, w.x, w.y, c);
    return r >= p ? r - p : r;
}

// Garner's CRT: x = r0 + p0 (v1 + p1 v2), 0 <= x < p0 p1 p2, as three limbs.
// Inputs may be any 64-bit residue representatives (lazy transforms).  With
// the offset set, x is the coefficient plus 2^159 (signed coefficients of
// magnitude below 2^159 come out nonnegative and exact).
__device__ __forceinline__ void crt3(const Crt3Consts& C, uint64_t y0, uint64_t y1, uint64_t y2, uint64_t& l0,
                                     uint64_t& l1, uint64_t& l2)
{
    const uint64_t r0s = crt_mul(y0, C.scale[0], C.p[0], C.c[0]);
    const uint64_t r1s = crt_mul(y1, C.scale[1], C.p[1], C.c[1]);
    const uint64_t r2o = crt_mul(y2, C.scale[2], C.p[2], C.c[2]);
    const uint64_t r0 = add_mod(r0s, C.off[0], C.p[0]);
    const uint64_t r1 = add_mod(r1s, C.off[1], C.p[1]);
    const uint64_t r2 = add_mod(r2o, C.off[2], C.p[2]);
    const uint64_t r0m1 = r0 >= C.p[1] ? r0 - C.p[1] : r0;
    const uint64_t v1 = crt_mul(sub_mod(r1, r0m1, C.p[1]), C.inv01, C.p[1], C.c[1]);
    const uint64_t r0m2 = r0 >= C.p[2] ? r0 - C.p[2] : r0;
    uint64_t t = sub_mod(r2, r0m2, C.p[2]);
    t = sub_mod(t, crt_mul(v1, C.p0m2, C.p[2], C.c[2]), C.p[2]);
    const uint64_t v2 = crt_mul(t, C.inv012, C.p[2], C.c[2]);
    // p0 * v1 + r0 = v1 + (c0 v1) 2^32 + r0 with two 32 x 32 products
    const uint64_t x = (uint64_t)C.c[0] * (uint32_t)v1, y = (uint64_t)C.c[0] * (uint32_t)(v1 >> 32);
    uint64_t a0 = v1 + (x << 32), a1 = (x >> 32) + y + (a0 < v1);
    a0 += r0;
    a1 += (a0 < r0);
    // (p0 p1) * v2
    const uint64_t b0 = C.p0p1_lo * v2;
    uint64_t b1 = mulhi64(C.p0p1_lo, v2);
    const uint64_t t1 = C.p0p1_hi * v2;
    uint64_t b2 = mulhi64(C.p0p1_hi, v2);
    b1 += t1;
    b2 += (b1 < t1);
    l0 = a0 + b0;
    const uint64_t c0 = l0 < b0;
    uint64_t s1 = a1 + b1;
    uint64_t c1 = s1 < b1;
    s1 += c0;
    c1 += (s1 < c0);
    l1 = s1;
    l2 = b2 + c1;
}

// Shared tail of the limb conversions: limb digits (T = D_i + C_(i-1)) -> words
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

// Three-prime residues y[q * pstride + j] -> words.  Limb i (64 bits)
// collects x_i.l0 + x_(i-1).l1 + x_(i-2).l2 (< 3 * 2^64).  One CTA handles
// limbs [i0, i0 + kCrtLPC) of one product; slot t of xs holds coefficient
// i0 - 3 + t.
__device__ __forceinline__ void crt3_block(const uint64_t* __restrict__ Y, size_t pstride, size_t ncoef,
                                           const Crt3Consts& C, uint32_t* __restrict__ z, size_t zw, int64_t i0,
                                           uint32_t* agg_slot)
{
    __shared__ uint64_t xs[kCrtSlots * 3];
    const int64_t climit = (int64_t)((zw + 1) / 2);  // limbs this product needs
    for (int t = threadIdx.x; t < (int)kCrtSlots; t += blockDim.x) {
        const int64_t j = i0 - 3 + t;
        uint64_t l0 = 0, l1 = 0, l2 = 0;
        if (j >= 0 && (size_t)j < ncoef && j < climit)
            crt3(C, Y[j], Y[pstride + j], Y[2 * pstride + j], l0, l1, l2);
        xs[3 * t] = l0;
        xs[3 * t + 1] = l1;
        xs[3 * t + 2] = l2;
    }
    __syncthreads();
    uint64_t dig[kCvtLPT];
    uint32_t gen[kCvtLPT];
#pragma unroll
    for (int u = 0; u < kCvtLPT; u++) {
        const int l = threadIdx.x * kCvtLPT + u;  // limb i0 + l, xs slot l + 3
        dig[u] = 0;
        gen[u] = 0;
        if (l < (int)kCrtLPC) {
            const int li = l + 3;
            uint64_t slo = xs[3 * li], shi = 0;
            add128(slo, shi, xs[3 * (li - 1) + 1]);
            add128(slo, shi, xs[3 * (li - 2) + 2]);
            uint64_t plo = xs[3 * (li - 1)], phi = 0;
            add128(plo, phi, xs[3 * (li - 2) + 1]);
            add128(plo, phi, xs[3 * (li - 3) + 2]);
            const uint64_t d = slo + phi;
            dig[u] = d;
            gen[u] = d < slo;
        }
    }
    // words past this CTA's limbs belong to the next CTA
    const size_t zend = 2 * ((size_t)i0 + kCrtLPC);
    limbs_to_words(dig, gen, (size_t)i0 + threadIdx.x * kCvtLPT, z, zw < zend ? zw : zend, agg_slot);
}

__global__ void __launch_bounds__(kCvtThreads) crt3_k1(const uint64_t* __restrict__ Y, size_t N, size_t ncoef,
                                                       Crt3Consts C, uint32_t* __restrict__ z, size_t zw,
                                                       uint32_t* agg)
{
    crt3_block(Y, N, ncoef, C, z, zw, (int64_t)blockIdx.x * (int64_t)kCrtLPC, agg + blockIdx.x);
}

// Batched: product i has residues at Y + i * istride (+ q * pstride), zlen[i]
// words out at z + i * zcap; cpp CTAs per product.
__global__ void __launch_bounds__(kCvtThreads) crt3_batch_k1(const uint64_t* __restrict__ Y, size_t istride,
                                                             size_t pstride, size_t ncoef, Crt3Consts C,
                                                             uint32_t* __restrict__ z, uint32_t zcap,
                                                             const uint32_t* __restrict__ zlen, size_t cpp,
                                                             uint32_t* agg)
{
    const size_t prod = blockIdx.x / cpp, lc = blockIdx.x % cpp;
    crt3_block(Y + prod * istride, pstride, ncoef, C, z + prod * (size_t)zcap, zlen[prod],
               (int64_t)lc * (int64_t)kCrtLPC, agg + blockIdx.x);
}

// Coefficients c_j at bit offsets bits * j (8 <= bits <= 16) -> words.  Limb
// i (bits [64i, 64i+64)) collects lo64(c_j << r_j) for the j with
// floor(bits j / 64) == i and hi64(c_j << r_j) for those with i - 1, where
// r_j = bits j mod 64.  A loader supplies c_j (< 2^64).
constexpr int kStageMax = (int)(64 * (kCvtLPC + 2) / 8 + 2);

__device__ __forceinline__ int64_t first_coef(int64_t limb, int bits)
{
    return limb <= 0 ? 0 : (64 * limb + bits - 1) / bits;
}

__device__ __forceinline__ void limb_sum(const uint64_t* cs, int64_t jlo, int64_t limb, int bits, uint64_t& lo,
                                         uint64_t& hi)
{
    lo = 0;
    hi = 0;
    if (limb < 0) return;
    const int64_t a = first_coef(limb - 1, bits), b = first_coef(limb, bits), c = first_coef(limb + 1, bits);
    if (limb >= 1)
        for (int64_t j = a; j < b; j++) {
            const int r = (int)((bits * j) & 63);
            if (r) add128(lo, hi, cs[j - jlo] >> (64 - r));
        }
    for (int64_t j = b; j < c; j++) add128(lo, hi, cs[j - jlo] << ((bits * j) & 63));
}

struct NttCoefLoader {
    const uint64_t* c;
    uint64_t scale, p, pinv;
    __device__ __forceinline__ uint64_t operator()(size_t j, double&) const
    {
        uint64_t v = c[j];
        return scale ? mont_mul(v, scale, p, pinv) : v;
    }
};

struct FftCoefLoader {
    const double2* T;
    double scale;
    __device__ __forceinline__ uint64_t operator()(size_t j, double& emax) const
    {
        const double f = T[j].x * scale;
        const double r = rint(f);
        const double e = fabs(f - r);
        if (e > emax) emax = e;
        return r > 0 ? (uint64_t)r : 0;
    }
};

template <class Loader>
__global__ void __launch_bounds__(kCvtThreads) coefbits_k1(Loader ld, size_t ncoef, int bits,
                                                           uint32_t* __restrict__ z, size_t zw, uint32_t* agg,
                                                           unsigned long long* err_bits)
{
    __shared__ uint64_t cs[kStageMax];
    const int64_t i0 = (int64_t)blockIdx.x * (int64_t)kCvtLPC;
    const int64_t jlo = first_coef(i0 - 2, bits), jhi = first_coef(i0 + (int64_t)kCvtLPC, bits);
    double emax = 0.0;
    for (int64_t t = threadIdx.x; t < jhi - jlo; t += blockDim.x) {
        const int64_t j = jlo + t;
        cs[t] = (j < (int64_t)ncoef) ? ld((size_t)j, emax) : 0;
    }
    if (err_bits) {
#pragma unroll
        for (int off = 16; off; off >>= 1) emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, off));
        if ((threadIdx.x & 31) == 0 && emax > 0.0) atomicMax(err_bits, (unsigned long long)__double_as_longlong(emax));
    }
    __syncthreads();
    uint64_t dig[kCvtLPT];
    uint32_t gen[kCvtLPT];
#pragma unroll
    for (int u = 0; u < kCvtLPT; u++) {
        const int64_t i = i0 + threadIdx.x * kCvtLPT + u;
        uint64_t slo, shi, plo, phi;
        limb_sum(cs, jlo, i, bits, slo, shi);
        limb_sum(cs, jlo, i - 1, bits, plo, phi);
        const uint64_t d = slo + phi;
        dig[u] = d;
        gen[u] = d < slo;
    }
    limbs_to_words(dig, gen, (size_t)i0 + threadIdx.x * kCvtLPT, z, zw, agg + blockIdx.x);
}

// The same for the widths of the reference's layouts (16-bit NTT points, 8-bit
// FFT points): a limb starts exactly 64 / BITS coefficients, so every shift and
// place is a compile-time constant; shared memory is padded for threads that
// read two limbs' coefficients apart.  2^22 16-bit coefficients: 39 us with the
// run-time loops, 12.6 here; 2^19 8-bit ones 21.6 and 9.8 us.
template <int BITS, class Loader>
__global__ void __launch_bounds__(kCvtThreads) coeflimbs_k1(Loader ld, size_t ncoef, uint32_t* __restrict__ z,
                                                            size_t zw, uint32_t* agg, unsigned long long* err_bits)
{
    constexpr int NC = 64 / BITS, N = (int)(kCvtLPC + 2) * NC;
    __shared__ uint64_t cs[crt_slot(N)];
    const int64_t i0 = (int64_t)blockIdx.x * (int64_t)kCvtLPC;
    const int64_t j0 = (i0 - 2) * NC;
    double emax = 0.0;
    for (int t = threadIdx.x; t < N; t += kCvtThreads) {
        const int64_t j = j0 + t;
        cs[crt_slot(t)] = (j >= 0 && j < (int64_t)ncoef) ? ld((size_t)j, emax) : 0;
    }
    if (err_bits) {
#pragma unroll
        for (int off = 16; off; off >>= 1) emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, off));
        if ((threadIdx.x & 31) == 0 && emax > 0.0) atomicMax(err_bits, (unsigned long long)__double_as_longlong(emax));
    }
    __syncthreads();
    // sums of limbs 2 t - 1, 2 t, 2 t + 1 (limb l's coefficients at slot (l + 2) NC)
    uint64_t lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
    const int b = (int)threadIdx.x * kCvtLPT * NC;
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
        for (int t = 0; t < NC; t++) {
            const uint64_t c = cs[crt_slot(b + u * NC + t)];
            if (u > 0) add128(lo[u - 1], hi[u - 1], c << (BITS * t));
            if (u < 3 && t > 0) add128(lo[u], hi[u], c >> (64 - BITS * t));
        }
    uint64_t dig[kCvtLPT];
    uint32_t gen[kCvtLPT];
#pragma unroll
    for (int u = 0; u < kCvtLPT; u++) {
        const uint64_t d = lo[u + 1] + hi[u];
        dig[u] = d;
        gen[u] = d < lo[u + 1];
    }
    limbs_to_words(dig, gen, (size_t)i0 + threadIdx.x * kCvtLPT, z, zw, agg + blockIdx.x);
}

// Carries between the CTAs of a coefficient-bits conversion (kCvtLPC limbs
// per CTA; the CRT conversions own kCrtLPC and ripple with kCrtWPC).
static void finish_scan(uint32_t* z, size_t zw, uint32_t* agg, size_t nctas, cudaStream_t s)
{
    carry_fix(z, zw, kCvtWPC, agg, nctas, s);
}

void coef16_to_words(const uint64_t* c, size_t ncoef, uint64_t scale_mont, uint64_t p, uint64_t pinv_neg,
                     uint32_t* z, size_t zw, cudaStream_t s)
{
    if (zw == 0) return;
    const size_t nlimbs = (zw + 1) / 2;
    const size_t nctas = (nlimbs + kCvtLPC - 1) / kCvtLPC;
    DevBuf<uint32_t> agg(carry_agg_words(1, nctas), s);
    ProfScope ps(KC_CRT, 8.0 * (double)ncoef + 4.0 * (double)zw, s);
    coeflimbs_k1<16, NttCoefLoader><<<(unsigned)nctas, kCvtThreads, 0, s>>>(
        NttCoefLoader{c, scale_mont, p, pinv_neg}, ncoef, z, zw, agg.get(), nullptr);
    PIC_CHECK_LAUNCH();
    count_launch();
    finish_scan(z, zw, agg.get(), nctas, s);
}

double fft_coef_to_words(const double2* T, size_t ncoef, double scale, int bits, uint32_t* z, size_t zw,
                         cudaStream_t s)
{
    PIC_REQUIRE(bits >= 8 && bits <= 16, PIC_ERR_INVALID, "FFT piece width out of range");
    if (zw == 0) return 0.0;
    const size_t nlimbs = (zw + 1) / 2;
    const size_t nctas = (nlimbs + kCvtLPC - 1) / kCvtLPC;
    DevBuf<uint32_t> agg(carry_agg_words(1, nctas), s);
    DevBuf<unsigned long long> err(1, s);
    PIC_CUDA(cudaMemsetAsync(err.get(), 0, sizeof(unsigned long long), s));
    ProfScope ps(KC_CRT, 16.0 * (double)ncoef + 4.0 * (double)zw, s);
    if (bits == 8)
        coeflimbs_k1<8, FftCoefLoader><<<(unsigned)nctas, kCvtThreads, 0, s>>>(FftCoefLoader{T, scale}, ncoef, z, zw,
                                                                              agg.get(), err.get());
    else
        coefbits_k1<FftCoefLoader><<<(unsigned)nctas, kCvtThreads, 0, s>>>(FftCoefLoader{T, scale}, ncoef, bits, z,
                                                                          zw, agg.get(), err.get());
    PIC_CHECK_LAUNCH();
    count_launch();
    finish_scan(z, zw, agg.get(), nctas, s);
    unsigned long long eb = 0;
    read_words((uint32_t*)&eb, (const uint32_t*)err.get(), 2, s);
    double e;
    memcpy(&e, &eb, sizeof e);
    return e;
}

// Scale folded into the CRT: multiplying by R^depth N^-1 undoes `depth`
// pointwise Montgomery products (each contributes R^-1) and the unscaled
// inverse (N).  Every constant is a Shoup pair (value, companion).
static Crt3Consts make_crt3(int k, int depth)
{
    Crt3Consts C;
    const uint64_t N = (uint64_t)1 << k;
    auto pair = [](uint64_t w, uint64_t p) { return make_ulonglong2(w, shoup_companion(w, p)); };
    for (int q = 0; q < 3; q++) {
        const uint64_t p = kProductPrimes[q];
        C.p[q] = p;
        C.c[q] = (uint32_t)(p >> 32);
        uint64_t sc = host_powmod(N % p, p - 2, p);
        for (int d = 0; d < depth; d++) sc = to_mont(sc, p);
        C.scale[q] = pair(sc, p);  // y * N^-1 R^depth
    }
    const uint64_t p0 = C.p[0], p1 = C.p[1], p2 = C.p[2];
    C.inv01 = pair(host_powmod(p0 % p1, p1 - 2, p1), p1);
    C.p0m2 = pair(p0 % p2, p2);
    const uint64_t p01m2 = host_mulmod(p0 % p2, p1 % p2, p2);
    C.inv012 = pair(host_powmod(p01m2, p2 - 2, p2), p2);
    const unsigned __int128 p01 = (unsigned __int128)p0 * p1;
    C.p0p1_lo = (uint64_t)p01;
    C.p0p1_hi = (uint64_t)(p01 >> 64);
    for (int q = 0; q < 3; q++) C.off[q] = 0;
    return C;
}

static NttBatch ntt3_batch(uint64_t* data, int k)
{
    NttBatch bat;
    bat.data = data;
    bat.stride = (size_t)1 << k;
    bat.count = 3;
    bat.per_prime = 1;
    for (int q = 0; q < 3; q++) bat.prime[q] = prime_tables(kProductPrimes[q]).dev;
    return bat;
}

void ntt3_forward_operand(uint64_t* out, int k, const uint32_t* a, size_t na, cudaStream_t s)
{
    const size_t N = (size_t)1 << k;
    {
        ProfScope ps(KC_SPLIT, 4.0 * (double)na + 24.0 * (double)N, s);
        split3_kernel<<<grid_for(N, 256), 256, 0, s>>>(out, a, na, N, kProductPrimes[0], kProductPrimes[1],
                                                       kProductPrimes[2]);
        PIC_CHECK_LAUNCH();
        count_launch();
    }
    ntt_forward_dif(ntt3_batch(out, k), k, s);
}

void ntt3_pointwise(uint64_t* a, const uint64_t* b, int k, cudaStream_t s)
{
    ntt_pointwise_mont(ntt3_batch(a, k), b, k, s);
}

void ntt3_inverse_to_words(uint64_t* y, int k, size_t ncoef, int depth, uint32_t* z, size_t zw, cudaStream_t s)
{
    ntt_inverse_dit(ntt3_batch(y, k), k, s);
    const Crt3Consts C = make_crt3(k, depth);
    const size_t nlimbs = (zw + 1) / 2;
    const size_t nctas = (nlimbs + kCrtLPC - 1) / kCrtLPC;
    DevBuf<uint32_t> agg(carry_agg_words(1, nctas), s);
    ProfScope ps(KC_CRT, 24.0 * (double)ncoef + 4.0 * (double)zw, s);
    crt3_k1<<<(unsigned)nctas, kCvtThreads, 0, s>>>(y, (size_t)1 << k, ncoef, C, z, zw, agg.get());
    PIC_CHECK_LAUNCH();
    count_launch();
    carry_fix(z, zw, kCrtWPC, agg.get(), nctas, s);
}

void ntt3_batch_to_words(const uint64_t* y, size_t istride, size_t pstride, size_t count, int k, uint32_t* z,
                         uint32_t zcap, const uint32_t* zlen, cudaStream_t s, size_t ncoef, bool offset)
{
    if (count == 0) return;
    if (ncoef == 0) ncoef = (size_t)1 << k;
    Crt3Consts C = make_crt3(k, 1);
    if (offset)
        for (int q = 0; q < 3; q++) C.off[q] = host_powmod(2, 159, C.p[q]);
    const size_t cpp = (((size_t)zcap + 1) / 2 + kCrtLPC - 1) / kCrtLPC;
    const size_t nctas = count * cpp;
    DevBuf<uint32_t> agg(carry_agg_words(count, cpp), s);
    {
        ProfScope ps(KC_CRT, (24.0 * (double)ncoef + 4.0 * zcap) * (double)count, s);
        crt3_batch_k1<<<(unsigned)nctas, kCvtThreads, 0, s>>>(y, istride, pstride, ncoef, C, z, zcap, zlen,
                                                              cpp, agg.get());
        PIC_CHECK_LAUNCH();
        count_launch();
    }
    carry_fix_batch(z, zcap, zlen, kCrtWPC, agg.get(), count, cpp, s);
}

// Pieces used by the allocation-free product (noalloc.cu): the same split and
// CRT + carry kernels, with every buffer supplied by the caller.
void split3_into(uint64_t* out, int k, const uint32_t* a, size_t na, const uint64_t primes[3], cudaStream_t s)
{
    const size_t N = (size_t)1 << k;
    split3_kernel<<<grid_for(N, 256), 256, 0, s>>>(out, a, na, N, primes[0], primes[1], primes[2]);
    PIC_CHECK_LAUNCH();
    count_launch();
}

size_t crt3_scratch_ctas(size_t zw) { return ((zw + 1) / 2 + kCrtLPC - 1) / kCrtLPC; }

void crt3_to_words_scratch(const uint64_t* y, int k, size_t ncoef, uint32_t* z, size_t zw, uint32_t* agg,
                           cudaStream_t s)
{
    const Crt3Consts C = make_crt3(k, 1);
    const size_t nctas = crt3_scratch_ctas(zw);
    PIC_REQUIRE(carry_groups(nctas) == 0, PIC_ERR_LENGTH, "product too long for the scratch form");
    crt3_k1<<<(unsigned)nctas, kCvtThreads, 0, s>>>(y, (size_t)1 << k, ncoef, C, z, zw, agg);
    PIC_CHECK_LAUNCH();
    count_launch();
    carry_fix(z, zw, kCrtWPC, agg, nctas, s);
}

// Wrapped products.  A product of operands of sa and sb pieces has
// L = sa + sb - 1 coefficients c_0..c_(L-1).  When L exceeds the main
// transform length Nm (but sa, sb <= Nm), the cyclic product of length Nm
// holds c_j + c_(Nm+j) for j < W = L - Nm.  The W top coefficients depend only
// on the top W pieces of each operand (a from index Nm - sb + 1, b from
// Nm - sa + 1): the product of those pieces, d, gives c_(Nm+j) = d_(W-1+j),
// and its cyclic length T >= 2W - 1 keeps those indices free of wrap.  For
// each of the W positions:
//   y[j] <- y[j] - h (kept nonnegative by adding p), y[Nm + j] <- h
// (inverse outputs arrive in [0, 8p) and are first brought below 4p),
// with h = d_(W-1+j) * Nm / T so that both halves carry the same scale Nm.
// y items have stride ystride >= Nm + W; tail items have stride T.  `item`
// selects which children hold products (all for P, the even ones for Q, R).
__global__ void wrap_fix_kernel(uint64_t* __restrict__ y, size_t ystride, const uint64_t* __restrict__ tail,
                                size_t T, size_t nitems, size_t item_mul, size_t nchild, size_t Nm, size_t W,
                                Mod64 m0, Mod64 m1, Mod64 m2, uint64_t c0, uint64_t c1, uint64_t c2)
{
    const size_t total = 3 * nitems * W;
    for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < total; g += (size_t)gridDim.x * blockDim.x) {
        const size_t q = g / (nitems * W);
        const size_t r = g - q * nitems * W;
        const size_t it = r / W, j = r - it * W;
        const Mod64& M = q == 0 ? m0 : (q == 1 ? m1 : m2);
        const uint64_t cT = q == 0 ? c0 : (q == 1 ? c1 : c2);
        const size_t child = q * nchild + it * item_mul;
        const uint64_t h = mont_mul(tail[child * T + W - 1 + j], cT, M);  // < p
        uint64_t* yi = y + child * ystride;
        const uint64_t p4 = 4 * M.p;
        uint64_t v = yi[j];  // lazy inverse output, < 8p
        v = v >= p4 ? v - p4 : v;
        yi[j] = v + M.p - h;  // < 5p < 2^64: the CRT reduces any 64-bit input
        yi[Nm + j] = h;
    }
}

void launch_wrap_fix(uint64_t* y, size_t ystride, const uint64_t* tail, size_t T, size_t nitems, size_t item_mul,
                     size_t nchild, size_t Nm, size_t W, const uint64_t cT[3], cudaStream_t s)
{
    const Mod64 m0 = make_mod(kProductPrimes[0]), m1 = make_mod(kProductPrimes[1]), m2 = make_mod(kProductPrimes[2]);
    wrap_fix_kernel<<<grid_for(3 * nitems * W, 256), 256, 0, s>>>(y, ystride, tail, T, nitems, item_mul, nchild, Nm,
                                                                W, m0, m1, m2, cT[0], cT[1], cT[2]);
    PIC_CHECK_LAUNCH();
}

// ---- products ----------------------------------------------------------------
static bool g_mul_wrap = true;
void mul_set_wrap(bool on) { g_mul_wrap = on; }
bool mul_wrap() { return g_mul_wrap; }

static NttBatch ntt3_batch_stride(uint64_t* data, size_t stride)
{
    NttBatch bat;
    bat.data = data;
    bat.stride = stride;
    bat.count = 3;
    bat.per_prime = 1;
    for (int q = 0; q < 3; q++) bat.prime[q] = prime_tables(kProductPrimes[q]).dev;
    return bat;
}

// ---- a held forward transform (transform reuse in the Newton steps) ----------
// While an OperandHold for (src, n) is alive on this thread, three-prime
// products that take that operand reuse its forward transform at main length
// 2^k instead of transforming it again: the first such product computes it
// (split + forward, stride 2^k) and keeps it, later ones read it.  The plain
// product at 2^k and the main part of a wrapped product at Nm = 2^k split the
// operand the same way (pieces 0 .. 2^k - 1, zero above), so one transform
// serves both.  Only the operand's words, length and k decide a match.
namespace {
struct HeldOperand {
    const uint32_t* src = nullptr;
    size_t n = 0;
    int k = -1;
    int form = kFormInt;
    DevBuf<uint64_t> T;  // 3 x 2^k residues, transforms 2^k apart, bit-reversed order
};
thread_local HeldOperand* t_held = nullptr;
std::atomic<uint64_t> g_held_reuses{0};
}  // namespace

OperandHold::OperandHold(const uint32_t* src, size_t n) : prev_(t_held)
{
    auto* h = new HeldOperand;
    h->src = src;
    h->n = n;
    held_ = h;
    t_held = h;
}

OperandHold::~OperandHold()
{
    t_held = static_cast<HeldOperand*>(prev_);
    delete static_cast<HeldOperand*>(held_);
}

uint64_t held_transform_reuses() { return g_held_reuses.load(); }

static bool is_held(const uint32_t* x, size_t n) { return t_held && t_held->src == x && t_held->n == n; }

// The integer form: the held operand's forward transform at length 2^k (stride
// 2^k), computed on first use at that length.
static const uint64_t* held_transform(int k, cudaStream_t s)
{
    HeldOperand* h = t_held;
    if (h->k != k || h->form != kFormInt) {
        h->T = DevBuf<uint64_t>(3 * ((size_t)1 << k), s);
        ntt3_forward_operand(h->T.get(), k, h->src, h->n, s);
        h->k = k;
        h->form = kFormInt;
    } else {
        g_held_reuses.fetch_add(1);
    }
    return h->T.get();
}

// The FP64 form: the held operand's spectrum at length 2^k (stride 2^k); *ready
// tells whether an earlier product has filled it, else this one must.
static uint64_t* held_spectrum(int k, bool* ready, cudaStream_t s)
{
    HeldOperand* h = t_held;
    *ready = h->k == k && h->form == kFormDbl;
    if (!*ready) {
        h->T = DevBuf<uint64_t>(3 * ((size_t)1 << k), s);
        h->k = k;
        h->form = kFormDbl;
    } else {
        g_held_reuses.fetch_add(1);
    }
    return h->T.get();
}

// Copies three transforms of 2^k residues from stride `from` to stride `to`.
static void copy_transforms(uint64_t* dst, size_t to, const uint64_t* src, size_t from, int k, cudaStream_t s)
{
    PIC_CUDA(cudaMemcpy2DAsync(dst, to * sizeof(uint64_t), src, from * sizeof(uint64_t),
                               sizeof(uint64_t) << k, 3, cudaMemcpyDeviceToDevice, s));
}

// The wrapped form of mul_ntt3 (see wrap_fix_kernel): main transforms of
// length Nm = 2^km, tails of length 2^kt over the top W pieces.
static void mul_ntt3_wrapped(uint32_t* z, const uint32_t* a, size_t na, const uint32_t* b, size_t nb, int km,
                             int kt, cudaStream_t s)
{
    const size_t zw = na + nb;
    const size_t pa = (na + 1) / 2, pb = (nb + 1) / 2;
    const size_t L = pa + pb - 1;
    const size_t Nm = (size_t)1 << km, T = (size_t)1 << kt, W = L - Nm;
    const size_t ST = Nm + ((W + 15) & ~(size_t)15);
    const bool square = (a == b && na == nb);
    const uint64_t P0 = kProductPrimes[0], P1 = kProductPrimes[1], P2 = kProductPrimes[2];
    // a held b (or a held square) brings its main transform with it
    const uint64_t* held = is_held(b, nb) ? held_transform(km, s) : nullptr;
    DevBuf<uint64_t> A(3 * ST, s), B(square || held ? 0 : 3 * ST, s), tA(3 * T, s), tB(square ? 0 : 3 * T, s);
    {
        ProfScope ps(KC_SPLIT, 4.0 * (double)(na + nb) + 24.0 * (double)(2 * (Nm + T)), s);
        if (!(held && square))
            split3_off_kernel<<<grid_for(Nm, 256), 256, 0, s>>>(A.get(), ST, a, na, 0, Nm, P0, P1, P2);
        split3_off_kernel<<<grid_for(T, 256), 256, 0, s>>>(tA.get(), T, a, na, Nm - pb + 1, T, P0, P1, P2);
        if (!square) {
            if (!held)
                split3_off_kernel<<<grid_for(Nm, 256), 256, 0, s>>>(B.get(), ST, b, nb, 0, Nm, P0, P1, P2);
            split3_off_kernel<<<grid_for(T, 256), 256, 0, s>>>(tB.get(), T, b, nb, Nm - pa + 1, T, P0, P1, P2);
        }
        PIC_CHECK_LAUNCH();
        count_launch((held && square ? 0 : 1) + 1 + (square ? 0 : (held ? 1 : 2)));
    }
    const NttBatch mA = ntt3_batch_stride(A.get(), ST), mB = ntt3_batch_stride(B.get(), ST);
    const NttBatch xA = ntt3_batch_stride(tA.get(), T), xB = ntt3_batch_stride(tB.get(), T);
    if (held && square) copy_transforms(A.get(), ST, held, Nm, km, s);
    else ntt_forward_dif(mA, km, s);
    ntt_forward_dif(xA, kt, s);
    if (!square) {
        if (!held) ntt_forward_dif(mB, km, s);
        ntt_forward_dif(xB, kt, s);
    }
    if (held) ntt_pointwise_mont(mA, held, km, s, Nm);
    else ntt_pointwise_mont(mA, square ? A.get() : B.get(), km, s);
    ntt_pointwise_mont(xA, square ? tA.get() : tB.get(), kt, s);
    ntt_inverse_dit(mA, km, s);
    ntt_inverse_dit(xA, kt, s);
    uint64_t cT[3];
    for (int q = 0; q < 3; q++) cT[q] = to_mont((uint64_t)(Nm / T), kProductPrimes[q]);
    {
        ProfScope ps(KC_NTT_POINTWISE, 3.0 * (double)W * 24.0, s);
        launch_wrap_fix(A.get(), ST, tA.get(), T, 1, 1, 1, Nm, W, cT, s);
        count_launch();
    }
    const Crt3Consts C = make_crt3(km, 1);
    const size_t nctas = crt3_scratch_ctas(zw);
    DevBuf<uint32_t> agg(carry_agg_words(1, nctas), s);
    ProfScope ps(KC_CRT, 24.0 * (double)L + 4.0 * (double)zw, s);
    crt3_k1<<<(unsigned)nctas, kCvtThreads, 0, s>>>(A.get(), ST, L, C, z, zw, agg.get());
    PIC_CHECK_LAUNCH();
    count_launch();
    carry_fix(z, zw, kCrtWPC, agg.get(), nctas, s);
}

void mul_ntt3(uint32_t* z, const uint32_t* a, size_t na, const uint32_t* b, size_t nb, cudaStream_t s)
{
    if (is_held(a, na) && !(a == b && na == nb)) {  // the held operand goes second
        std::swap(a, b);
        std::swap(na, nb);
    }
    const size_t zw = na + nb;
    const size_t pa = (na + 1) / 2, pb = (nb + 1) / 2;
    const size_t ncoef = pa + pb - 1;
    int k = ceil_log2(ncoef);
    if (k < 1) k = 1;
    PIC_REQUIRE(k <= 30, PIC_ERR_LENGTH, "product too long for the three-prime NTT (2^30 points)");
    const size_t N = (size_t)1 << k;
    if (g_mul_wrap && k >= 4) {
        // wrapped when the product just exceeds a power of two and the tail is short
        const size_t Nm = N / 2;
        if (std::max(pa, pb) <= Nm && ncoef > Nm) {
            const size_t W = ncoef - Nm;
            int kt = ceil_log2(2 * W - 1);
            if (kt < 2) kt = 2;
            if (((size_t)1 << kt) <= Nm / 2) {
                mul_ntt3_wrapped(z, a, na, b, nb, k - 1, kt, s);
                return;
            }
        }
    }
    const bool square = (a == b && na == nb);
    const uint64_t* held = is_held(b, nb) ? held_transform(k, s) : nullptr;
    DevBuf<uint64_t> A(3 * N, s);
    DevBuf<uint64_t> B(square || held ? 0 : 3 * N, s);
    if (held && square) copy_transforms(A.get(), N, held, N, k, s);
    else ntt3_forward_operand(A.get(), k, a, na, s);
    if (!square && !held) ntt3_forward_operand(B.get(), k, b, nb, s);
    ntt3_pointwise(A.get(), held ? held : (square ? A.get() : B.get()), k, s);
    ntt3_inverse_to_words(A.get(), k, ncoef, 1, z, zw, s);
}

// ---- the FP64 three-prime form ---------------------------------------------
// Operands in 56-bit pieces (piece j = bits 56 j .. 56 j + 55), residues
// modulo kDblPrimes held as doubles (fp64mod.cuh), the same transform passes
// with FP64 butterflies, pointwise products without a Montgomery factor, and a
// CRT that places coefficient j (below p0 p1 p2 < 2^141) at bit 56 j.  Inverse
// outputs arrive with |y| <= 15 p (unscaled), 15.75 p with a wrapped tail taken
// out of them, below 2^51.

size_t pieces56(size_t nwords) { return (32 * nwords + 55) / 56; }

static NttBatch ntt3d_batch_stride(uint64_t* data, size_t stride)
{
    NttBatch bat;
    bat.data = data;
    bat.stride = stride;
    bat.count = 3;
    bat.per_prime = 1;
    for (int q = 0; q < 3; q++) bat.prime[q] = dbl_prime_tables(kDblPrimes[q]).dev;
    return bat;
}

static void dbl_pair(uint64_t w, uint64_t p, double& d, double& dp)
{
    d = (double)w;
    dp = d / (double)p;
}

CrtDConsts make_crtd(int k, bool offset)
{
    CrtDConsts C;
    const uint64_t P0 = kDblPrimes[0], P1 = kDblPrimes[1], P2 = kDblPrimes[2];
    for (int q = 0; q < 3; q++) {
        const uint64_t p = kDblPrimes[q];
        C.p[q] = (double)p;
        C.pinv[q] = 1.0 / C.p[q];
        dbl_pair(host_powmod(((uint64_t)1 << k) % p, p - 2, p), p, C.sw[q], C.swp[q]);
        C.off[q] = offset ? (double)host_powmod(2, 140, p) : 0.0;
    }
    dbl_pair(host_powmod(P0 % P1, P1 - 2, P1), P1, C.i01, C.i01p);
    dbl_pair(host_powmod(host_mulmod(P0 % P2, P1 % P2, P2), P2 - 2, P2), P2, C.i012, C.i012p);
    dbl_pair(host_powmod(P1 % P2, P2 - 2, P2), P2, C.q012, C.q012p);
    C.off[0] -= 2 * C.p[0];
    const uint64_t c0 = P0 >> 32, c1 = P1 >> 32;
    C.c0 = (uint32_t)c0;
    C.c01 = (uint32_t)(c0 + c1);
    C.cc = (uint32_t)(c0 * c1);
    return C;
}

// 128 threads convert 127 groups of 8 coefficients and the three before them
// (1019 coefficients, eight per thread), eight CTAs per SM.  Bound by instruction
// issue (about 150 a coefficient, 57 of them FP64).  2^24-word operands: 255 us
// with three-limb coefficients of one thread each, 234 with the coefficients
// spread over the threads, 207 with base-2^56 digits and the short products of
// c 2^32 + 1, 152 with the next residues loaded ahead and the words written
// through shared memory.
constexpr int kCrtDThreads = 128;
constexpr int kCrtDGroups = 127;
constexpr size_t kCrtDWPC = 14 * (size_t)kCrtDGroups;  // words per CTA
constexpr int kCrtDCoefs = 8 * kCrtDGroups + 3;
constexpr int kCrtDSlots = crt_slot(kCrtDCoefs);

// Coefficients with words below zw.
__device__ __forceinline__ int64_t crt_limit(size_t ncoef, size_t zw)
{
    const int64_t climit = (int64_t)((32 * zw + 55) / 56);
    return climit < (int64_t)ncoef ? climit : (int64_t)ncoef;
}

CrtWrap crt_wrap(const uint64_t* tail, size_t istride, size_t pstride, size_t T, size_t N, size_t W)
{
    CrtWrap w{tail, istride, pstride, (int64_t)N, (int64_t)W, (double)(N / T), {}};  // N / T: below every prime
    for (int q = 0; q < 3; q++) w.cwp[q] = w.cw / (double)kDblPrimes[q];
    return w;
}

// Residues of coefficient j of one product.  Wrapped: from N on they are the
// tail's h(j - N) = d_(W - 1 + j - N) N / T, and the first W have h(j) taken out.
// Three kernels of their own that rewrote those residues took 34 ms of a
// computation of 1e9 digits, at the bandwidth of the memory; here it is one more
// read of the tail (1.217 -> 1.195 s for the whole).
template <bool WRAP>
struct CrtSource {
    const uint64_t *Y, *D;  // the product's residues, its tail's from W - 1 on
    size_t pstride;

    __device__ __forceinline__ void load(const CrtWrap& w, int64_t j, double& y0, double& y1, double& y2) const
    {
        const bool tail = WRAP && j >= w.N;
        const uint64_t* p = tail ? D + (j - w.N) : Y + j;
        const size_t st = tail ? w.pstride : pstride;
        y0 = dbits(p[0]);
        y1 = dbits(p[st]);
        y2 = dbits(p[2 * st]);
    }
    __device__ __forceinline__ void fix(const CrtWrap& w, const CrtDConsts& C, int64_t j, double& y0, double& y1,
                                        double& y2) const
    {
        if constexpr (WRAP) {
            if (j >= w.N) {
                y0 = dmul_tw(y0, w.cw, w.cwp[0], C.p[0]);
                y1 = dmul_tw(y1, w.cw, w.cwp[1], C.p[1]);
                y2 = dmul_tw(y2, w.cw, w.cwp[2], C.p[2]);
            } else if (j < w.W) {
                y0 = __dadd_rn(y0, -dmul_tw(dbits(D[j]), w.cw, w.cwp[0], C.p[0]));
                y1 = __dadd_rn(y1, -dmul_tw(dbits(D[w.pstride + j]), w.cw, w.cwp[1], C.p[1]));
                y2 = __dadd_rn(y2, -dmul_tw(dbits(D[2 * w.pstride + j]), w.cw, w.cwp[2], C.p[2]));
            }
        }
    }
};

template <bool WRAP>
__device__ __forceinline__ void crt3d_block(const CrtSource<WRAP>& S, const CrtWrap& wrap, size_t ncoef,
                                            const CrtDConsts& C, uint32_t* __restrict__ z, size_t zw, int64_t cta,
                                            uint32_t* agg_slot)
{
    __shared__ CrtDigits<kCrtDSlots> X;
    const int64_t j0 = 8 * cta * kCrtDGroups - 3, jlim = crt_limit(ncoef, zw);
    crt_coefs(X, kCrtDCoefs, C, [&](int i) { return j0 + i < jlim ? j0 + i : (int64_t)-1; },
              [&](int64_t j, double& y0, double& y1, double& y2) { S.load(wrap, j, y0, y1, y2); },
              [&](int64_t j, double& y0, double& y1, double& y2) { S.fix(wrap, C, j, y0, y1, y2); });
    __syncthreads();
    uint64_t t[8];
    const bool mine = threadIdx.x < kCrtDGroups;
    if (mine) crt_group(X, 8 * (int)threadIdx.x + 3, t);
    uint32_t* W = reinterpret_cast<uint32_t*>(&X);
    digits_to_words(t, mine, false, W, agg_slot);
    const size_t w0 = (size_t)cta * kCrtDWPC;
    const int n = w0 >= zw ? 0 : (int)(zw - w0 < kCrtDWPC ? zw - w0 : kCrtDWPC);
    for (int i = threadIdx.x; i < n; i += kCrtDThreads) z[w0 + i] = W[i];
}

// A single CTA posts the top word; several leave their carries to carry_fix.
template <bool WRAP>
__global__ void __launch_bounds__(kCrtDThreads, 8) crt3d_k1(const uint64_t* __restrict__ Y, size_t pstride,
                                                            size_t ncoef, const __grid_constant__ CrtDConsts C,
                                                            const __grid_constant__ CrtWrap wrap, uint32_t* z,
                                                            size_t zw, uint32_t* agg, MailRef mail)
{
    const CrtSource<WRAP> S{Y, WRAP ? wrap.tail + wrap.W - 1 : nullptr, pstride};
    crt3d_block(S, wrap, ncoef, C, z, zw, (int64_t)blockIdx.x, agg + blockIdx.x);
    if (mail.slot == nullptr) return;
    __syncthreads();
    if (threadIdx.x == 0) mail_post(mail, z[zw - 1]);
}

template <bool WRAP>
__global__ void __launch_bounds__(kCrtDThreads, 8) crt3d_batch_k1(const uint64_t* __restrict__ Y, size_t istride,
                                                                  size_t pstride, size_t ncoef,
                                                                  const __grid_constant__ CrtDConsts C,
                                                                  const __grid_constant__ CrtWrap wrap,
                                                                  uint32_t* __restrict__ z, uint32_t zcap,
                                                                  const uint32_t* __restrict__ zlen, size_t cpp,
                                                                  uint32_t* agg)
{
    const size_t prod = blockIdx.x / cpp, lc = blockIdx.x % cpp;
    const CrtSource<WRAP> S{Y + prod * istride, WRAP ? wrap.tail + prod * wrap.istride + wrap.W - 1 : nullptr, pstride};
    crt3d_block(S, wrap, ncoef, C, z + prod * (size_t)zcap, zlen[prod], (int64_t)lc,
                agg + blockIdx.x);
}

// Short products: `per` groups each, `pack` products per CTA (at most 128 groups
// and kCrtDCoefs coefficients), where one product would leave most of a CTA idle.
template <bool WRAP>
__global__ void __launch_bounds__(kCrtDThreads, 8) crt3d_pack_k1(const uint64_t* __restrict__ Y, size_t istride,
                                                                 size_t pstride, size_t ncoef,
                                                                 const __grid_constant__ CrtDConsts C,
                                                                 const __grid_constant__ CrtWrap wrap,
                                                                 uint32_t* __restrict__ z, uint32_t zcap,
                                                                 const uint32_t* __restrict__ zlen, size_t count,
                                                                 int per, int pack)
{
    __shared__ CrtDigits<kCrtDSlots> X;
    __shared__ uint32_t s_agg;
    const int stride = 8 * per + 3;  // a product's coefficients, three zeros first
    const size_t p0 = (size_t)blockIdx.x * pack;
    const int n = (int)(count - p0 < (size_t)pack ? count - p0 : (size_t)pack);
    auto source = [&](int64_t at) {
        const size_t prod = p0 + (size_t)(at >> 32);
        return CrtSource<WRAP>{Y + prod * istride, WRAP ? wrap.tail + prod * wrap.istride + wrap.W - 1 : nullptr, pstride};
    };
    crt_coefs(X, n * stride, C,
              [&](int i) {
                  const int q = i / stride, j = i - q * stride - 3;
                  return j >= 0 && j < crt_limit(ncoef, zlen[p0 + q]) ? ((int64_t)q << 32) + j : (int64_t)-1;
              },
              [&](int64_t at, double& y0, double& y1, double& y2) {
                  source(at).load(wrap, (int64_t)(uint32_t)at, y0, y1, y2);
              },
              [&](int64_t at, double& y0, double& y1, double& y2) {
                  if constexpr (WRAP) source(at).fix(wrap, C, (int64_t)(uint32_t)at, y0, y1, y2);
              });
    __syncthreads();
    uint64_t t[8];
    const int q = (int)threadIdx.x / per, g = (int)threadIdx.x - q * per;
    const bool mine = q < n;
    if (mine) crt_group(X, q * stride + 8 * g + 3, t);
    uint32_t* W = reinterpret_cast<uint32_t*>(&X);
    digits_to_words(t, mine, g == per - 1, W, &s_agg);
    const int words = 14 * per;
    for (int i = threadIdx.x; i < n * words; i += kCrtDThreads) {
        const int r = i / words, w = i - r * words;
        if ((uint32_t)w < zlen[p0 + r]) z[(p0 + r) * (size_t)zcap + w] = W[i];
    }
}

static size_t crt3d_ctas(size_t zw) { return (zw + kCrtDWPC - 1) / kCrtDWPC; }

// Inverse-transformed residues (product length 2^k, prime q at y + q pstride)
// -> zw words; mail receives the top one.
static void crt3d_to_words(const uint64_t* y, size_t pstride, int k, size_t ncoef, const CrtWrap& wrap, uint32_t* z,
                           size_t zw, Mail* mail, cudaStream_t s)
{
    const CrtDConsts C = make_crtd(k, false);
    const size_t nctas = crt3d_ctas(zw);
    DevBuf<uint32_t> agg(carry_agg_words(1, nctas), s);
    const MailRef m = mail ? mail->ref() : MailRef{};
    ProfScope ps(KC_CRT, 24.0 * (double)ncoef + 4.0 * (double)zw, s);
    auto kern = wrap.tail ? crt3d_k1<true> : crt3d_k1<false>;
    kern<<<(unsigned)nctas, kCrtDThreads, 0, s>>>(y, pstride, ncoef, C, wrap, z, zw, agg.get(),
                                                 nctas == 1 ? m : MailRef{});
    PIC_CHECK_LAUNCH();
    count_launch();
    if (nctas > 1) carry_fix(z, zw, kCrtDWPC, agg.get(), nctas, s, m);
}

void ntt3d_batch_to_words(const uint64_t* y, size_t istride, size_t pstride, size_t count, int k, uint32_t* z,
                          uint32_t zcap, const uint32_t* zlen, cudaStream_t s, size_t ncoef, bool offset,
                          const CrtWrap& wrap)
{
    if (count == 0) return;
    if (ncoef == 0) ncoef = (size_t)1 << k;
    const CrtDConsts C = make_crtd(k, offset);
    // products of at most half a CTA's groups share CTAs
    const int per = (int)((zcap + 13) / 14);
    const int pack = std::min(kCrtDThreads / std::max(per, 1), kCrtDCoefs / (8 * per + 3));
    if (per >= 1 && pack >= 2) {
        ProfScope ps(KC_CRT, (24.0 * (double)ncoef + 4.0 * zcap) * (double)count, s);
        auto kern = wrap.tail ? crt3d_pack_k1<true> : crt3d_pack_k1<false>;
        kern<<<(unsigned)((count + pack - 1) / pack), kCrtDThreads, 0, s>>>(y, istride, pstride, ncoef, C, wrap, z, zcap,
                                                                            zlen, count, per, pack);
        PIC_CHECK_LAUNCH();
        count_launch();
        return;
    }
    const size_t cpp = crt3d_ctas(zcap);
    const size_t nctas = count * cpp;
    DevBuf<uint32_t> agg(carry_agg_words(count, cpp), s);
    {
        ProfScope ps(KC_CRT, (24.0 * (double)ncoef + 4.0 * zcap) * (double)count, s);
        auto kern = wrap.tail ? crt3d_batch_k1<true> : crt3d_batch_k1<false>;
        kern<<<(unsigned)nctas, kCrtDThreads, 0, s>>>(y, istride, pstride, ncoef, C, wrap, z, zcap, zlen, cpp, agg.get());
        PIC_CHECK_LAUNCH();
        count_launch();
    }
    carry_fix_batch(z, zcap, zlen, kCrtDWPC, agg.get(), count, cpp, s);
}

// Largest shorter operand (in pieces) the FP64 form multiplies exactly:
// coefficients below 2^28 (2^56 - 1)^2 < p0 p1 p2.
constexpr size_t kDblMaxPieces = (size_t)1 << 28;

// The operands' column passes (straight from the words), the fused middle pass
// and the inverse column passes of one product at length 2^k: pieces from
// index fa of a times pieces from index fb of b, residues at out + q stride.
// spec: the held operand's spectrum at this length (see ProductMiddle).
constexpr int kDblMinBits = 4;  // shortest transform of ntt_product_middle

static void ntt3d_product(uint64_t* out, size_t stride, int k, const uint32_t* a, size_t na, size_t fa,
                          const uint32_t* b, size_t nb, size_t fb, bool square, uint64_t* spec, bool spec_ready,
                          cudaStream_t s)
{
    PIC_REQUIRE(na < ((size_t)1 << 32) && nb < ((size_t)1 << 32), PIC_ERR_LENGTH, "operand too long for the FP64 form");
    auto source = [](const uint32_t* x, size_t n, size_t first) {
        SplitSrc src;
        src.words = x;
        src.n = (uint32_t)n;
        src.first = first;
        return src;
    };
    const int rows = middle_row_bits(k);
    const size_t N = (size_t)1 << k;
    const bool cols = rows < k;
    const bool need_a = !(square && spec_ready), need_b = !square && !spec_ready;
    ProductMiddle m{};
    m.out = out;
    m.out_stride = stride;
    m.square = square;
    m.sa = source(a, na, fa);
    m.sb = source(b, nb, fb);
    m.spec = spec;
    m.spec_ready = spec_ready;
    DevBuf<uint64_t> B;
    if (cols && need_a) {
        NttBatch bt = ntt3d_batch_stride(out, stride);
        bt.src = m.sa;
        ntt_forward_cols(bt, k, rows, s);
        m.a = out;
        m.a_stride = stride;
    }
    if (cols && need_b) {
        // a held b's column passes run in the buffer its spectrum will fill
        if (!spec) B = DevBuf<uint64_t>(3 * N, s);
        NttBatch bt = ntt3d_batch_stride(spec ? spec : B.get(), N);
        bt.src = m.sb;
        ntt_forward_cols(bt, k, rows, s);
        m.b = bt.data;
        m.b_stride = N;
    }
    ntt_product_middle(m, k, s);
    if (cols) ntt_inverse_cols(ntt3d_batch_stride(out, stride), k, rows, s);
}

// The wrapped form (see wrap_fix_kernel): main transforms of length 2^km, tails
// of length 2^kt over the top W pieces.
static void mul_ntt3d_wrapped(uint32_t* z, const uint32_t* a, size_t na, const uint32_t* b, size_t nb, int km,
                              int kt, Mail* mail, cudaStream_t s)
{
    const size_t zw = na + nb;
    const size_t pa = pieces56(na), pb = pieces56(nb);
    const size_t L = pa + pb - 1;
    const size_t Nm = (size_t)1 << km, T = (size_t)1 << kt, W = L - Nm;
    const bool square = (a == b && na == nb);
    bool ready = false;
    uint64_t* spec = is_held(b, nb) ? held_spectrum(km, &ready, s) : nullptr;
    DevBuf<uint64_t> A(3 * Nm, s), tA(3 * T, s);
    ntt3d_product(A.get(), Nm, km, a, na, 0, b, nb, 0, square, spec, ready, s);
    ntt3d_product(tA.get(), T, kt, a, na, Nm - pb + 1, b, nb, Nm - pa + 1, square, nullptr, false, s);
    crt3d_to_words(A.get(), Nm, km, L, crt_wrap(tA.get(), 0, T, T, Nm, W), z, zw, mail, s);
}

// The FP64 form of mul_ntt3 (PIC_MUL_NTT3D): products whose shorter operand
// has more than 2^28 pieces go to the integer form.
void mul_ntt3d(uint32_t* z, const uint32_t* a, size_t na, const uint32_t* b, size_t nb, cudaStream_t s, Mail* mail)
{
    if (is_held(a, na) && !(a == b && na == nb)) {  // the held operand goes second
        std::swap(a, b);
        std::swap(na, nb);
    }
    const size_t zw = na + nb;
    const size_t pa = pieces56(na), pb = pieces56(nb);
    if ((pa < pb ? pa : pb) > kDblMaxPieces) {
        mul_ntt3(z, a, na, b, nb, s);
        return;
    }
    const size_t ncoef = pa + pb - 1;
    int k = ceil_log2(ncoef);
    if (k < kDblMinBits) k = kDblMinBits;
    PIC_REQUIRE(k <= 30, PIC_ERR_LENGTH, "product too long for the FP64 three-prime NTT (2^30 points)");
    if (k <= kSmallMaxBits) {
        mul_small(z, a, na, b, nb, s, mail);
        return;
    }
    const size_t N = (size_t)1 << k;
    if (g_mul_wrap && k > kDblMinBits + 1) {
        const size_t Nm = N / 2;
        if (std::max(pa, pb) <= Nm && ncoef > Nm) {
            const size_t W = ncoef - Nm;
            int kt = ceil_log2(2 * W - 1);
            if (kt < kDblMinBits) kt = kDblMinBits;
            if (((size_t)1 << kt) <= Nm / 2) {
                mul_ntt3d_wrapped(z, a, na, b, nb, k - 1, kt, mail, s);
                return;
            }
        }
    }
    const bool square = (a == b && na == nb);
    bool ready = false;
    uint64_t* spec = is_held(b, nb) ? held_spectrum(k, &ready, s) : nullptr;
    DevBuf<uint64_t> A(3 * N, s);
    ntt3d_product(A.get(), N, k, a, na, 0, b, nb, 0, square, spec, ready, s);
    crt3d_to_words(A.get(), N, k, ncoef, CrtWrap{}, z, zw, mail, s);
}

void mul_ntt_ref(uint32_t* z, const uint32_t* a, size_t na, const uint32_t* b, size_t nb, cudaStream_t s)
{
    const size_t zw = na + nb;
    int k = ceil_log2(4 * zw);  // BigFloat.cpp:380-385
    PIC_REQUIRE(k <= 32, PIC_ERR_LENGTH, "product too long for the reference layout");
    const size_t N = (size_t)1 << k;
    const uint64_t p = reference_prime(k);
    const PrimeDev P = prime_tables(p).dev;
    const bool square = (a == b && na == nb);
    NttBatch bat;
    bat.stride = N;
    bat.count = 1;
    bat.per_prime = 1;
    bat.prime[0] = P;
    DevBuf<uint64_t> A(N, s), B(square ? 0 : N, s);
    split16_kernel<<<grid_for(N, 256), 256, 0, s>>>(A.get(), N, a, na);
    PIC_CHECK_LAUNCH();
    count_launch();
    bat.data = A.get();
    ntt_forward_dif(bat, k, s);
    if (!square) {
        split16_kernel<<<grid_for(N, 256), 256, 0, s>>>(B.get(), N, b, nb);
        PIC_CHECK_LAUNCH();
        count_launch();
        NttBatch bb = bat;
        bb.data = B.get();
        ntt_forward_dif(bb, k, s);
    }
    ntt_pointwise_mont(bat, square ? A.get() : B.get(), k, s);
    ntt_inverse_dit(bat, k, s);
    const uint64_t ninv = host_powmod(N % p, p - 2, p);
    coef16_to_words(A.get(), 2 * zw, to_mont(to_mont(ninv, p), p), p, P.pinv_neg, z, zw, s);
}

// ---- schoolbook ----------------------------------------------------------------
// One CTA per product, in register blocks whose rows are split where they leave
// threads idle (block_product).  Bound by latency: column sums, a
// thread a column, took computePI of 10,000 digits (43 such products) 2.09 ms for
// 1.99, a division and inverse square root of 300,007 words 3.91 for 3.84.
constexpr int kSchThreads = 256;

__global__ void __launch_bounds__(kSchThreads) school_kernel(uint32_t* __restrict__ z, const uint32_t* __restrict__ a,
                                                             uint32_t na, const uint32_t* __restrict__ b, uint32_t nb,
                                                             MailRef mail)
{
    extern __shared__ __align__(16) uint32_t sch[];
    __shared__ uint32_t s_w[32];
    block_product(sch, s_w, a, na, b, nb, [&](uint32_t w, uint32_t v) {
        z[w] = v;
        if (w + 1 == na + nb) mail_post(mail, v);  // the top word
    });
}

void mul_school(uint32_t* z, const uint32_t* a, size_t na, const uint32_t* b, size_t nb, cudaStream_t s, Mail* mail)
{
    PIC_REQUIRE(na + nb <= kSchoolMaxWords, PIC_ERR_INVALID, "schoolbook product too long");
    const size_t smem = 4 * (size_t)BlockProduct((uint32_t)na, (uint32_t)nb, kSchThreads).words();
    allow_smem(school_kernel, smem, kSchoolMaxSmem);
    ProfScope ps(KC_SCHOOL, 4.0 * (double)(2 * (na + nb)), s);
    school_kernel<<<1, kSchThreads, smem, s>>>(z, a, (uint32_t)na, b, (uint32_t)nb, mail ? mail->ref() : MailRef{});
    PIC_CHECK_LAUNCH();
    count_launch();
}

// ---- dispatch ------------------------------------------------------------------
static int64_t g_school_max_words = 256;
static int64_t g_fft_max_words = 0;

void mul_set_thresholds(int64_t school_max, int64_t fft_max)
{
    if (school_max >= 0) g_school_max_words = school_max;
    if (fft_max >= 0) g_fft_max_words = fft_max;
}
int64_t mul_school_max() { return g_school_max_words; }
int64_t mul_fft_max() { return g_fft_max_words; }

// The three-prime form AUTO and the binary splitting use: kFormInt,
// kFormDbl, or kFormChosen (per product, the form with less transform work).
static int g_ntt_form = kFormInt;
void mul_set_ntt_form(int form)
{
    PIC_REQUIRE(form == kFormInt || form == kFormDbl || form == kFormChosen, PIC_ERR_INVALID,
                "unknown product form");
    g_ntt_form = form;
}
int mul_ntt_form() { return g_ntt_form; }

// Butterfly work (sum of N log2 N over the transforms) of a three-prime
// product with `coefs` coefficients and operands of at most per_max pieces,
// under the plain / wrapped rule of mul_ntt3 and mul_ntt3d.
static double ntt_work(size_t coefs, size_t per_max, bool wrap)
{
    int k = ceil_log2(coefs);
    if (k < 1) k = 1;
    const size_t N = (size_t)1 << k;
    if (wrap && k >= 4) {
        const size_t Nm = N / 2;
        if (per_max <= Nm && coefs > Nm) {
            int kt = ceil_log2(2 * (coefs - Nm) - 1);
            if (kt < 2) kt = 2;
            if (((size_t)1 << kt) <= Nm / 2) return (double)Nm * (k - 1) + (double)((size_t)1 << kt) * kt;
        }
    }
    return (double)N * k;
}

// The FP64 form's cost per butterfly relative to the integer form's, at equal
// transform length, as timed on passes launched apart (isolated products of 2^20 ..
// 2^26 points: 0.83 - 0.90).  With the fused middle passes whole products of 2^20,
// 2^24 and 2^27 words take 0.79, 0.78 and 0.75 of the integer form's time (2^16:
// 0.98), so near the line this still favours the integer form.
constexpr double kDblWorkRatio = 0.87;

int ntt_form_for(size_t pieces_int_a, size_t pieces_int_b, size_t pieces_dbl_a, size_t pieces_dbl_b, bool wrap)
{
    if (g_ntt_form != kFormChosen) return g_ntt_form;
    const double wi = ntt_work(pieces_int_a + pieces_int_b - 1, std::max(pieces_int_a, pieces_int_b), wrap);
    const double wd = ntt_work(pieces_dbl_a + pieces_dbl_b - 1, std::max(pieces_dbl_a, pieces_dbl_b), wrap);
    return wd * kDblWorkRatio < wi ? kFormDbl : kFormInt;
}

static int product_form(size_t na, size_t nb)
{
    return ntt_form_for((na + 1) / 2, (nb + 1) / 2, pieces56(na), pieces56(nb), g_mul_wrap);
}

int mul_auto_mode(size_t na, size_t nb)
{
    const size_t mn = na < nb ? na : nb;
    const size_t zw = na + nb;
    if (zw <= kSchoolMaxWords && (mn <= 48 || (int64_t)zw <= g_school_max_words)) return PIC_MUL_SCHOOL;
    if ((int64_t)zw <= g_fft_max_words) return PIC_MUL_FFT;
    return product_form(na, nb) == kFormDbl ? PIC_MUL_NTT3D : PIC_MUL_NTT3;
}

void mul_auto_settings(std::vector<uint32_t>& out)
{
    // zw, which the thresholds are compared with, is below 2^32 in every batch
    auto word = [](int64_t v) { return (uint32_t)std::min<int64_t>(v, 0xffffffff); };
    out.push_back(word(g_school_max_words));
    out.push_back(word(g_fft_max_words));
    out.push_back((uint32_t)g_ntt_form);
    out.push_back(g_mul_wrap ? 1u : 0u);
}

static std::atomic<uint64_t> g_fft_err_bits{0};
static std::atomic<uint64_t> g_fft_err_max_bits{0};  // largest since fft_reset_max_err
double fft_last_max_err()
{
    uint64_t b = g_fft_err_bits.load();
    double d;
    memcpy(&d, &b, sizeof d);
    return d;
}
double fft_max_err_seen()
{
    uint64_t b = g_fft_err_max_bits.load();
    double d;
    memcpy(&d, &b, sizeof d);
    return d;
}
void fft_reset_max_err() { g_fft_err_max_bits.store(0); }
void fft_note_max_err(double e)
{
    uint64_t b;
    memcpy(&b, &e, sizeof b);
    g_fft_err_bits.store(b);
    // nonnegative doubles order like their bit patterns
    uint64_t cur = g_fft_err_max_bits.load();
    while (b > cur && !g_fft_err_max_bits.compare_exchange_weak(cur, b)) {
    }
}

// Largest accepted distance to the nearest integer of an FFT product's
// coefficients; past it the product is recomputed with the three-prime NTT.
// 0.25 is the production value; tests lower it to force the recompute.
static double g_fft_accept = 0.25;
void mul_set_fft_accept(double max_dist) { g_fft_accept = max_dist; }
double mul_fft_accept() { return g_fft_accept; }

void mul_dispatch(uint32_t* z, const uint32_t* a, size_t na, const uint32_t* b, size_t nb, int mode,
                  cudaStream_t s, Mail* mail)
{
    PIC_REQUIRE(na > 0 && nb > 0, PIC_ERR_INVALID, "empty operand");
    if (mode == PIC_MUL_AUTO) mode = mul_auto_mode(na, nb);
    count_products(1);
    switch (mode) {
    case PIC_MUL_SCHOOL:
        if (na + nb <= kSchoolMaxWords) {
            mul_school(z, a, na, b, nb, s, mail);
            return;
        }
        mul_ntt3(z, a, na, b, nb, s);
        return;
    case PIC_MUL_NTT_REF: mul_ntt_ref(z, a, na, b, nb, s); return;
    case PIC_MUL_NTT3: mul_ntt3(z, a, na, b, nb, s); return;
    case PIC_MUL_NTT3D: mul_ntt3d(z, a, na, b, nb, s, mail); return;
    case PIC_MUL_FFT: {
        double e = 0;
        if (!mul_fft(z, a, na, b, nb, s, &e) || e > g_fft_accept) {
            // the NTT is the oracle: a product whose rounding distance passed
            // the acceptance threshold is redone exactly
            ctx().fft_recomputes.fetch_add(1);
            if (product_form(na, nb) == kFormDbl) mul_ntt3d(z, a, na, b, nb, s);
            else mul_ntt3(z, a, na, b, nb, s);
        }
        return;
    }
    default: throw Error(PIC_ERR_INVALID, "unknown multiply mode");
    }
}

// ---- reference-API conversions ---------------------------------------------------
void int_to_ntt_dev(uint64_t* T, int k, const uint32_t* A, size_t AL, cudaStream_t s)
{
    const size_t N = (size_t)1 << k;
    PIC_REQUIRE(2 * AL <= N, PIC_ERR_LENGTH, "FFT length is too small.");
    split16_kernel<<<grid_for(N, 256), 256, 0, s>>>(T, N, A, AL);
    PIC_CHECK_LAUNCH();
    count_launch();
}

void ntt_to_int_dev(const uint64_t* T, int k, uint32_t* A, size_t AL, cudaStream_t s)
{
    const size_t N = (size_t)1 << k;
    PIC_REQUIRE(N >= 2 * AL, PIC_ERR_LENGTH, "FFT length is too small.");  // NTT.cpp:352-353
    coef16_to_words(T, 2 * AL, 0, 0, 0, A, AL, s);
}

}  // namespace pic
