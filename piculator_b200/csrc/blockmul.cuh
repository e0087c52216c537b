// Schoolbook products in 8 x 8-word register blocks.
//
// An operand of n words is ceil(n / 8) blocks.  Thread d of a product of na by
// nb blocks (na <= nb) takes the blocks (i, (d - i) mod nb) for i = 0 .. na-1:
// first the diagonal d, then, past the wrap, the diagonal d + nb, so every
// thread does the same work (a thread per diagonal or per column would do
// between none and all of it) and block i of the first operand is one address
// for all threads.  A diagonal's sum (17 words) goes to shared memory, where
// three neighbouring diagonals make a result word.
#pragma once
#include <stdint.h>

namespace pic {

constexpr int kDiagWords = 17;  // 16 words and the overflow of up to 2^32 blocks; odd: no bank conflicts

constexpr int kDiagZeros = kDiagWords + 1;  // zero words in front of a CTA's first diagonal

// e[0..8] += a * (b0, b2, b4, b6) at even distances (e[8]: the carry out)
__device__ __forceinline__ void mad_row(uint32_t* e, uint32_t a, uint32_t b0, uint32_t b2, uint32_t b4, uint32_t b6)
{
    asm("mad.lo.cc.u32 %0,%9,%10,%0; madc.hi.cc.u32 %1,%9,%10,%1;"
        "madc.lo.cc.u32 %2,%9,%11,%2; madc.hi.cc.u32 %3,%9,%11,%3;"
        "madc.lo.cc.u32 %4,%9,%12,%4; madc.hi.cc.u32 %5,%9,%12,%5;"
        "madc.lo.cc.u32 %6,%9,%13,%6; madc.hi.cc.u32 %7,%9,%13,%7; addc.u32 %8,%8,0;"
        : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(e[8])
        : "r"(a), "r"(b0), "r"(b2), "r"(b4), "r"(b6));
}

// x[0..17) += y[0..16)
__device__ __forceinline__ void add16(uint32_t* x, const uint32_t* y)
{
    asm("add.cc.u32 %0,%0,%17; "
        "addc.cc.u32 %1,%1,%18; addc.cc.u32 %2,%2,%19; addc.cc.u32 %3,%3,%20; addc.cc.u32 %4,%4,%21; "
        "addc.cc.u32 %5,%5,%22; addc.cc.u32 %6,%6,%23; addc.cc.u32 %7,%7,%24; addc.cc.u32 %8,%8,%25; "
        "addc.cc.u32 %9,%9,%26; addc.cc.u32 %10,%10,%27; addc.cc.u32 %11,%11,%28; addc.cc.u32 %12,%12,%29; "
        "addc.cc.u32 %13,%13,%30; addc.cc.u32 %14,%14,%31; addc.cc.u32 %15,%15,%32; addc.u32 %16,%16,0;"
        : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]), "+r"(x[7]), "+r"(x[8]),
          "+r"(x[9]), "+r"(x[10]), "+r"(x[11]), "+r"(x[12]), "+r"(x[13]), "+r"(x[14]), "+r"(x[15]), "+r"(x[16])
        : "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]), "r"(y[4]), "r"(y[5]), "r"(y[6]), "r"(y[7]),
          "r"(y[8]), "r"(y[9]), "r"(y[10]), "r"(y[11]), "r"(y[12]), "r"(y[13]), "r"(y[14]), "r"(y[15]));
}

// acc[0..17) += a[0..8) * b[0..8).  The products at even and at odd word
// distances are summed apart, each a chain of 64-bit multiply-adds whose carry
// ends in a word that was zero; the two sums are then added to acc.
__device__ __forceinline__ void mac_block(uint32_t (&acc)[kDiagWords], const uint32_t (&a)[8], const uint32_t (&b)[8])
{
    uint32_t e[18], o[18];  // o[k]: word k as well; o[0] stays 0
#pragma unroll
    for (int x = 0; x < 18; x++) e[x] = o[x] = 0;
#pragma unroll
    for (int x = 0; x < 8; x++) {
        mad_row((x & 1 ? o : e) + x, a[x], b[0], b[2], b[4], b[6]);
        mad_row((x & 1 ? e : o) + x + 1, a[x], b[1], b[3], b[5], b[7]);
    }
    add16(acc, e);
    add16(acc, o);
}

__device__ __forceinline__ void load_block(uint32_t (&x)[8], const uint32_t* p)
{
    const uint4 lo = *reinterpret_cast<const uint4*>(p), hi = *reinterpret_cast<const uint4*>(p + 4);
    x[0] = lo.x, x[1] = lo.y, x[2] = lo.z, x[3] = lo.w;
    x[4] = hi.x, x[5] = hi.y, x[6] = hi.z, x[7] = hi.w;
}

// Thread d's share of a product of na x nb blocks (na <= nb, d < nb): diagonals
// d and d + nb (where there are) to diag[kDiagWords * diagonal].
__device__ __forceinline__ void block_diagonals(const uint32_t* a, int na, const uint32_t* b, int nb, int d,
                                                uint32_t* diag)
{
    uint32_t acc[kDiagWords];
#pragma unroll
    for (int w = 0; w < kDiagWords; w++) acc[w] = 0;
    int j = d;
    uint32_t* out = diag + kDiagWords * d;
#pragma unroll 1
    for (int i = 0; i < na; i++) {
        if (j < 0) {  // past the wrap
            j += nb;
#pragma unroll
            for (int w = 0; w < kDiagWords; w++) {
                out[w] = acc[w];
                acc[w] = 0;
            }
            out += kDiagWords * nb;
        }
        uint32_t x[8], y[8];
        load_block(x, a + 8 * i);
        load_block(y, b + 8 * j);
        mac_block(acc, x, y);
        j--;
    }
#pragma unroll
    for (int w = 0; w < kDiagWords; w++) out[w] = acc[w];
}

// The words of one result block before carries.  `lo` is its diagonal.  A product
// is followed by a zero diagonal, which is also the one before the next product's
// first; before a CTA's first are kDiagZeros words of zero (and any word before
// them: alone it makes no carry).  Word r takes the low half of its own diagonal, the high
// half of the one before and, as the lowest word, the overflow of the one before
// that; its digit adds the carry of the sum one word below.  *gen and *prop: a bit
// for each word that makes a carry, and that passes one on (never both: a digit
// that makes a carry is at most 1).
__device__ __forceinline__ void block_digits(const uint32_t* lo, uint32_t (&t)[8], uint32_t* gen, uint32_t* prop)
{
    const uint32_t* hi = lo - kDiagWords + 8;
    uint32_t g = 0, p = 0;
    uint32_t up = (uint32_t)(((uint64_t)lo[7 - kDiagWords] + hi[7 - kDiagWords]) >> 32);
#pragma unroll
    for (int r = 0; r < 8; r++) {
        uint64_t s = (uint64_t)lo[r] + hi[r];
        if (r == 0) s += lo[16 - 2 * kDiagWords];
        t[r] = (uint32_t)s + up;
        g |= (uint32_t)(t[r] < up) << r;
        p |= (uint32_t)(t[r] == 0xffffffffu) << r;
        up = (uint32_t)(s >> 32);
    }
    *gen = g;
    *prop = p;
}

// Bit i: the carry into word i, from generate and propagate bits and a carry in.
__device__ __forceinline__ uint32_t carry_bits(uint32_t gen, uint32_t prop, uint32_t cin)
{
    return (((gen << 1) | cin) + prop) ^ prop;
}

// The carry into the calling thread's words, threads in order, each with a
// generate and a propagate bit (never both); `cin` into the first, *cout out of
// the last (whole warps, at most 32; s_w: 32 words for each call before the next
// barrier after it).  Ballots and additions in place of a scan by shuffles.
__device__ __forceinline__ uint32_t block_carry(uint32_t gen, uint32_t prop, uint32_t cin, uint32_t* s_w, uint32_t* cout)
{
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t g = __ballot_sync(0xffffffffu, gen), p = __ballot_sync(0xffffffffu, prop);
    const uint64_t sum = ((uint64_t)g << 1) + p;
    if (lane == 0) s_w[wid] = (uint32_t)(sum >> 32) | ((uint32_t)(p == 0xffffffffu) << 1);
    __syncthreads();
    const uint32_t w = lane < nw ? s_w[lane] : 0u;
    const uint32_t gw = __ballot_sync(0xffffffffu, w & 1u), pw = __ballot_sync(0xffffffffu, w >> 1);
    const uint64_t cw = ((((uint64_t)gw << 1) | cin) + pw) ^ pw;  // bit i: into warp i
    *cout = (uint32_t)(cw >> nw) & 1u;
    return (uint32_t)((((((uint64_t)g << 1) | ((cw >> wid) & 1u)) + p) ^ p) >> lane) & 1u;
}

// One product by a whole CTA of T threads (whole warps): rows of at most T
// threads, and where they leave threads idle the first operand's blocks are split
// into up to eight runs, each with diagonals of its own.
struct BlockProduct {
    uint32_t ma, mb, S;  // blocks of the shorter and of the longer operand; runs
    __host__ __device__ BlockProduct(uint32_t na, uint32_t nb, uint32_t T)
    {
        const uint32_t x = (na + 7) / 8, y = (nb + 7) / 8;
        ma = x < y ? x : y;
        mb = x < y ? y : x;
        S = mb ? T / mb : 1;
        if (S > 8) S = 8;
        if (S > ma) S = ma;
        if (S < 1) S = 1;
    }
    __host__ __device__ uint32_t words() const { return (ma + mb) * (8 + S * kDiagWords); }
};

// put(w, v): word w of a * b, w < na + nb, from one thread each.  sm: 16-byte
// aligned, words() words; s_w: 32 words.  Ends without a barrier.
template <class Put>
__device__ __forceinline__ void block_product(uint32_t* sm, uint32_t* s_w, const uint32_t* __restrict__ a, uint32_t na,
                                              const uint32_t* __restrict__ b, uint32_t nb, const Put& put)
{
    const uint32_t T = blockDim.x, tid = threadIdx.x, lane = tid & 31, zw = na + nb;
    if (na > nb) {
        const uint32_t* p = a;
        a = b, b = p;
        const uint32_t n = na;
        na = nb, nb = n;
    }
    const BlockProduct P(na, nb, T);
    const uint32_t slots = P.ma + P.mb;
    uint32_t* sa = sm;
    uint32_t* sb = sa + 8 * P.ma;
    uint32_t* diag = sb + 8 * P.mb;
    for (uint32_t i = tid; i < 8 * P.ma; i += T) sa[i] = i < na ? a[i] : 0u;
    for (uint32_t i = tid; i < 8 * P.mb; i += T) sb[i] = i < nb ? b[i] : 0u;
    for (uint32_t i = tid; i < P.S * slots * kDiagWords; i += T) diag[i] = 0;  // slots a run does not reach
    __syncthreads();
    for (uint32_t t = tid; t < P.S * P.mb; t += T) {
        const uint32_t run = t / P.mb, d = t - run * P.mb;
        const uint32_t i0 = run * P.ma / P.S, i1 = (run + 1) * P.ma / P.S;
        block_diagonals(sa + 8 * i0, (int)(i1 - i0), sb, (int)P.mb, (int)d, diag + kDiagWords * (run * slots + i0));
    }
    __syncthreads();
    // a thread per word; sums of at most 2^32 (2 S + 1): digits as in block_digits
    auto sum = [&](uint32_t w) {
        const uint32_t c = w >> 3, r = w & 7;
        uint64_t s = 0;
        for (uint32_t run = 0; run < P.S; run++) {
            const uint32_t* p = diag + kDiagWords * (run * slots + c) + r;
            s += p[0];
            if (c >= 1) s += p[8 - kDiagWords];
            if (c >= 2 && r == 0) s += p[16 - 2 * kDiagWords];
        }
        return s;
    };
    uint32_t cin = 0;
    for (uint32_t base = 0; base < zw; base += T) {
        const uint32_t w = base + tid;
        const uint64_t s = w < zw ? sum(w) : 0;
        uint32_t up = __shfl_up_sync(0xffffffffu, (uint32_t)(s >> 32), 1);
        if (lane == 0) up = w > 0 && w < zw ? (uint32_t)(sum(w - 1) >> 32) : 0u;
        const uint32_t t = (uint32_t)s + up;
        uint32_t cout;
        const uint32_t c = block_carry(t < up, t == 0xffffffffu, cin, s_w, &cout);
        cin = cout;
        if (w < zw) put(w, t + c);
        if (base + T < zw) __syncthreads();  // s_w again
    }
}

}  // namespace pic
