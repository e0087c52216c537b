// Carry (and borrow) resolution over long word arrays.
//
// Every linear step of the path -- the product's coefficient-to-word
// conversion (ntt_to_int NTT.cpp:343-369, fft_to_int FFT.cpp:520-571), uadd /
// usub (BigFloat.cpp:184-287) and mul(uint32) (BigFloat.cpp:156-183) -- is a
// sequential carry loop in the reference.  Here each word first gets a raw
// digit d_i and a "generate" bit g_i (carry out no matter what comes in); the
// carry into word i is then the carry-lookahead prefix
//     c_(i+1) = g_i | (p_i & c_i),   p_i = (d_i == all-ones)   [add]
//     b_(i+1) = g_i | (p_i & b_i),   p_i = (d_i == 0)          [subtract]
// which is associative, so it runs as a block scan inside each CTA plus a
// second launch for the carries between CTAs (no inter-CTA waiting, no spin
// loops):
//   K1  raw digits -> in-block resolved words + one (G, P) per CTA
//   K2  each CTA takes its carry-in from the aggregates below it and, if it is
//       1, ripples it through its own words.
// A chunk passes a carry on only when all its words are all-ones (zero), so
// the aggregate just below decides almost always; where it does not, the CTA
// scans all those below it.  Of more than kCarryDirect chunks a launch between
// the two makes one (G, P) per kCarryGroup chunks, and a CTA scans those of the
// groups below and its own group's: scanning every chunk below takes time that
// grows with the square of a run of all-ones (zero) words, 28 ms of the
// difference of two equal numbers of 4e8 words where their words take 4; the
// launch costs 3 us, a scan of as many chunks as the line allows some 25.
// Against a scan launch and a ripple launch (three in all): division and inverse
// square root at 300,007 words 9.65 -> 4.17 ms together with the results posted
// to the host (common.cuh) and the comparison of a difference left on the
// device.  Doing K2 in the CTA of K1 that finishes last was slower (6.1 ms): its
// fences, and the runs of all-ones words that a Newton step's x r ~ 1 leaves to
// that one CTA.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace pic {

// (g, p) packed as bit0 = generate, bit1 = propagate.  Identity = propagate.
constexpr uint32_t kGPIdentity = 2u;

__device__ __forceinline__ uint32_t gp_combine(uint32_t lo, uint32_t hi)
{
    const uint32_t g = (hi & 1u) | ((hi >> 1) & lo & 1u);
    const uint32_t p = (hi >> 1) & (lo >> 1) & 1u;
    return g | (p << 1);
}

// Exclusive block scan of one (g, p) per thread, threads in position order.
// Returns the exclusive prefix; *total receives the block aggregate.  Must be
// called by every thread of the block (blockDim.x a multiple of 32, <= 1024).
__device__ __forceinline__ uint32_t block_gp_scan(uint32_t gp, uint32_t* total)
{
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_tot;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nw = (blockDim.x + 31) >> 5;
    uint32_t v = gp;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        uint32_t o = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= off) v = gp_combine(o, v);
    }
    uint32_t excl = __shfl_up_sync(0xffffffffu, v, 1);
    if (lane == 0) excl = kGPIdentity;
    if (lane == 31) s_warp[wid] = v;
    __syncthreads();
    if (wid == 0) {
        uint32_t w = lane < nw ? s_warp[lane] : kGPIdentity;
        uint32_t iv = w;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t o = __shfl_up_sync(0xffffffffu, iv, off);
            if (lane >= off) iv = gp_combine(o, iv);
        }
        uint32_t ex = __shfl_up_sync(0xffffffffu, iv, 1);
        if (lane == 0) ex = kGPIdentity;
        if (lane == 31) s_tot = iv;
        __syncwarp();
        s_warp[lane] = ex;
    }
    __syncthreads();
    const uint32_t res = gp_combine(s_warp[wid], excl);
    const uint32_t tot = s_tot;
    __syncthreads();
    *total = tot;
    return res;
}

// Warp-reduced max / min: one shared or global atomic per warp instead of one
// per qualifying element (a single hot address serialises per-element atomics).
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v)
{
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, off);
        v = o > v ? o : v;
    }
    return v;
}

__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v)
{
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, off);
        v = o < v ? o : v;
    }
    return v;
}

// Block-wide max of one value per thread (all threads call; blockDim % 32 == 0).
__device__ __forceinline__ unsigned long long block_max_u64(unsigned long long v)
{
    __shared__ unsigned long long s_m;
    if (threadIdx.x == 0) s_m = 0;
    __syncthreads();
    v = warp_max_u64(v);
    if ((threadIdx.x & 31) == 0 && v) atomicMax(&s_m, v);
    __syncthreads();
    const unsigned long long r = s_m;
    __syncthreads();
    return r;
}

__device__ __forceinline__ unsigned long long block_min_u64(unsigned long long v)
{
    __shared__ unsigned long long s_m;
    if (threadIdx.x == 0) s_m = ~0ull;
    __syncthreads();
    v = warp_min_u64(v);
    if ((threadIdx.x & 31) == 0 && v != ~0ull) atomicMin(&s_m, v);
    __syncthreads();
    const unsigned long long r = s_m;
    __syncthreads();
    return r;
}

// The last CTA of a launch: true in exactly one of `nctas` CTAs, after every
// other one has arrived; what those wrote before is visible to it through
// loads that bypass L1 (__ldcg).  *ticket is zero before the launch and after it.
__device__ __forceinline__ bool last_cta(uint32_t* ticket, uint32_t nctas)
{
    __shared__ bool s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == nctas - 1;
        if (s_last) {
            *ticket = 0;
            __threadfence();
        }
    }
    __syncthreads();
    return s_last;
}

constexpr size_t kCarryDirect = 8192, kCarryGroup = 512;

// Groups of an item of cpp chunks (0: none), and the words its aggregates take:
// `count` items of cpp chunks, then their groups.
inline size_t carry_groups(size_t cpp) { return cpp > kCarryDirect ? (cpp + kCarryGroup - 1) / kCarryGroup : 0; }
inline size_t carry_agg_words(size_t count, size_t cpp) { return count * (cpp + carry_groups(cpp)); }

// The aggregates of one item as K2 reads them.
struct CarryAgg {
    const uint32_t* chunk;
    const uint32_t* group;  // null: none
    __host__ __device__ CarryAgg item(size_t i, size_t cpp) const
    {
        return CarryAgg{chunk + i * cpp, group ? group + i * ((cpp + kCarryGroup - 1) / kCarryGroup) : nullptr};
    }
};
// Makes the groups of `count` items where there are any (agg: carry_agg_words).
CarryAgg carry_group(uint32_t* agg, size_t count, size_t cpp, cudaStream_t s);

// The carry into chunk c of an item from the (G, P) of chunks 0 .. c - 1 (every
// thread calls, the same result in each).
__device__ __forceinline__ uint32_t chunk_carry_in(const CarryAgg& A, size_t c)
{
    if (c == 0) return 0;
    const uint32_t below = A.chunk[c - 1];
    if (!(below & 2u)) return below & 1u;
    const size_t ng = A.group ? c / kCarryGroup : 0, c0 = ng * kCarryGroup, n = ng + (c - c0);
    const size_t per = (n + blockDim.x - 1) / blockDim.x;
    const size_t b = threadIdx.x * per < n ? threadIdx.x * per : n, e = b + per < n ? b + per : n;
    uint32_t acc = kGPIdentity;
    for (size_t i = b; i < e; i++) acc = gp_combine(acc, i < ng ? A.group[i] : A.chunk[c0 + (i - ng)]);
    uint32_t total;
    block_gp_scan(acc, &total);
    return total & 1u;
}

// A carry (borrow) of one into words z[b, e): passed on over words equal to
// `stop` (which become ~stop) to the first that takes it.
__device__ __forceinline__ void chunk_ripple(uint32_t* z, size_t b, size_t e, bool sub)
{
    const uint32_t stop = sub ? 0u : 0xffffffffu;
    if (b >= e) return;
    const uint32_t w = z[b];
    if (w != stop) {  // the same for every thread: they have all read it
        __syncthreads();
        if (threadIdx.x == 0) z[b] = sub ? w - 1u : w + 1u;
        return;
    }
    unsigned long long mine = ~0ull;
    for (size_t i = b + threadIdx.x; i < e; i += blockDim.x)
        if (z[i] != stop && i < mine) mine = i;
    const size_t f = (size_t)block_min_u64(mine);
    for (size_t i = b + threadIdx.x; i < e && i < f; i += blockDim.x) z[i] = ~stop;
    if (threadIdx.x == 0 && f < e) z[f] += sub ? 0xffffffffu : 1u;
}

// K2 (carry.cu).  agg[c] = (G, P) of CTA c, which owns words_per_cta words;
// carry_agg_words(1, nctas) words.  mail: receives the top word z[nwords - 1].
void carry_fix(uint32_t* z, size_t nwords, size_t words_per_cta, uint32_t* agg, size_t nctas, cudaStream_t s,
               MailRef mail = MailRef{});
// For batches of products: `count` segments of `cpp` CTAs; product i writes
// zlen[i] words at z + i * zcap; agg of carry_agg_words(count, cpp) words.
void carry_fix_batch(uint32_t* z, uint32_t zcap, const uint32_t* zlen, size_t words_per_cta, uint32_t* agg,
                     size_t count, size_t cpp, cudaStream_t s, bool sub = false);

}  // namespace pic
