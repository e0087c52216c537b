// Cross-CTA carry phases and the BigFloat linear kernels (windowed add/sub,
// multiply by a 32-bit word, leading-zero search, magnitude compare).
#include <cooperative_groups.h>

#include "carry.cuh"
#include "common.cuh"
#include "linear.cuh"

namespace cg = cooperative_groups;

namespace pic {

// ---- groups of chunks ---------------------------------------------------------
__global__ void __launch_bounds__(256) carry_group_kernel(const uint32_t* __restrict__ agg, size_t cpp, size_t groups,
                                                          uint32_t* __restrict__ out)
{
    const size_t item = blockIdx.x / groups, g = blockIdx.x - item * groups;
    const uint32_t* a = agg + item * cpp;
    constexpr int IPT = (int)kCarryGroup / 256;
    const size_t i0 = g * kCarryGroup + (size_t)threadIdx.x * IPT;
    uint32_t acc = kGPIdentity;
#pragma unroll
    for (int u = 0; u < IPT; u++)
        if (i0 + u < cpp) acc = gp_combine(acc, a[i0 + u]);
    uint32_t total;
    block_gp_scan(acc, &total);
    if (threadIdx.x == 0) out[blockIdx.x] = total;
}

CarryAgg carry_group(uint32_t* agg, size_t count, size_t cpp, cudaStream_t s)
{
    const size_t groups = carry_groups(cpp);
    if (groups == 0) return CarryAgg{agg, nullptr};
    uint32_t* out = agg + count * cpp;
    carry_group_kernel<<<(unsigned)(count * groups), 256, 0, s>>>(agg, cpp, groups, out);
    PIC_CHECK_LAUNCH();
    count_launch();
    return CarryAgg{agg, out};
}

// ---- K2 ---------------------------------------------------------------------
__global__ void __launch_bounds__(256) carry_fix_kernel(uint32_t* z, size_t n, size_t wpc,
                                                        CarryAgg agg, size_t nctas, MailRef mail)
{
    const size_t c = blockIdx.x;
    const size_t b = c * wpc, e = b + wpc < n ? b + wpc : n;
    if (chunk_carry_in(agg, c)) chunk_ripple(z, b, e, false);
    if (mail.slot != nullptr && c == nctas - 1) {
        __syncthreads();
        if (threadIdx.x == 0) mail_post(mail, z[n - 1]);
    }
}

void carry_fix(uint32_t* z, size_t nwords, size_t words_per_cta, uint32_t* agg, size_t nctas, cudaStream_t s,
               MailRef mail)
{
    ProfScope ps(KC_CARRY, 4.0 * (double)nctas, s);
    const CarryAgg A = carry_group(agg, 1, nctas, s);
    carry_fix_kernel<<<(unsigned)nctas, 256, 0, s>>>(z, nwords, words_per_cta, A, nctas, mail);
    PIC_CHECK_LAUNCH();
    count_launch();
}

__global__ void __launch_bounds__(256) carry_fix_batch_kernel(uint32_t* z, uint32_t zcap,
                                                              const uint32_t* __restrict__ zlen, size_t wpc,
                                                              CarryAgg agg, size_t cpp, bool sub)
{
    const size_t prod = blockIdx.x / cpp, c = blockIdx.x - prod * cpp;
    const size_t n = zlen[prod];
    const size_t b = c * wpc, e = b + wpc < n ? b + wpc : n;
    if (b >= e || !chunk_carry_in(agg.item(prod, cpp), c)) return;
    chunk_ripple(z + prod * (size_t)zcap, b, e, sub);
}

void carry_fix_batch(uint32_t* z, uint32_t zcap, const uint32_t* zlen, size_t words_per_cta, uint32_t* agg,
                     size_t count, size_t cpp, cudaStream_t s, bool sub)
{
    if (cpp <= 1) return;  // one CTA per product: no carries between CTAs
    ProfScope ps(KC_CARRY, 4.0 * (double)(count * cpp), s);
    const CarryAgg A = carry_group(agg, count, cpp, s);
    carry_fix_batch_kernel<<<(unsigned)(count * cpp), 256, 0, s>>>(z, zcap, zlen, words_per_cta, A, cpp, sub);
    PIC_CHECK_LAUNCH();
    count_launch();
}

// ---- K1 for the linear ops --------------------------------------------------
// Each thread owns kLinIPT consecutive words; a CTA owns blockDim * kLinIPT.
constexpr int kLinIPT = 8;
constexpr int kLinThreads = 256;
constexpr size_t kLinWPC = (size_t)kLinIPT * kLinThreads;

__device__ __forceinline__ uint32_t word_at(const uint32_t* T, int64_t exp, int64_t L, int64_t mag)
{
    // BigFloat::word_at, BigFloat.cpp:109-122
    const int64_t i = mag - exp;
    return (i >= 0 && i < L) ? T[i] : 0u;
}

// How a linear operation on z[0, n) ends: the word above it and the result.
enum LinKind { kLinAdd = 0, kLinSub = 1, kLinMul = 2 };

struct LinEnd {
    int kind;
    uint32_t* carry_out;  // the carry's (kLinMul: the top word's) place, may be null
    uint32_t top_hi;      // kLinMul: the top word's part of the last product, set by the kernels
    const int* order;     // kLinSub: posted beside the length
    unsigned long long* diff;  // kLinSub over several CTAs: zero before and after
    uint32_t* ticket;
    MailRef mail;
};

// The end of the CTA that holds words [b, e) of z, its carry-in resolved
// (`carry` out of it).  Every thread calls.
__device__ __forceinline__ void lin_end(const LinEnd& E, const uint32_t* z, size_t b, size_t e, uint32_t carry,
                                        uint32_t nctas)
{
    if (E.kind == kLinSub) {
        if (E.mail.slot == nullptr) return;
        __syncthreads();
        unsigned long long mine = 0;
        for (size_t i = b + threadIdx.x; i < e; i += blockDim.x)
            if (z[i] != 0u) mine = i + 1;
        mine = block_max_u64(mine);
        if (nctas > 1) {
            if (threadIdx.x == 0 && mine) atomicMax(E.diff, mine);
            if (!last_cta(E.ticket, nctas)) return;
            if (threadIdx.x == 0) {
                mine = __ldcg(E.diff);
                *E.diff = 0;
            }
        }
        if (threadIdx.x == 0) mail_post(E.mail, mine, E.order == nullptr || *E.order > 0 ? 1u : 0u);
        return;
    }
    if (blockIdx.x == nctas - 1 && threadIdx.x == 0) {
        const uint32_t v = carry + (E.kind == kLinMul ? E.top_hi : 0u);
        if (E.carry_out != nullptr) *E.carry_out = v;
        mail_post(E.mail, v);
    }
}

// K2 of the linear operations (several CTAs).
__global__ void __launch_bounds__(kLinThreads) lin_fix_kernel(uint32_t* z, size_t n, CarryAgg agg, uint32_t nctas,
                                                              LinEnd E, const uint32_t* a, uint32_t x)
{
    const size_t c = blockIdx.x;
    const size_t b = c * kLinWPC, e = b + kLinWPC < n ? b + kLinWPC : n;
    const uint32_t cin = chunk_carry_in(agg, c);
    const uint32_t gp = agg.chunk[c];
    if (cin) chunk_ripple(z, b, e, E.kind == kLinSub);
    if (E.kind == kLinMul) E.top_hi = (uint32_t)(((uint64_t)a[n - 1] * x) >> 32);
    lin_end(E, z, b, e, (gp & 1u) | ((gp >> 1) & cin), nctas);
}

// Windowed add / subtract of two magnitudes: z[c] = a(bot+c) +/- b(bot+c).
// order (subtract): b - a when *order is not positive.  A single CTA ends the
// operation itself.
__global__ void __launch_bounds__(kLinThreads) addsub_k1(uint32_t* z, size_t TL, WordView va, WordView vb,
                                                         int64_t bot, uint32_t* agg, LinEnd E)
{
    const bool ord = E.order == nullptr || *E.order > 0, add = E.kind == kLinAdd;
    const WordView a = ord ? va : vb, b = ord ? vb : va;
    const size_t i0 = (size_t)blockIdx.x * kLinWPC + (size_t)threadIdx.x * kLinIPT;
    uint32_t d[kLinIPT], gg[kLinIPT];
    uint32_t gp = kGPIdentity;
#pragma unroll
    for (int u = 0; u < kLinIPT; u++) {
        const size_t i = i0 + u;
        uint32_t g = 0, dig = 0;
        if (i < TL) {
            const int64_t mag = bot + (int64_t)i;
            const uint32_t x = word_at(a.T, a.exp, a.L, mag), y = word_at(b.T, b.exp, b.L, mag);
            if (add) {
                const uint64_t s = (uint64_t)x + y;
                dig = (uint32_t)s;
                g = (uint32_t)(s >> 32);
            } else {
                dig = x - y;
                g = x < y;
            }
        }
        const uint32_t p = add ? (dig == 0xffffffffu) : (dig == 0u);
        d[u] = dig;
        gg[u] = g;
        if (i < TL) gp = gp_combine(gp, g | (p << 1));  // padding is the scan identity
    }
    uint32_t total;
    uint32_t cin = block_gp_scan(gp, &total) & 1u;
#pragma unroll
    for (int u = 0; u < kLinIPT; u++) {
        const size_t i = i0 + u;
        if (i >= TL) break;
        const uint32_t dig = d[u];
        uint32_t p;
        if (add) {
            z[i] = dig + cin;
            p = dig == 0xffffffffu;
        } else {
            z[i] = dig - cin;
            p = dig == 0u;
        }
        cin = gg[u] | (p & cin);
    }
    if (gridDim.x > 1) {
        if (threadIdx.x == 0) agg[blockIdx.x] = total;
    } else {
        lin_end(E, z, 0, TL, total & 1u, 1);
    }
}

// z[c] = low(a_c x) + high(a_(c-1) x), carries inside each CTA resolved (several
// CTAs: lin_one serves shorter numbers); lin_fix passes on the others and writes z[L].
__global__ void __launch_bounds__(kLinThreads) mulu32_k1(uint32_t* z, const uint32_t* a, size_t L, uint32_t x,
                                                         uint32_t* agg)
{
    const size_t i0 = (size_t)blockIdx.x * kLinWPC + (size_t)threadIdx.x * kLinIPT;
    uint32_t d[kLinIPT], gg[kLinIPT];
    uint32_t gp = kGPIdentity;
    uint32_t prev_hi = 0;
    if (i0 > 0 && i0 - 1 < L) prev_hi = (uint32_t)(((uint64_t)a[i0 - 1] * x) >> 32);
#pragma unroll
    for (int u = 0; u < kLinIPT; u++) {
        const size_t i = i0 + u;
        uint32_t g = 0, dig = 0;
        if (i < L) {
            const uint64_t pr = (uint64_t)a[i] * x;
            const uint64_t s = (uint64_t)(uint32_t)pr + prev_hi;
            dig = (uint32_t)s;
            g = (uint32_t)(s >> 32);
            prev_hi = (uint32_t)(pr >> 32);
        }
        d[u] = dig;
        gg[u] = g;
        if (i < L) gp = gp_combine(gp, g | ((uint32_t)(dig == 0xffffffffu) << 1));
    }
    uint32_t total;
    uint32_t cin = block_gp_scan(gp, &total) & 1u;
#pragma unroll
    for (int u = 0; u < kLinIPT; u++) {
        const size_t i = i0 + u;
        if (i >= L) break;
        z[i] = d[u] + cin;
        cin = gg[u] | ((uint32_t)(d[u] == 0xffffffffu) & cin);
    }
    if (threadIdx.x == 0) agg[blockIdx.x] = total;
}

__global__ void set_words_kernel(uint32_t* p, uint32_t lo, uint32_t hi, int n)
{
    p[0] = lo;
    if (n > 1) p[1] = hi;
}

void lin_set(uint32_t* p, uint32_t lo, uint32_t hi, int n, cudaStream_t s)
{
    set_words_kernel<<<1, 1, 0, s>>>(p, lo, hi, n);
    PIC_CHECK_LAUNCH();
    count_launch();
}

static size_t lin_ctas(size_t n) { return (n + kLinWPC - 1) / kLinWPC; }

static void lin_fix(uint32_t* z, size_t n, uint32_t* agg, size_t nctas, const LinEnd& E, const uint32_t* a,
                    uint32_t x, cudaStream_t s)
{
    if (nctas <= 1) return;
    ProfScope ps(KC_CARRY, 4.0 * (double)nctas, s);
    const CarryAgg A = carry_group(agg, 1, nctas, s);
    lin_fix_kernel<<<(unsigned)nctas, kLinThreads, 0, s>>>(z, n, A, (uint32_t)nctas, E, a, x);
    PIC_CHECK_LAUNCH();
    count_launch();
}

static void addsub(uint32_t* z, size_t TL, const WordView& a, const WordView& b, int64_t bot, const LinEnd& E,
                   cudaStream_t s)
{
    const size_t nctas = lin_ctas(TL);
    DevBuf<uint32_t> agg(carry_agg_words(1, nctas), s);
    ProfScope ps(KC_LINEAR, 12.0 * (double)TL, s);
    addsub_k1<<<(unsigned)nctas, kLinThreads, 0, s>>>(z, TL, a, b, bot, agg.get(), E);
    PIC_CHECK_LAUNCH();
    count_launch();
    lin_fix(z, TL, agg.get(), nctas, E, nullptr, 0, s);
}

void lin_addsub(uint32_t* z, size_t TL, const WordView& a, const WordView& b, int64_t bot, bool sub,
                cudaStream_t s)
{
    if (TL == 0) return;
    LinEnd E{};
    E.kind = sub ? kLinSub : kLinAdd;
    addsub(z, TL, a, b, bot, E, s);
}

// The words of ctx().scratch: kernels of the library's stream run one after
// another, so one set serves them all.
static uint32_t* scratch_ticket() { return ctx().scratch; }
static int* scratch_order() { return reinterpret_cast<int*>(ctx().scratch + 1); }
static unsigned long long* scratch_diff() { return reinterpret_cast<unsigned long long*>(ctx().scratch + 2); }

// ---- a whole operation in one launch ------------------------------------------
// Numbers of up to kOneWords words: a cluster of one to eight CTAs holds all of
// the window's words in registers (eight a thread), so the comparison that orders
// a difference, the carries between the CTAs and the highest nonzero word go
// through distributed shared memory, where the longer form launches a comparison,
// the digits and the carries apart: a difference of 30,000 words costs one launch
// of 6 us for three of 3.8, 4.1 and 6 us, computePI of 10,000 digits 2.25 -> 2.11
// ms, of a million 5.55 -> 5.14, a reciprocal of 300,000 digits 4.25 -> 3.92.
// Eight CTAs are the largest cluster that every device schedules; above it the
// words no longer fit one and the longer form's bandwidth counts.
constexpr int kOneIPT = 8;
constexpr int kOneCtas = 8;
constexpr size_t kOneWords = (size_t)1024 * kOneIPT * kOneCtas;

struct OneArgs {
    uint32_t* z;
    int64_t n;           // words of the window
    int kind;            // LinKind
    int ask;             // kLinSub: compare first
    const uint32_t *a, *b;
    int64_t da, db, la, lb;  // the window's word i is a[i + da] (0 outside [0, la)), b likewise
    uint32_t x;          // kLinMul
    MailRef mail;
};

// The largest of the CTAs' values (every thread of the cluster calls).
__device__ __forceinline__ unsigned long long cluster_max(cg::cluster_group& cluster, unsigned long long* s_v,
                                                          unsigned long long v)
{
    v = block_max_u64(v);
    if (threadIdx.x == 0) *s_v = v;
    cluster.sync();
    unsigned long long m = 0;
    for (unsigned r = 0; r < cluster.num_blocks(); r++) {
        const unsigned long long o = *cluster.map_shared_rank(s_v, r);
        m = o > m ? o : m;
    }
    return m;
}

__global__ void __launch_bounds__(1024) lin_one_kernel(const __grid_constant__ OneArgs A)
{
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ unsigned long long s_v[2];
    __shared__ uint32_t s_gp;
    const int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * kOneIPT;
    auto at = [](const uint32_t* p, int64_t i, int64_t l) -> uint32_t { return (uint64_t)i < (uint64_t)l ? p[i] : 0u; };
    const bool add = A.kind != kLinSub;
    uint32_t x[kOneIPT], y[kOneIPT];
#pragma unroll
    for (int u = 0; u < kOneIPT; u++) {
        const int64_t i = i0 + u;
        x[u] = i < A.n ? at(A.a, i + A.da, A.la) : 0u;
        y[u] = i < A.n && A.kind != kLinMul ? at(A.b, i + A.db, A.lb) : 0u;
    }
    bool swap = false;
    if (A.ask) {
        unsigned long long mine = 0;
#pragma unroll
        for (int u = 0; u < kOneIPT; u++)
            if (x[u] != y[u]) mine = (unsigned long long)(i0 + u + 1);
        // equal in the window: zero in either order, whatever lies under it (a search
        // there by one cluster took 31 ms for two numbers of 2^24 words)
        const int64_t i = (int64_t)cluster_max(cluster, &s_v[0], mine) - 1;
        swap = i < 0 || at(A.a, i + A.da, A.la) < at(A.b, i + A.db, A.lb);
    }
    uint32_t d[kOneIPT], gg[kOneIPT];
    uint32_t gp = kGPIdentity;
    uint32_t prev_hi = 0;
    if (A.kind == kLinMul && i0 > 0 && i0 - 1 < A.n) prev_hi = (uint32_t)(((uint64_t)A.a[i0 - 1] * A.x) >> 32);
#pragma unroll
    for (int u = 0; u < kOneIPT; u++) {
        uint64_t s;
        if (A.kind == kLinMul) {
            const uint64_t pr = (uint64_t)x[u] * A.x;
            s = (uint64_t)(uint32_t)pr + prev_hi;
            prev_hi = (uint32_t)(pr >> 32);
        } else if (add) {
            s = (uint64_t)x[u] + y[u];
        } else {
            s = swap ? (uint64_t)y[u] - x[u] : (uint64_t)x[u] - y[u];
        }
        d[u] = (uint32_t)s;
        gg[u] = (uint32_t)(s >> 32) & 1u;
        const uint32_t p = add ? (d[u] == 0xffffffffu) : (d[u] == 0u);
        if (i0 + u < A.n) gp = gp_combine(gp, gg[u] | (p << 1));
    }
    const uint32_t last = A.kind == kLinMul ? A.a[A.n - 1] : 0u;
    uint32_t total;
    const uint32_t pre = block_gp_scan(gp, &total);
    if (threadIdx.x == 0) s_gp = total;
    cluster.sync();  // every word of the operands has been read: z may be one of them
    uint32_t cc = 0;  // carry into this CTA, then out of the last one
    for (unsigned r = 0; r < blockIdx.x; r++) {
        const uint32_t o = *cluster.map_shared_rank(&s_gp, r);
        cc = (o & 1u) | ((o >> 1) & cc);
    }
    uint32_t cin = (pre & 1u) | ((pre >> 1) & cc);
    unsigned long long top = 0;
#pragma unroll
    for (int u = 0; u < kOneIPT; u++) {
        if (i0 + u >= A.n) break;
        const uint32_t w = add ? d[u] + cin : d[u] - cin;
        const uint32_t p = add ? (d[u] == 0xffffffffu) : (d[u] == 0u);
        A.z[i0 + u] = w;
        if (w) top = (unsigned long long)(i0 + u + 1);
        cin = gg[u] | (p & cin);
    }
    if (!add) {
        top = cluster_max(cluster, &s_v[1], top);
        if (blockIdx.x == 0 && threadIdx.x == 0) mail_post(A.mail, top, swap ? 0u : 1u);
    } else if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        uint32_t v = (total & 1u) | ((total >> 1) & cc);
        if (A.kind == kLinMul) v += (uint32_t)(((uint64_t)last * A.x) >> 32);
        A.z[A.n] = v;
        mail_post(A.mail, v);
    }
    cluster.sync();  // the others may still read this CTA's shared words
}

static uint64_t lin_one(OneArgs& A, uint32_t* bits)
{
    const cudaStream_t s = ctx().stream;
    Mail mail(s);
    A.mail = mail.ref();
    const unsigned threads = A.n <= 256 * kOneIPT ? 256 : 1024;
    const unsigned ctas = (unsigned)((A.n + threads * kOneIPT - 1) / (threads * kOneIPT));
    ProfScope ps(KC_LINEAR, 12.0 * (double)A.n, s);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    PIC_CUDA(cudaLaunchKernelEx(&cfg, lin_one_kernel, A));
    count_launch();
    return mail.wait(bits);
}

static OneArgs one_args(uint32_t* z, size_t TL, const WordView& a, const WordView& b, int64_t bot, int kind)
{
    OneArgs A{};
    A.z = z;
    A.n = (int64_t)TL;
    A.kind = kind;
    A.a = a.T;
    A.b = b.T;
    A.da = bot - a.exp;
    A.db = bot - b.exp;
    A.la = a.L;
    A.lb = b.L;
    return A;
}

uint32_t lin_add(uint32_t* z, size_t TL, const WordView& a, const WordView& b, int64_t bot)
{
    if (TL == 0) {
        PIC_CUDA(cudaMemsetAsync(z, 0, sizeof(uint32_t), ctx().stream));
        return 0;
    }
    if (TL <= kOneWords) {
        OneArgs A = one_args(z, TL, a, b, bot, kLinAdd);
        return (uint32_t)lin_one(A, nullptr);
    }
    Mail mail(ctx().stream);
    LinEnd E{};
    E.kind = kLinAdd;
    E.carry_out = z + TL;
    E.mail = mail.ref();
    addsub(z, TL, a, b, bot, E, ctx().stream);
    return (uint32_t)mail.wait();
}

uint32_t lin_mul_u32(uint32_t* z, const uint32_t* a, size_t L, uint32_t x)
{
    const cudaStream_t s = ctx().stream;
    if (L <= kOneWords) {
        OneArgs A = one_args(z, L, WordView{a, 0, (int64_t)L}, WordView{a, 0, 0}, 0, kLinMul);
        A.x = x;
        return (uint32_t)lin_one(A, nullptr);
    }
    const size_t nctas = lin_ctas(L);
    Mail mail(s);
    DevBuf<uint32_t> agg(carry_agg_words(1, nctas), s);
    LinEnd E{};
    E.kind = kLinMul;
    E.carry_out = z + L;
    E.mail = mail.ref();
    {
        ProfScope ps(KC_LINEAR, 8.0 * (double)L, s);
        mulu32_k1<<<(unsigned)nctas, kLinThreads, 0, s>>>(z, a, L, x, agg.get());
        PIC_CHECK_LAUNCH();
        count_launch();
        lin_fix(z, L, agg.get(), nctas, E, a, x, s);
    }
    return (uint32_t)mail.wait();
}

// ---- leading zeros / compare -------------------------------------------------
__global__ void top_nonzero_kernel(const uint32_t* z, size_t n, unsigned long long* out)
{
    // out = 1 + highest index with z[i] != 0 (0 if all zero); out preset to 0
    unsigned long long mine = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        if (z[i] != 0) mine = i + 1;
    mine = warp_max_u64(mine);
    if ((threadIdx.x & 31) == 0 && mine) atomicMax(out, mine);
}

size_t lin_top_nonzero(const uint32_t* z, size_t n, cudaStream_t s)
{
    if (n == 0) return 0;
    DevBuf<unsigned long long> d(1, s);
    PIC_CUDA(cudaMemsetAsync(d.get(), 0, sizeof(unsigned long long), s));
    top_nonzero_kernel<<<grid_for(n, 256), 256, 0, s>>>(z, n, d.get());
    PIC_CHECK_LAUNCH();
    count_launch();
    uint32_t h[2];
    read_words(h, (const uint32_t*)d.get(), 2, s);
    return (size_t)h[0] | ((size_t)h[1] << 32);
}

// Highest magnitude position where the two windows differ (atomicMax over
// mag - lo + 1, zero before and after); the last CTA compares the words there:
// *order = 1, 0 or -1 as |a| >, =, < |b|, posted too.
__global__ void __launch_bounds__(256) ucmp_kernel(WordView a, WordView b, int64_t lo, int64_t hi,
                                                   unsigned long long* diff, uint32_t* ticket, int* order,
                                                   MailRef mail)
{
    const int64_t n = hi - lo;
    unsigned long long mine = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t mag = lo + i;
        if (word_at(a.T, a.exp, a.L, mag) != word_at(b.T, b.exp, b.L, mag)) mine = (unsigned long long)(i + 1);
    }
    mine = warp_max_u64(mine);
    if ((threadIdx.x & 31) == 0 && mine) atomicMax(diff, mine);
    if (!last_cta(ticket, gridDim.x)) return;
    if (threadIdx.x == 0) {
        const unsigned long long r = __ldcg(diff);
        int c = 0;
        if (r) {
            const int64_t mag = lo + (int64_t)r - 1;
            c = word_at(a.T, a.exp, a.L, mag) < word_at(b.T, b.exp, b.L, mag) ? -1 : 1;
        }
        *diff = 0;
        *order = c;
        mail_post(mail, 0, (uint32_t)(c + 1));
    }
}

// The comparison's launch on the library's stream (magnitudes equal).
static void ucmp_launch(const WordView& a, const WordView& b, MailRef mail)
{
    const int64_t lo = a.exp < b.exp ? a.exp : b.exp, hi = a.exp + a.L;
    ucmp_kernel<<<grid_for((size_t)(hi - lo), 256), 256, 0, ctx().stream>>>(a, b, lo, hi, scratch_diff(),
                                                                           scratch_ticket(), scratch_order(), mail);
    PIC_CHECK_LAUNCH();
    count_launch();
}

int lin_ucmp(const WordView& a, const WordView& b, cudaStream_t)
{
    // BigFloat::ucmp, BigFloat.cpp:123-147
    if (const int c = lin_mag_order(a, b)) return c;
    if (a.exp + a.L <= (a.exp < b.exp ? a.exp : b.exp)) return 0;
    Mail mail(ctx().stream);
    {
        std::lock_guard<std::recursive_mutex> pair(ctx().lock);
        ucmp_launch(a, b, mail.ref());
    }
    uint32_t c;
    mail.wait(&c);
    return (int)c - 1;
}

size_t lin_diff(uint32_t* z, size_t TL, const WordView& a, const WordView& b, int64_t bot, int* order)
{
    const bool ask = *order == 0;
    if (TL == 0) {
        if (ask) *order = -1;
        return 0;
    }
    const int64_t reach = a.exp + a.L > b.exp + b.L ? a.exp + a.L : b.exp + b.L;
    if (TL <= kOneWords && bot + (int64_t)TL >= reach) {  // the comparison sees no word above the window
        OneArgs A = *order >= 0 ? one_args(z, TL, a, b, bot, kLinSub) : one_args(z, TL, b, a, bot, kLinSub);
        A.ask = ask ? 1 : 0;
        uint32_t greater;
        const uint64_t nz = lin_one(A, &greater);
        if (ask) *order = greater ? 1 : -1;
        return (size_t)nz;
    }
    Mail mail(ctx().stream);
    LinEnd E{};
    E.kind = kLinSub;
    E.order = ask ? scratch_order() : nullptr;
    E.diff = scratch_diff();
    E.ticket = scratch_ticket();
    E.mail = mail.ref();
    {
        // another thread's comparison may not come between this one and its use
        std::lock_guard<std::recursive_mutex> pair(ctx().lock);
        if (ask) ucmp_launch(a, b, MailRef{});
        addsub(z, TL, *order >= 0 ? a : b, *order >= 0 ? b : a, bot, E, ctx().stream);
    }
    uint32_t greater;
    const uint64_t nz = mail.wait(&greater);
    if (ask) *order = greater ? 1 : -1;
    return (size_t)nz;
}

}  // namespace pic
