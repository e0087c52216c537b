/* The FP64 form's short column passes into the rows and out of them, run from the
 * repository's own device templates (cols.cuh, middle.cuh, passes.cuh,
 * fp64mod.cuh through cuda_shim) beside 128-bit integer arithmetic.
 *
 * Forward: pieces at their largest residues, with column signs that reinforce
 * each other, through a pass of LC rows, then the first radix-8 round of a row.
 * A row accepts |x| <= 2 p.  Inverse: the largest values a row may leave, 15.75 p,
 * through the pass of LC rows: |y| <= 15 p with p for each level still to come.
 * Every value an integer and congruent, every quotient in the rounding constant's
 * range.  Usage: fp64_columns_check COUNT; prints "bad=N" and exits nonzero on any
 * failure. */
#include <stdio.h>
#include <stdlib.h>

#include "cols.cuh"

using namespace pic;

static long bad;
static uint64_t st = 88172645463325252ull;
static uint64_t rnd()
{
    st ^= st << 13;
    st ^= st >> 7;
    st ^= st << 17;
    return st;
}
static int64_t mod(__int128 v, int64_t p)
{
    const __int128 m = v % p;
    return (int64_t)(m < 0 ? m + p : m);
}
static void check(double x, int64_t e, double limit, int64_t p)
{
    if (x != floor(x) || !(fabs(x) <= limit) || mod((__int128)(int64_t)x, p) != e) bad++;
}

/* The butterflies of one group, exactly: twiddle of level l, butterfly u. */
template <int B, class Tw>
static void exact(int64_t (&e)[1 << B], bool inv, int64_t p, const Tw& tw)
{
    for (int s = 0; s < B; s++) {
        const int l = inv ? B - 1 - s : s, hm = 1 << (B - 1 - l);
        for (int m = 0; m < (1 << B); m++) {
            if (m & hm) continue;
            const __int128 a = e[m], b = e[m + hm], w = tw(l, m & (hm - 1));
            if (inv) {
                const __int128 t = b * w % p;
                e[m] = mod(a + t, p);
                e[m + hm] = mod(a - t, p);
            } else {
                e[m] = mod(a + b, p);
                e[m + hm] = mod((__int128)mod(a - b, p) * w, p);
            }
        }
    }
}

/* Random twiddles of one group; u = 0 of the smallest stride is 1. */
template <int B, int LST>
static void twiddles(GroupTw<B, LST>& t, int64_t p)
{
    for (int l = 0; l < B; l++)
        for (int u = 0; u < (1 << (B - 1 - l)); u++)
            t.w[(1 << B) - (1 << (B - l)) + u] = LST == 0 && u == 0 ? 1.0 : (double)(rnd() % (uint64_t)p);
}

template <int LC>
static void run(long count)
{
    constexpr int BL = LC < 3 ? LC : 3, E = 1 << BL;
    const int64_t primes[3] = {140496970186753ll, 140458315481089ll, 140449725546497ll};
    for (long it = 0; it < count; it++) {
        const int64_t p = primes[it % 3];
        const Dbl::Ctx L{(double)p, 1.0 / (double)p};
        GroupTw<BL, 0> tail;
        twiddles(tail, p);
        auto tw = [&](int l, int u) { return (int64_t)tail.at(l, u); };
        ColTwiddle<false, LC> F;
        ColTwiddle<true, LC> I;
        double fx[E][8];
        int64_t fe[E][8];
        const int64_t wg = LC > 3 ? (int64_t)(rnd() % (uint64_t)p) : 1;
        const unsigned signs = (unsigned)rnd();
        for (int c = 0; c < 8; c++) {  /* eight columns meet in a row's first round */
            double x[E];
            int64_t e[E];
            const int s = it & 1 ? (int)(signs >> c) & 1 : (__builtin_popcount((unsigned)c & (signs & 7)) & 1);
            for (int i = 0; i < E; i++) {
                uint64_t v = rnd() >> 8;  /* a 56-bit piece */
                if (it & 6) {
                    const int64_t m = 1 + (int64_t)(rnd() % 511), h = (p - 1) / 2 - (1ll << 31) - (int64_t)(rnd() & 255);
                    v = (uint64_t)(m * p + (s ? -h : h));
                }
                x[i] = dpiece56(v, L.p, L.pinv);
                e[i] = (int64_t)(v % (uint64_t)p);
                if (LC > 3) {  /* rounds before this one: up to 2 p */
                    const int64_t h = 2 * p - (int64_t)(rnd() & 255);
                    x[i] = (double)(s ? -h : h);
                    e[i] = mod(s ? -h : h, p);
                }
            }
            F.q[1] = (double)(rnd() % (uint64_t)p);
            F.powers(L);
            F.forward_tail(x, tail, (double)wg, L);
            exact<BL>(e, false, p, tw);
            for (int i = 0; i < E; i++) {
                const int r = brev3(i, BL);
                e[i] = mod((__int128)mod((__int128)e[i] * wg, p) * (r ? mod((__int128)(int64_t)F.q[r], p) : 1), p);
                check(x[i], e[i], 2 * L.p, p);
                fx[i][c] = x[i];
                fe[i][c] = e[i];
            }
        }
        GroupTw<3, 8> row;
        twiddles(row, p);
        for (int i = 0; i < E; i++) {
            fwd_group<3, 8>(fx[i], row, L);
            exact<3>(fe[i], false, p, [&](int l, int u) { return (int64_t)row.at(l, u); });
            for (int m = 0; m < 8; m++) check(fx[i][m], fe[i][m], 2 * L.p, p);
        }
        double y[E];
        int64_t e[E];
        for (int i = 0; i < E; i++) {
            int64_t v = 63 * p / 4 - (int64_t)(rnd() & 255);
            if ((signs >> i) & 1) v = -v;
            if ((it & 6) == 0) v = (int64_t)(rnd() % (31 * (uint64_t)p)) - 31 * p / 2;
            y[i] = (double)v;
            e[i] = mod(v, p);
        }
        I.q[1] = (double)(rnd() % (uint64_t)p);
        I.powers(L);
        for (int i = 0; i < E; i++) {
            const int r = brev3(i, BL);
            e[i] = mod((__int128)mod((__int128)e[i] * wg, p) * (r ? mod((__int128)(int64_t)I.q[r], p) : 1), p);
        }
        I.inverse_head(y, tail, (double)wg, L);
        exact<BL>(e, true, p, tw);
        for (int i = 0; i < E; i++) check(y[i], e[i], (15 - (LC > 3 ? LC - 3 : 0)) * L.p, p);
    }
}

int main(int argc, char** argv)
{
    const long count = argc > 1 ? atol(argv[1]) : 10000;
    run<1>(count);
    run<2>(count);
    run<3>(count);
    run<4>(count);
    run<10>(count);
    run<11>(count);
    bad += shim_bad;
    printf("bad=%ld\n", bad);
    return bad != 0;
}
