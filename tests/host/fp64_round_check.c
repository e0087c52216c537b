/* Host restatement of the FP64 form's forward register rounds (radix 2 .. 16:
 * dmul_w's product with the quotient from fl(y w), and the reductions of the
 * last level that reduce_sum / reduce_unit name), run beside 128-bit integer
 * arithmetic from the largest inputs a round may get: 2 p in magnitude for
 * radix 2 .. 8, p for radix 16.  Every value inside must stay below 2^51, every
 * output within the round's input range and congruent to the exact butterflies.
 * Built with -ffp-contract=off.  Usage: fp64_round_check B COUNT; prints
 * "bad=N" and exits nonzero on any failure. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

static const double C = 6755399441055744.0; /* 1.5 * 2^52 */

static double dmul_w(double y, double w, double p, double pinv)
{
    double h = y * w;
    double l = fma(y, w, -h);
    double q = fma(h, pinv, C) - C;
    return fma(-q, p, h) + l;
}

static double dreduce(double s, double p, double pinv)
{
    double q = fma(s, pinv, C) - C;
    return fma(-q, p, s);
}

static uint64_t st = 88172645463325252ull;
static uint64_t rnd(void)
{
    st ^= st << 13;
    st ^= st >> 7;
    st ^= st << 17;
    return st;
}

static int64_t mod(__int128 v, int64_t p)
{
    __int128 m = v % p;
    return (int64_t)(m < 0 ? m + p : m);
}

int main(int argc, char** argv)
{
    const int B = argc > 1 ? atoi(argv[1]) : 3;
    const long count = argc > 2 ? atol(argv[2]) : 100000;
    const int64_t primes[3] = {140496970186753ll, 140458315481089ll, 140449725546497ll};
    const double lim51 = 2251799813685248.0;
    long bad = 0;
    for (long it = 0; it < count; it++) {
        const int64_t p = primes[it % 3];
        const double pd = (double)p, pinv = 1.0 / pd;
        const int64_t X = B == 4 ? p : 2 * p;
        const int unit = (it >> 2) & 1; /* the smallest stride: unit twiddles at the last level */
        double x[16];
        int64_t e[16];
        for (int m = 0; m < (1 << B); m++) {
            int64_t v;
            switch (rnd() & 3) {
            case 0: v = X - (int64_t)(rnd() & 3); break;
            case 1: v = -X + (int64_t)(rnd() & 3); break;
            default: v = (int64_t)(rnd() % (2 * (uint64_t)X + 1)) - X; break;
            }
            if (it & 8) v = (it & 16) ? X : -X; /* every sum at its largest */
            x[m] = (double)v;
            e[m] = mod(v, p);
        }
        for (int l = 0; l < B; l++) {
            const int hm = 1 << (B - 1 - l), last = l == B - 1;
            for (int m = 0; m < (1 << B); m++) {
                if (m & hm) continue;
                const int red = last && (B == 4 || (m & 3) == 0);
                const double s = x[m] + x[m + hm], d = x[m] - x[m + hm];
                const int64_t w = (rnd() & 1) ? (int64_t)(rnd() % (uint64_t)p) : p - 1 - (int64_t)(rnd() & 3);
                const __int128 es = (__int128)e[m] + e[m + hm], ed = (__int128)e[m] - e[m + hm];
                if (fabs(s) >= lim51 || fabs(d) >= lim51) bad++;
                x[m] = red ? dreduce(s, pd, pinv) : s;
                e[m] = mod(es, p);
                if (last && unit) {
                    x[m + hm] = red ? dreduce(d, pd, pinv) : d;
                    e[m + hm] = mod(ed, p);
                } else {
                    x[m + hm] = dmul_w(d, (double)w, pd, pinv);
                    e[m + hm] = mod((__int128)mod(ed, p) * w, p);
                    if (fabs(x[m + hm]) > pd) bad++;
                }
            }
        }
        for (int m = 0; m < (1 << B); m++)
            if (x[m] != floor(x[m]) || fabs(x[m]) > (double)X || mod((__int128)(int64_t)x[m], p) != e[m]) bad++;
    }
    printf("bad=%ld\n", bad);
    return bad != 0;
}
