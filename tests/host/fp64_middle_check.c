/* Host restatement of the FP64 form's last forward round, pointwise product and
 * first inverse round of 2^LR rows, whose unit twiddles take no product: from
 * the largest inputs (2 p) every value stays below 2^51, a product of a raw and a
 * reduced factor below 0.75 p, and a sum of TERMS of them, after the inverse
 * round and p for each level after it, below 15.75 p; all congruent to exact
 * arithmetic.  Built with -ffp-contract=off.  Usage: fp64_middle_check LR TERMS
 * COUNT; prints "bad=N" and exits nonzero on any failure. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

static const double C = 6755399441055744.0; /* 1.5 * 2^52 */
static long bad;
static double pd, pinv;

static double dmul(double a, double b)
{
    double h = a * b, l = fma(a, b, -h), q = fma(h, pinv, C) - C;
    return fma(-q, pd, h) + l;
}
static double dred(double s) { return fma(-(fma(s, pinv, C) - C), pd, s); }

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
static double in51(double x)
{
    if (fabs(x) >= 2251799813685248.0) bad++;
    return x;
}

int main(int argc, char** argv)
{
    const int LR = atoi(argv[1]), terms = atoi(argv[2]), B = LR % 3 ? LR % 3 : 3;
    const long count = atol(argv[3]);
    const int64_t primes[3] = {140496970186753ll, 140458315481089ll, 140449725546497ll};
    const int head = B > 1 && 4 * 0.75 * terms + (LR - 2) <= 15.75;
    for (long it = 0; it < count; it++) {
        const int64_t p = primes[it % 3];
        pd = (double)p;
        pinv = 1.0 / pd;
        int64_t w[7], es[8] = {0};
        double sum[8] = {0};
        for (int i = 0; i < 7; i++) w[i] = (rnd() & 1) ? (int64_t)(rnd() % (uint64_t)p) : p - 1 - (int64_t)(rnd() & 3);
        for (int t = 0; t < terms; t++) {
            double f[2][8];
            int64_t e[2][8];
            for (int a = 0; a < 2; a++) {
                for (int m = 0; m < (1 << B); m++) {
                    int64_t v = (int64_t)(rnd() % (4 * (uint64_t)p + 1)) - 2 * p;
                    if (it & 8) v = (it & 16) ? 2 * p : ((m * 5 + t) & 2 ? -2 * p : 2 * p);
                    f[a][m] = (double)v;
                    e[a][m] = mod(v, p);
                }
                for (int l = 0; l < B; l++)
                    for (int m = 0, hm = 1 << (B - 1 - l); m < (1 << B); m++) {
                        if (m & hm) continue;
                        const int u = m & (hm - 1);
                        const double s = in51(f[a][m] + f[a][m + hm]), d = in51(f[a][m] - f[a][m + hm]);
                        const int64_t x = mod((__int128)e[a][m] + e[a][m + hm], p);
                        const int64_t y = mod((__int128)e[a][m] - e[a][m + hm], p);
                        f[a][m] = s;
                        f[a][m + hm] = u ? dmul(d, (double)w[hm - 1 + u]) : d;
                        e[a][m] = x;
                        e[a][m + hm] = u ? mod((__int128)y * w[hm - 1 + u], p) : y;
                    }
            }
            for (int m = 0; m < (1 << B); m++) {
                const double x = dmul(f[0][m], dred(f[1][m]));
                if (fabs(x) > 0.75 * pd) bad++;
                sum[m] += x;
                es[m] = mod((__int128)e[0][m] * e[1][m] + es[m], p);
            }
        }
        for (int l = B - 1; l >= 0; l--)
            for (int m = 0, hm = 1 << (B - 1 - l); m < (1 << B); m++) {
                if (m & hm) continue;
                const int u = m & (hm - 1);
                const int unit = head ? u == 0 && !(B == 3 && l == 0) : l == B - 1;
                const int64_t t = u ? w[hm - 1 + u] : 1;
                const double b = unit ? sum[m + hm] : dmul(in51(sum[m + hm]), (double)t);
                const int64_t eb = mod((__int128)es[m + hm] * t, p), ea = es[m];
                sum[m + hm] = sum[m] - b;
                sum[m] = sum[m] + b;
                es[m] = mod((__int128)ea + eb, p);
                es[m + hm] = mod((__int128)ea - eb, p);
            }
        for (int m = 0; m < (1 << B); m++)
            if (sum[m] != floor(sum[m]) || mod((__int128)(int64_t)sum[m], p) != es[m] ||
                fabs(sum[m]) + (LR - B) * pd > 15.75 * pd)
                bad++;
    }
    printf("bad=%ld\n", bad);
    return bad != 0;
}
