/* Host restatement of the FP64 form's CRT (crt3d in crt56.cuh): residues given by
 * any representatives up to 15.75 p in magnitude, scaled by N^-1, Garner's steps
 * with the first two digits taken at or below zero, and the sum assembled as
 * base-2^56 digits with signed parts; checked against the coefficient itself for
 * random ones and the smallest and largest, with and without the offset 2^140.
 * Built with -ffp-contract=off.  Usage: crt56_check COUNT; prints "bad=N". */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

typedef unsigned __int128 u128;
static const double C = 6755399441055744.0;
static const uint64_t P[3] = {140496970186753ull, 140458315481089ull, 140449725546497ull};

static uint64_t mulmod(uint64_t a, uint64_t b, uint64_t p) { return (uint64_t)((u128)a * b % p); }
static uint64_t powmod(uint64_t a, uint64_t e, uint64_t p)
{
    uint64_t r = 1;
    for (a %= p; e; e >>= 1, a = mulmod(a, a, p))
        if (e & 1) r = mulmod(r, a, p);
    return r;
}
static double dmul_tw(double y, double w, double wp, double p)
{
    double q = fma(y, wp, C) - C, h = y * w, l = fma(y, w, -h);
    return fma(-q, p, h) + l;
}
static int64_t to_i64(double x)
{
    union { double d; int64_t i; } u;
    u.d = x + C;
    return u.i - 0x4338000000000000ll;
}
static uint64_t st = 88172645463325252ull;
static uint64_t rnd(void)
{
    st ^= st << 13;
    st ^= st >> 7;
    st ^= st << 17;
    return st;
}
/* x = xh 2^112 + xl, xl < 2^112 */
static uint64_t mod3(u128 xl, uint64_t xh, uint64_t p)
{
    return (uint64_t)((xl % p + (u128)mulmod(xh % p, powmod(2, 112, p), p)) % p);
}

int main(int argc, char** argv)
{
    const long count = argc > 1 ? atol(argv[1]) : 100000;
    const uint64_t m56 = ((uint64_t)1 << 56) - 1;
    const uint64_t c0 = P[0] >> 32, c1 = P[1] >> 32, c01 = c0 + c1, cc = c0 * c1;
    const uint64_t i01 = powmod(P[0], P[1] - 2, P[1]), i012 = powmod(mulmod(P[0] % P[2], P[1] % P[2], P[2]), P[2] - 2, P[2]);
    const uint64_t q012 = powmod(P[1], P[2] - 2, P[2]);
    long bad = 0;
    for (long it = 0; it < count; it++) {
        const int off = it & 1, k = 4 + (int)(rnd() % 24);
        /* the value the digits must give: below 2^140, or 2^140 +- 2^139 */
        u128 xl = ((u128)rnd() << 64 | rnd()) & (((u128)1 << 112) - 1);
        uint64_t xh = rnd() & ((1u << 28) - 1);
        if (it % 7 == 0) xl = rnd() % 4, xh = 0;
        if (it % 7 == 1) xl = (((u128)1 << 112) - 1) - rnd() % 4, xh = (1u << 28) - 1;
        if (it % 7 == 2) xl %= P[0] + 5, xh = 0;
        if (off) xh = (1u << 28) - (1u << 27) + (xh >> ((it & 2) ? 1 : 0)); /* 2^139 .. 1.5 2^140 */
        double y[3];
        for (int q = 0; q < 3; q++) {
            const uint64_t p = P[q], N = powmod(2, k, p), o = off ? powmod(2, 140, p) : 0;
            const uint64_t r = mulmod((mod3(xl, xh, p) + p - o) % p, N, p);
            const int s = (int)(rnd() % 31) - 15; /* representative r + s p, |.| <= 15.75 p */
            y[q] = (double)((int64_t)r + (int64_t)s * (int64_t)p);
            if (fabs(y[q]) > 15.75 * (double)p) y[q] = (double)(int64_t)r;
        }
        double r[3];
        for (int q = 0; q < 3; q++) {
            const double p = (double)P[q], sw = (double)powmod(powmod(2, k, P[q]), P[q] - 2, P[q]);
            double o = off ? (double)powmod(2, 140, P[q]) : 0.0;
            if (q == 0) o -= 2 * p;
            r[q] = dmul_tw(y[q], sw, sw / p, p) + o;
        }
        const double p1 = (double)P[1], p2 = (double)P[2];
        const double v1 = dmul_tw(r[1] - r[0], (double)i01, (double)i01 / p1, p1) - p1;
        const double a = dmul_tw(r[2] - r[0], (double)i012, (double)i012 / p2, p2);
        const double b = dmul_tw(v1, (double)q012, (double)q012 / p2, p2);
        const double s = a - b, qq = fma(s, 1.0 / p2, C) - C;
        double v2 = fma(-qq, p2, s);
        v2 = v2 < 0 ? v2 + p2 : v2;
        const int64_t V1 = to_i64(v1), V2 = to_i64(v2), A = to_i64(r[0]) + V1 + V2;
        const __int128 Bx = (__int128)V1 * (int64_t)c0 + (__int128)V2 * (int64_t)c01;
        const int64_t B = (int64_t)Bx;
        if (Bx != B) bad++;
        const uint64_t lo = (uint64_t)(uint32_t)V2 * cc, hi = (uint64_t)(V2 >> 32) * cc + (lo >> 32);
        const uint64_t D = (hi << 32) | (uint32_t)lo;
        const int64_t t0 = A + (int64_t)(((uint64_t)B & 0xffffffu) << 32);
        const int64_t t1 = (t0 >> 56) + (B >> 24) + (int64_t)((D << 8) & m56);
        const uint64_t d0 = (uint64_t)t0 & m56, d1 = (uint64_t)t1 & m56;
        const uint32_t d2 = (uint32_t)((t1 >> 56) + (int64_t)(hi >> 16));
        if (d0 != ((uint64_t)xl & m56) || d1 != ((uint64_t)(xl >> 56) & m56) || d2 != xh) bad++;
    }
    printf("bad=%ld\n", bad);
    return bad != 0;
}
