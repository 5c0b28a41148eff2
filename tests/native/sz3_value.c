/*
 * Test helper: sz3_value (zccl_gb300/csrc/zk_szp3d.cu) restated in C with IEEE
 * float operations and fmaf, checked against (float)((double)q * twice)
 * (ZCCLd_float.c:2857) for random bounds, for bounds with few bits (whose
 * products meet exact ties and powers of two), and for integers of every
 * magnitude.  Prints mismatches, checks, and how many integers below 2^24 took the double steps;
 * built and run by tests/test_szp3d_sums.py with -ffp-contract=off.
 */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static uint32_t u_of(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }

static long slow;

static float value(int32_t q, double d, float thi, float tlo)
{
    const float qf = (float)q;
    if (d >= 0x1p-60 && d <= 0x1p60 && fabsf(qf) < 16777216.0f) {
        const float hi = qf * thi;
        const float lo = fmaf(qf, tlo, fmaf(qf, thi, -hi));
        const float r = hi + lo;
        const float e = lo - (r - hi);
        if (fmaf(e, 1.00000762939453125f, r) == r) return r;
        slow++;
    }
    return (float)((double)q * d);
}

static uint64_t st = 0x9E3779B97F4A7C15ull;
static uint64_t rnd(void)
{
    st ^= st << 13;
    st ^= st >> 7;
    st ^= st << 17;
    return st;
}

int main(int argc, char **argv)
{
    const long rounds = argc > 1 ? atol(argv[1]) : 20000;
    long bad = 0, checks = 0;
    for (long it = 0; it < rounds; it++) {
        double d = ldexp(1.0 + (double)(rnd() >> 12) * 0x1p-52, (int)(rnd() % 100) - 50);
        if (it % 3 == 1) d = (double)(float)d;                          /* a float, as most bounds are */
        if (it % 3 == 2) d = ldexp((double)(rnd() % 65536 + 1), (int)(rnd() % 40) - 30); /* few bits */
        if (it % 50 == 7) d = ldexp(1.0, (int)(rnd() % 160) - 80);
        const float hi = (float)d, lo = (float)(d - (double)hi);
        for (int k = 0; k < 250; k++) {
            int32_t q = (int32_t)rnd() >> (int)(rnd() % 32);
            if (k % 5 == 0) { /* next to a tie of the product */
                const double t = ldexp((double)((rnd() % 16777216) + 16777216) + 0.5, (int)(rnd() % 20) - 30);
                const double z = nearbyint(t / d);
                if (fabs(z) < 2147483647.0) q = (int32_t)z;
            }
            checks++;
            if (u_of(value(q, d, hi, lo)) != u_of((float)((double)q * d))) bad++;
        }
    }
    printf("%ld %ld %ld\n", bad, checks, slow);
    return bad != 0;
}
