/*
 * Test helper: the quantization forms of the 3-D compressor's row kernel
 * (sz3_quantize_f with its test, sz3_quantize_any and sz3_quantize_wide,
 * zccl_gb300/csrc/zk_szp3d.cu) restated in C with IEEE float operations and
 * fmaf, against (int)floor((double)x * inv + 0.5) (ZCCL_float.h:57-61) for
 * bounds of all kinds and values around multiples and middles of the step, up
 * to 2^25 steps.  Prints, for the three forms, mismatches and values taken, and
 * all values; built and run by tests/test_szp3d_large.py with
 * -ffp-contract=off.
 */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

static uint64_t state = 88172645463325252ull;
static uint64_t rnd(void)
{
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    return state;
}
static double uni(void) { return (double)(rnd() >> 11) * 0x1p-53; }

#define MAGIC 12582912.0f
#define SURE 0.499999761581420898f

static long bad[3], taken[3], all;

static void check(float x, double inv)
{
    const float hi = (float)inv, lo = (float)(inv - (double)hi);
    const double v = floor((double)x * inv + 0.5);
    if (!(fabs(v) < 0x1p25)) return;
    all++;
    { /* the float form and its second form */
        const float n = fmaf(x, hi, MAGIC) - MAGIC, d = fmaf(x, lo, fmaf(x, hi, -n));
        if (fabsf(n) < 4194304.0f && fabsf(d) < SURE) {
            taken[0]++;
            bad[0] += (double)n != v;
        }
        const float c = (d + MAGIC) - MAGIC;
        if (fabsf(n) < 4194304.0f && fabsf(d - c) < SURE) {
            taken[1]++;
            bad[1] += (double)(n + c) != v;
        }
        if (fabsf(n) < 4194304.0f && fabs(v) > 0x1p22) bad[1]++;
    }
    {
        const float p = x * hi, n = rintf(p), d = fmaf(x, lo, fmaf(x, hi, -n)), c = (d + MAGIC) - MAGIC;
        if (fabsf(p) < 16777200.0f && fabsf(d - c) < SURE) {
            taken[2]++;
            bad[2] += (double)(n + c) != v;
        }
    }
}

int main(int argc, char **argv)
{
    const long rounds = argc > 1 ? atol(argv[1]) : 100000;
    for (long r = 0; r < rounds; r++) {
        double inv = exp2(uni() * 80 - 40) * (1 + uni());
        if (r % 4 == 1) inv = (double)(float)inv;               /* a float */
        if (r % 4 == 2) inv = 0.5 / (double)(float)(0.5 / inv); /* of a bound that is one */
        if (r % 16 == 3) inv = exp2(rint(uni() * 80 - 40));
        for (int k = 0; k < 40; k++) {
            const double q = rint(exp2(uni() * 25)) * (k & 1 ? -1 : 1);
            const double f = k % 4 == 0 ? 0.5 : k % 4 == 1 ? 0.0 : k % 4 == 2 ? 0.5 + (uni() - 0.5) * 1e-5 : uni();
            float x = (float)((q + f) / inv);
            check(x, inv);
            check(nextafterf(x, INFINITY), inv);
            check(nextafterf(x, -INFINITY), inv);
        }
    }
    printf("%ld %ld %ld %ld %ld %ld %ld\n", bad[0], taken[0], bad[1], taken[1], bad[2], taken[2], all);
    return 0;
}
