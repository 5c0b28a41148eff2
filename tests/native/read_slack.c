/*
 * Test helper: how far past a block's last byte its decoders read (the
 * addresses of decode_octet, decode_small_f, decode_mid_f and decode_add_any,
 * zdev.cuh, restated) against the slack the buffers have (zg_octet_slack,
 * zg_lane_slack), for every block length, width and element count.  Prints
 * blocks checked and reads beyond the slack; built and run by
 * tests/test_read_slack.py.
 */
#include <stdio.h>

#include "zgeom.h"

static uint32_t far_; /* one past the last byte read */
static void words(uint32_t a, uint32_t n) /* n words from the one that holds byte a on */
{
    const uint32_t e = (a & ~3u) + 4u * n;
    if (e > far_) far_ = e;
}

static void octet(uint32_t o, uint32_t b, uint32_t n, uint32_t g, uint32_t fmt)
{
    uint32_t B, r;
    if (b)
        zg_split(fmt, b, &B, &r);
    else
        B = r = 0;
    const uint32_t gr = 8u * g < n ? g : 0u, hb = o + 1u + (n + 7u) / 8u;
    words(o + 1u + gr, 1);
    words(hb + B * n + gr * r, 3);
    if (B <= 1)
        words(hb + 8u * gr, 3);
    else if (B == 2)
        words(hb + 16u * gr, 5);
    else
        words(hb + (8u * gr + 7u) * B, 2);
}

static void lane(uint32_t o, uint32_t b, uint32_t n, int any)
{
    const uint32_t B = b >> 3, r = b & 7u, hb = o + 1u + (n + 7u) / 8u, lb = hb + n * B;
    words(o + 1u, 3);
    words(lb + 3u * r, 3);
    if (any)
        words(hb + 31u * B, 2);
    else if (b < 16)
        words(hb, 9);
    else
        words(hb, 17);
}

int main(void)
{
    long checked = 0, over = 0;
    for (uint32_t L = 1; L <= ZG_MAX_L; L++)
        for (uint32_t fmt = 0; fmt < 2; fmt++)
            for (uint32_t n = 0; n <= L; n++)
                for (uint32_t b = 0; b <= (n ? 32u : 0u); b++)
                    for (uint32_t o = 0; o < 4; o++) {
                        const uint32_t end = o + zg_block_bytes_f(fmt, b, n);
                        far_ = 0;
                        for (uint32_t g = 0; g < (L + 7u) / 8u; g++) octet(o, b, n, g, fmt);
                        checked++;
                        over += far_ > end + zg_octet_slack(L);
                        if (L != 32 || fmt) continue;
                        for (int any = 0; any < 2; any++) {
                            if (!any && b > 23) continue;
                            far_ = 0;
                            lane(o, b, n, any);
                            over += far_ > end + (n == 32 && b < 16 && !any ? zg_octet_slack(L) : zg_lane_slack());
                        }
                    }
    printf("%ld %ld\n", checked, over);
    return 0;
}
