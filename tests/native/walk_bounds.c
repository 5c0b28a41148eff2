/*
 * Test helper: the header walk's windows and groups of them (zgeom.h:
 * walk_chunk, walk_windows) for headers with valid, alternating, random and
 * damaged chunk offsets, against the scratch that is sized for them
 * (walk_max_windows, walk_max_groups).  Prints headers checked, headers whose
 * windows or groups exceed the scratch, and valid headers that were refused;
 * built and run by tests/test_walk_bounds.py.
 */
#include <stdio.h>
#include <stdlib.h>

#include "zgeom.h"

static uint64_t rng_state = 88172645463325252ull;
static uint64_t rnd(uint64_t below)
{
    rng_state ^= rng_state << 13;
    rng_state ^= rng_state >> 7;
    rng_state ^= rng_state << 17;
    return below ? rng_state % below : 0;
}

static long checked, over, refused;

static void header(const ZGeom *g, const uint64_t *rel, uint64_t avail, int valid)
{
    const uint32_t G = walk_group(zg_block_bytes(32, g->L));
    uint64_t nwin = 0, ngrp = 0;
    uint32_t bad = 0;
    for (uint32_t s = 0; s < g->T; s++) {
        uint64_t P, R;
        const uint32_t e = walk_chunk(g, s, rel[s], s + 1 < g->T ? rel[s + 1] : 0, avail, zg_stream_worst(g), &P, &R);
        bad |= e;
        if (e || !g->nb_reg) continue;
        nwin += walk_windows(P, R);
        ngrp += (walk_windows(P, R) + G - 1) / G;
    }
    checked++;
    over += nwin > walk_max_windows(g) || ngrp > walk_max_groups(g);
    refused += valid && bad;
}

int main(void)
{
    static uint64_t rel[4096];
    const uint32_t Ls[] = {1, 8, 32, 36, 100, 256}, Ts[] = {1, 2, 3, 16, 72, 1000};
    const uint64_t ns[] = {4096, 70001, 1000003, 1ull << 24, 1ull << 33};
    for (int a = 0; a < 6; a++)
        for (int b = 0; b < 6; b++)
            for (int c = 0; c < 5; c++) {
                ZGeom g;
                if (zg_init(&g, ns[c], Ls[a], Ts[b])) continue;
                const uint64_t worst = zg_stream_worst(&g), seg = zg_seg_worst(g.tbs, g.L), body = worst - 8ull * g.T;
                const uint64_t least = 4 + g.nb_reg; /* a chunk of zero-width blocks */
                for (int kind = 0; kind < 40; kind++) {
                    uint64_t at = 0;
                    for (uint32_t s = 0; s < g.T; s++) {
                        rel[s] = kind == 0 ? s * seg                                  /* every chunk at its largest */
                                 : kind == 1 ? s * least                              /* and smallest */
                                 : kind < 10 ? at                                     /* anything between */
                                 : kind == 10 ? (s & 1 ? body : 0)                    /* alternating: each chunk the whole stream */
                                 : kind == 11 ? (s & 1 ? body / 2 : 0)
                                 : kind == 12 ? (s & 1 ? seg + 1 : 0)
                                 : kind == 13 ? (s % 3 == 2 ? body : 0)
                                 : kind < 25 ? rnd(body + 1)
                                 : kind < 30 ? rnd(~0ull)
                                             : (s && rnd(4) == 0 ? rnd(body + 1) : at);
                        at += least + rnd(seg - least + 1);
                    }
                    header(&g, rel, worst, kind < 10);
                    header(&g, rel, worst + rnd(1 << 20), kind < 10);
                    header(&g, rel, rnd(worst), 0);
                    header(&g, rel, ~0ull >> 8, kind < 10);
                }
            }
    printf("%ld %ld %ld\n", checked, over, refused);
    return 0;
}
