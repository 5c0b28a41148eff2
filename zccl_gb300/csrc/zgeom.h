/*
 * zgeom.h -- geometry of a fastmode1 stream, shared by host and device code.
 *
 * A stream of N floats written by T OpenMP threads with block size L
 * (ZCCL/src/ZCCL_float.c:532-545, ZCCL/src/ZCCLd_float.c:558-566):
 *
 *   tbs = N / T, rem = N % T
 *   segment s < T : elements [s*tbs, (s+1)*tbs)       -> chunk s
 *   segment T     : elements [T*tbs, N) when rem > 0  -> appended to chunk T-1
 *   a segment of len elements = raw int32 head + ceil((len-1)/L) blocks; all
 *   blocks hold L elements except the last, which holds (len-1) % L when
 *   that is non-zero.
 *
 * On the device a segment is cut into tiles of up to TB consecutive blocks;
 * tile 0 of a segment also owns the segment's head.  Tiles are numbered in
 * stream order, so the byte offset of a tile is the exclusive prefix sum of
 * the byte sizes of all tiles before it.  A tile's blocks are cut into ZG_SUB
 * groups of GB = TB / ZG_SUB blocks, one per warp of a codec CTA; the side
 * index has an entry per group.  Within a warp, G = ceil(L / 8) neighbouring
 * lanes share a block, eight elements each, so 32 / G blocks are worked on
 * at a time.
 */
#ifndef ZCCL_GB300_ZGEOM_H
#define ZCCL_GB300_ZGEOM_H

#include <stdint.h>

#include "zccl_err.h"

#ifdef __CUDACC__
#define ZG_HD __host__ __device__ __forceinline__
#else
#define ZG_HD static inline
#endif

#define ZG_MAX_L 256 /* largest block size the kernels accept */
#define ZG_SUB 8u    /* block groups per tile (compute warps of a codec CTA) */

typedef struct ZGeom {
    uint64_t n;       /* elements */
    uint64_t tbs;     /* elements per regular segment (n / T) */
    uint32_t T;       /* writer thread count = chunks in the header */
    uint32_t L;       /* block size */
    uint32_t rem;     /* n % T: length of the extra segment (0 = none) */
    uint32_t TB;      /* blocks per tile */
    uint64_t nb_reg;  /* blocks per regular segment */
    uint64_t nt_reg;  /* tiles per regular segment */
    uint64_t nb_rm;   /* blocks of the extra segment */
    uint64_t nt_rm;   /* tiles of the extra segment (0 when rem == 0) */
    uint64_t nblocks; /* all blocks */
    uint64_t ntiles;  /* all tiles */
    uint64_t gr_reg;  /* index groups per regular segment (at least 1: the head's) */
    uint64_t ngroups; /* all index groups */
    uint32_t fmt;     /* block magnitude layout: ZG_FASTMODE1 or ZG_FIXED_BYTES */
    uint32_t GB;      /* blocks per index group */
    uint32_t nt_rcp;  /* floor(2^32 / nt_reg) (2^32 - 1 for 1): division of tile numbers */
} ZGeom;

/* Block magnitude layouts.  fastmode1: B = b/8 whole bytes per magnitude
 * (little-endian), then its r = b%8 low bits as an MSB-first stream
 * (ZCCL/src/ZCCL_TypeManager.c:12-91).  The fixed-rate appendix codec keeps
 * whole bytes only, B = b/8 + 1 of them (at most 4), r = 0
 * (ZCCL/src/ZCCL_appendix.c:18-39).  Everything else is shared. */
#define ZG_FASTMODE1 0u
#define ZG_FIXED_BYTES 1u

/* Per-tile view computed from a tile index. */
typedef struct ZTile {
    uint64_t seg_start; /* first element (the head) of the segment */
    uint64_t seg_len;   /* elements of the segment */
    uint64_t blk0;      /* first block of the tile, index within the segment */
    uint64_t gblk0;     /* first block of the tile, index within the stream */
    uint64_t e_first;   /* first element of the first block (head + 1 + blk0*L) */
    uint64_t e_end;     /* one past the last element of the tile's last block */
    uint64_t grp0;      /* first index group of the tile, index within the stream */
    uint32_t seg;       /* segment index (T for the extra segment) */
    uint32_t nblk;      /* blocks in the tile (0 for a segment of length 1) */
    uint32_t has_head;  /* tile 0 of its segment */
} ZTile;

ZG_HD uint64_t zg_div_up(uint64_t a, uint64_t b) { return (a + b - 1) / b; }

ZG_HD uint32_t zg_tile_blocks(uint32_t L)
{
    if (L <= 32) return 256;
    uint32_t k = 4096u / (32u * L);
    return 32u * (k ? k : 1u);
}

/* Bytes of a block of n elements encoded at width b
 * (ZCCL/src/ZCCL_TypeManager.c:24-29 plus header and sign bytes). */
ZG_HD uint32_t zg_block_bytes(uint32_t b, uint32_t n)
{
    if (b == 0) return 1;
    return 1 + (n + 7) / 8 + (b >> 3) * n + ((b & 7) * n + 7) / 8;
}

/* Whole bytes B and low bits r per magnitude of a width-b block in layout fmt. */
ZG_HD void zg_split(uint32_t fmt, uint32_t b, uint32_t *B, uint32_t *r)
{
    if (fmt == ZG_FIXED_BYTES) {
        *B = (b >> 3) + 1 < 4 ? (b >> 3) + 1 : 4;
        *r = 0;
    } else {
        *B = b >> 3;
        *r = b & 7;
    }
}

/* zg_block_bytes in layout fmt; both layouts take the same bytes at width 32. */
ZG_HD uint32_t zg_block_bytes_f(uint32_t fmt, uint32_t b, uint32_t n)
{
    if (b == 0) return 1;
    uint32_t B, r;
    zg_split(fmt, b, &B, &r);
    return 1 + (n + 7) / 8 + B * n + (r * n + 7) / 8;
}

ZG_HD uint64_t zg_seg_blocks(uint64_t len, uint32_t L) { return len ? zg_div_up(len - 1, L) : 0; }

ZG_HD int zg_init(ZGeom *g, uint64_t n, uint32_t L, uint32_t T)
{
    if (T == 0 || L == 0 || L > ZG_MAX_L || n < T) return -1;
    g->n = n;
    g->T = T;
    g->L = L;
    g->fmt = ZG_FASTMODE1;
    g->GB = zg_tile_blocks(L) / ZG_SUB;
    g->tbs = n / T;
    g->rem = (uint32_t)(n % T);
    g->TB = zg_tile_blocks(L);
    g->nb_reg = zg_seg_blocks(g->tbs, L);
    g->nt_reg = g->nb_reg ? zg_div_up(g->nb_reg, g->TB) : 1;
    g->nb_rm = zg_seg_blocks(g->rem, L);
    g->nt_rm = g->rem ? (g->nb_rm ? zg_div_up(g->nb_rm, g->TB) : 1) : 0;
    g->nblocks = (uint64_t)T * g->nb_reg + g->nb_rm;
    g->ntiles = (uint64_t)T * g->nt_reg + g->nt_rm;
    if (g->ntiles >> 32) return -1; /* tile indices are 32-bit on the device */
    g->gr_reg = g->nb_reg ? zg_div_up(g->nb_reg, g->GB) : 1;
    g->ngroups = (uint64_t)T * g->gr_reg + (g->rem ? (g->nb_rm ? zg_div_up(g->nb_rm, g->GB) : 1) : 0);
    g->nt_rcp = g->nt_reg > 1 ? (uint32_t)((1ull << 32) / g->nt_reg) : 0xFFFFFFFFu;
    return 0;
}

/* t / nt_reg for t < 2^32 by the reciprocal: its floor, floor(2^32 / nt_reg)
 * t / 2^32, is at most one too small (t / 2^32 < 1 bounds the loss). */
ZG_HD uint32_t zg_seg_of(const ZGeom *g, uint32_t t)
{
    uint32_t s = (uint32_t)(((uint64_t)t * g->nt_rcp) >> 32);
    if (t - s * (uint32_t)g->nt_reg >= (uint32_t)g->nt_reg) s++;
    return s;
}

ZG_HD void zg_tile(const ZGeom *g, uint64_t t, ZTile *z)
{
    uint64_t k, nb;
    if (t < (uint64_t)g->T * g->nt_reg) {
        uint64_t s = zg_seg_of(g, (uint32_t)t); /* tiles and tiles per segment < 2^32 */
        k = t - s * g->nt_reg;
        z->seg = (uint32_t)s;
        z->seg_start = s * g->tbs;
        z->seg_len = g->tbs;
        nb = g->nb_reg;
        z->gblk0 = s * g->nb_reg + k * g->TB;
        z->grp0 = s * g->gr_reg + k * ZG_SUB;
    } else {
        k = t - (uint64_t)g->T * g->nt_reg;
        z->seg = g->T;
        z->seg_start = (uint64_t)g->T * g->tbs;
        z->seg_len = g->rem;
        nb = g->nb_rm;
        z->gblk0 = (uint64_t)g->T * g->nb_reg + k * g->TB;
        z->grp0 = (uint64_t)g->T * g->gr_reg + k * ZG_SUB;
    }
    z->blk0 = k * g->TB;
    uint64_t left = nb > z->blk0 ? nb - z->blk0 : 0;
    z->nblk = (uint32_t)(left < g->TB ? left : g->TB);
    z->has_head = (k == 0);
    z->e_first = z->seg_start + 1 + z->blk0 * g->L;
    uint64_t last = (z->blk0 + z->nblk) * g->L; /* elements after the head, capped below */
    if (last > z->seg_len - 1) last = z->seg_len - 1;
    z->e_end = z->seg_start + 1 + last;
}

/* Elements of block j (index within the segment) of a segment of len. */
ZG_HD uint32_t zg_block_len(uint64_t len, uint32_t L, uint64_t j)
{
    uint64_t left = len - 1 - j * L;
    return (uint32_t)(left < L ? left : L);
}

/* Upper bound on the bytes of a whole stream (every block at width 32). */
ZG_HD uint64_t zg_seg_worst(uint64_t len, uint32_t L)
{
    if (!len) return 0;
    uint64_t nfull = (len - 1) / L, ntail = (len - 1) % L;
    uint64_t s = 4 + nfull * zg_block_bytes(32, L);
    if (ntail) s += zg_block_bytes(32, (uint32_t)ntail);
    return s;
}

/* Bytes of the header: an offset per chunk (up to 2^31 of them). */
ZG_HD uint64_t zg_header_bytes(const ZGeom *g) { return 8ull * g->T; }

ZG_HD uint64_t zg_stream_worst(const ZGeom *g)
{
    return zg_header_bytes(g) + (uint64_t)g->T * zg_seg_worst(g->tbs, g->L) + zg_seg_worst(g->rem, g->L);
}

/* The header walk of a stream without an index reads every chunk's bytes in
 * windows of WALK_WW bytes, which it handles in groups. */
#define WALK_WW 2048u /* bytes per window */
#define WALK_GMAX 64u /* windows per group at most */

/* Windows per group: as many (a power of two) as their tables of M words fit
 * 128 KB of shared memory. */
ZG_HD uint32_t walk_group(uint32_t M)
{
    uint32_t G = WALK_GMAX;
    while (G > 1 && G * M * 4u > 128u * 1024u) G >>= 1;
    return G;
}

/* Windows of a chunk whose blocks lie in bytes [P, R). */
ZG_HD uint32_t walk_windows(uint64_t P, uint64_t R) { return (uint32_t)zg_div_up(R - P, WALK_WW); }

/* Most windows, and most groups of them, that the chunks of one header have:
 * walk_chunk takes no chunk above its worst size, and every chunk may end in
 * a part of a window and of a group. */
ZG_HD uint32_t walk_max_windows(const ZGeom *g) { return (uint32_t)(zg_stream_worst(g) / WALK_WW + g->T + 2); }

ZG_HD uint32_t walk_max_groups(const ZGeom *g)
{
    const uint32_t G = walk_group(zg_block_bytes(32, g->L));
    return (walk_max_windows(g) + G - 1) / G + g->T + 1;
}

/* Chunk s of a stream of `avail` readable bytes, none of them used from
 * end_bound on, whose header gives its offset `rel` and the next chunk's
 * `next` (s + 1 < T): *P its first block's byte, *R the end of the bytes its
 * blocks may take.  ZERR_* bits, 0 for a chunk that can be walked.  No chunk
 * takes more than a segment's worst size: a header whose offsets do not
 * increase could otherwise give many chunks the same bytes, and more windows
 * than walk_max_windows(). */
ZG_HD uint32_t walk_chunk(const ZGeom *g, uint32_t s, uint64_t rel, uint64_t next, uint64_t avail, uint64_t end_bound,
                          uint64_t *P, uint64_t *R)
{
    const uint64_t hdr = zg_header_bytes(g);
    uint32_t bad = s == 0 && rel != 0 ? ZERR_CORRUPT : 0u;
    *P = *R = 0;
    if (hdr > avail || rel > avail - hdr || hdr + rel + 4 > avail) return bad | ZERR_BOUNDS;
    const uint64_t worst = hdr + rel + zg_seg_worst(g->tbs, g->L); /* where its blocks end at the latest */
    *P = hdr + rel + 4;
    if (s + 1 < g->T) {
        *R = hdr + next;
        if (next > avail - hdr || *R < *P || *R > end_bound || *R > worst) bad |= ZERR_CORRUPT;
    } else { /* no later start bounds it (a remainder segment follows it and is walked apart) */
        *R = avail < end_bound ? avail : end_bound;
        if (*R > worst) *R = worst;
        if (*R < *P) *R = *P;
    }
    return bad;
}

ZG_HD uint32_t zg_a16(uint32_t v) { return (v + 15u) & ~15u; }

/* Largest tile in bytes: head + TB blocks at width 32. */
ZG_HD uint32_t zg_tile_worst(uint32_t L, uint32_t TB) { return TB * zg_block_bytes(32, L) + 4u; }

/* Bytes past a tile's last block that its decoders may read, and discard:
 * decode_octet (eight elements a lane), and the forms that take 32 elements a
 * lane also of a short block (its first bytes, then 31 elements of four bytes). */
ZG_HD uint32_t zg_octet_slack(uint32_t L) { return (L + 7u) / 8u + 8u * ((L + 7u) / 8u) + 24u; }
ZG_HD uint32_t zg_lane_slack(void) { return 136u; }

/* Bytes a packed tile of `total` bytes takes in the output ring (its bytes,
 * the packer's zeroed tail, 16-byte granularity), and the ring's size: the
 * largest tile fits; readers may look 32 bytes past a tile, so the region
 * behind the ring has that slack. */
ZG_HD uint32_t zg_ring_need(uint32_t total) { return (total + 8u + 15u) & ~15u; }
ZG_HD uint32_t zg_ring_bytes(uint32_t L, uint32_t TB) { return zg_ring_need(zg_tile_worst(L, TB)); }

#endif
