/*
 * zkern.cuh -- kernel argument blocks and launchers (internal interface
 * between the C-ABI layer and the kernels).
 */
#ifndef ZCCL_GB300_ZKERN_CUH
#define ZCCL_GB300_ZKERN_CUH

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "zdev.cuh"
#include "zgeom.h"
#include "zlaunch.h"

#define ZH_MAXP 32 /* most inputs one homomorphic-add launch accepts */

/* Per-call scratch in device memory: err | walk_err | ticket | role |
 * status[ntiles].  The first two stay until they are checked, the others are
 * zeroed before every compression and add. */
struct ZWork {
    uint32_t *err;      /* ZERR_* bits of the codec kernels */
    uint32_t *walk_err; /* ZERR_* bits of the index walk that ran before, if any */
    uint32_t *ticket;   /* next tile to hand out */
    uint32_t *role;     /* CTAs started: the first one scans */
    uint64_t *status;   /* one word per tile (of all jobs): its size, then its place */
    uint32_t spin;      /* polls before a wait on one gives up */
};

/* Side index of a resident stream: enough to find every block without
 * walking the 1-byte headers, and the place of and quantized value before
 * every group of blocks, so that decompression's warps, one per group, need
 * nothing from each other.  (12 bytes per group of 32 blocks of 32 floats:
 * 0.3 % of the floats' bytes.) */
struct ZIndex {
    uint8_t *widths;     /* [nblocks] width byte of every block, stream order */
    uint64_t *grp_off;   /* [ngroups] byte offset (from stream start) of each group's first unit */
    int32_t *grp_qprev;  /* [ngroups] quantized value of the element before the group's first block */
    uint64_t *size;      /* [1]       total stream bytes */
};

/* One buffer to compress: the kernels take a single job from their
 * arguments, or a batch of jobs from device memory, whose tiles then form
 * one ticket sequence (tile_job gives every batch tile its job, job_tile0
 * every job its first batch tile). */
struct alignas(16) CompressJob {
    ZGeom g;
    const float *x;
    uint8_t *out;
    uint64_t cap; /* writable bytes at `out` */
    ZIndex idx;
    float inv;        /* 1.0f / eb, computed on the host in float */
    uint32_t boxed;   /* batch job: batch.maps[job] views x as rows of 32 floats */
};

struct ZBatch {
    const void *jobs;          /* CompressJob[] or HomAddJob[]; null: the single job */
    const uint16_t *tile_job;  /* [ntiles] */
    const uint64_t *job_tile0; /* [njobs] */
    uint32_t njobs;
    uint64_t ntiles;  /* tiles of all jobs */
    const void *maps; /* compress: CUtensorMap[njobs] in device memory (used where a job is boxed), or null */
};

struct CompressArgs {
    CompressJob job; /* the single job (batch.jobs == null) */
    ZBatch batch;
    ZWork w;
    ZWidthTable wt;
    uint32_t grid; /* CTAs to launch, 0 = as many as fit */
    uint32_t ring; /* bytes of the ring of packed tiles (filled by the launcher) */
    int rows_map;  /* set by the launcher: its tensor map views job.x as rows of 32 floats */
};

struct HomInput {
    const uint8_t *bytes;
    uint64_t avail;
    const uint8_t *widths;
    const uint64_t *grp_off;
    const int32_t *grp_qprev;
};

/* One homomorphic sum of P streams. */
struct alignas(16) HomAddJob {
    ZGeom g;
    HomInput in[ZH_MAXP];
    uint32_t P;
    int qprev_valid;  /* every input's grp_qprev is valid */
    uint8_t *out;
    uint64_t cap;     /* writable bytes at `out` */
    ZIndex idx;       /* index of the output stream */
};

/* One indexed stream to decompress: the floats go to y, or are added to y
 * with accumulate. */
struct alignas(16) DecompressJob {
    ZGeom g;
    const uint8_t *in;
    uint64_t avail; /* readable bytes at `in` */
    float *y;
    ZIndex idx; /* widths and grp_off must be valid */
    float eb;
    int accumulate;
};

struct DecompressArgs {
    DecompressJob job; /* the single job (batch.jobs == null) */
    ZBatch batch;
    int qprev_valid;   /* grp_qprev valid; else (single job) recovered first and written */
    ZWork w;           /* err, walk_err */
    uint32_t grid;     /* CTAs to launch, 0 = as many as fit */
    uint32_t room, in_bytes; /* shared bytes for staged input, and with slack (filled by the launcher) */
};

struct HomAddArgs {
    HomAddJob job; /* the single job (batch.jobs == null) */
    ZBatch batch;
    unsigned long long *cases; /* optional [4]: both zero, first zero, second zero, both non-zero (P == 2) */
    ZWork w;
    ZWidthTable wt;
    uint32_t grid; /* CTAs to launch, 0 = as many as fit */
    uint32_t in_ring, in_bytes, ring; /* shared bytes of the input ring, with slack, and of the output ring (filled by the launcher) */
};

/* Device scratch of the header walk (part of the workspace). */
struct WalkScratch {
    uint64_t *seg_P;    /* [T]   first block byte of each regular segment */
    uint64_t *seg_R;    /* [T]   end of its byte region (next chunk start, or a bound) */
    uint64_t *seg_end;  /* [T]   byte after its last block, found by the walk */
    uint32_t *seg_ok;   /* [T]   header entries usable */
    uint32_t *win_base; /* [T+1] first window of each segment (prefix sum) */
    uint32_t *grp_base; /* [T+1] first window group of each segment */
    uint32_t *wtab;     /* [max_windows * M] exit offset << 16 | blocks, per entry offset; all ones: dead */
    uint64_t *gtab;     /* [max_groups * M]  blocks << 32 | exit offset, per group; top bit: dead, with the windows entered */
    uint32_t *gentry;   /* [max_groups] windows of the group that are entered << 16 | its true entry offset */
    uint64_t *gbase;    /* [max_groups] first block (in its segment) of each group */
    uint32_t *gwin;     /* [max_groups * M * G] per group, entry offset and window k of it:
                           blocks before k << 12 | entry offset of k */
};

struct WalkArgs {
    const uint8_t *in;
    uint64_t avail;     /* readable bytes at `in` */
    uint64_t end_bound; /* no stream of this geometry is longer */
    ZGeom g;
    ZIndex idx;
    uint32_t *err;
    WalkScratch ws;
    uint32_t max_windows, max_groups;
    uint32_t M, G;          /* largest full block in bytes, windows per group (filled by launch_walk) */
    uint32_t w1_warp_bytes; /* filled by launch_walk */
    uint32_t seg_batch;     /* group tables staged per step of W2b (filled by launch_walk) */
};

/* Grid of a persistent kernel: every CTA that fits on the device at once,
 * but no more CTAs than tiles. */
#define ZP_NONE (~0ull) /* no more tiles */

/* ------------------------------------------------------------------
 * Hand-off of packed tiles from the compute warps to the placer warp.
 *
 * The packed tiles wait in a ring of shared memory with ZR_SLOTS slots, so
 * that the compute warps can pack tile k + 1 while the placer still writes
 * out tile k.  The loader describes tile k in slot k % ZR_SLOTS when it
 * claims it (after the placer is done with the slot's previous tile); its
 * size goes to the placer (mbarrier `sized`, one arrival by thread 0) right
 * after the scan has found it, and `packed` (one arrival per packing warp)
 * then hands over its bytes.  Ring space is counted in running bytes: a tile
 * takes the next `need` bytes (skipping to the ring's start when it would
 * not fit before the end) and may be written once the placer's running
 * count of released bytes, `tail`, shows that the space is free.  Up to
 * ZR_SLOTS tiles are between sizing and write-out at once (the ring's bytes
 * hold one worst-case tile, far more typical ones), so the packing warps do
 * not wait for a placer whose tile's place is late; 16 measured 3.7 % faster
 * than 4 on the two-way add.  All waits are bounded: on time-out
 * ZERR_TIMEOUT is set and the caller goes on.
 * ------------------------------------------------------------------ */
#define ZR_SLOTS 16u

struct ZSlot {
    uint64_t ticket;    /* ZP_NONE ends the placer */
    uint8_t *out;       /* the stream, its writable bytes */
    uint64_t cap;
    uint64_t *grp_off;  /* index: the tile's first group's offset */
    uint8_t *hdr;       /* a segment's first tile: its chunk offset in the header, else null */
    uint64_t *size;     /* the stream's last tile: where its size goes, else null */
    uint64_t T8;        /* bytes before the first tile's: the header */
    uint32_t ngrp;      /* the tile's groups */
    uint32_t total, pos, mend;
    uint16_t goff[ZG_SUB]; /* where each of its groups starts in it (a tile is below 64 KB) */
};

struct ZRing {
    uint32_t placed; /* tiles written out (placer lane 0, release) */
    uint32_t tail;   /* running count of released ring bytes (release) */
    uint64_t sized[ZR_SLOTS], packed[ZR_SLOTS]; /* mbarriers */
    ZSlot slot[ZR_SLOTS];
};

__device__ __forceinline__ void ring_set(uint32_t *p, uint32_t v)
{
    asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}

__device__ __forceinline__ uint32_t ring_get(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
    return v;
}

/* One thread: wait until *p >= v (counted with wrap-around). */
static __device__ __noinline__ void ring_wait_slow(const uint32_t *p, uint32_t v, uint32_t *err)
{
    for (uint32_t i = 0; i < (1u << 24); i++) {
        if ((int32_t)(ring_get(p) - v) >= 0) return;
        __nanosleep(64);
    }
    atomicOr(err, ZERR_TIMEOUT);
}
__device__ __forceinline__ void ring_wait(const uint32_t *p, uint32_t v, uint32_t *err)
{
    if ((int32_t)(ring_get(p) - v) < 0) ring_wait_slow(p, v, err);
}

/* Thread 0, before the CTA's first barrier. */
__device__ __forceinline__ void ring_init(ZRing *r, uint32_t packers)
{
    r->placed = 0;
    r->tail = 0;
#pragma unroll 1
    for (uint32_t i = 0; i < ZR_SLOTS; i++) {
        mbar_init(&r->sized[i], 1);
        mbar_init(&r->packed[i], packers);
    }
}

/* The loader's lane 0: the slot of its k-th tile, free. */
__device__ __forceinline__ ZSlot &ring_slot(ZRing *r, uint32_t k, uint32_t *err)
{
    if (k >= ZR_SLOTS) ring_wait(&r->placed, k - ZR_SLOTS + 1, err);
    return r->slot[k % ZR_SLOTS];
}

/* ... and its description: batch ticket t, tile z (number `local`) of the
 * stream that goes to out. */
__device__ __forceinline__ void ring_describe(ZSlot &S, uint64_t t, uint64_t local, const ZTile &z, const ZGeom &g,
                                              uint8_t *out, uint64_t cap, const ZIndex &idx)
{
    S.ticket = t;
    S.out = out;
    S.cap = cap;
    S.grp_off = idx.grp_off + z.grp0;
    S.hdr = z.has_head && z.seg < g.T ? out + 8ull * z.seg : nullptr;
    S.size = local == g.ntiles - 1 ? idx.size : nullptr;
    S.T8 = zg_header_bytes(&g);
    S.ngrp = z.nblk ? (z.nblk + g.GB - 1u) / g.GB : 1u;
}

/* Thread 0: tile k's size for the placer. */
__device__ __forceinline__ void ring_sized(ZRing *r, uint32_t k, uint32_t total)
{
    r->slot[k % ZR_SLOTS].total = total;
    mbar_arrive(&r->sized[k % ZR_SLOTS]);
}

/* Every packing thread (the same result in each): the ring position of the
 * next tile of `need` bytes, after waiting until its bytes are free.  H is
 * the running count of ring bytes taken (compared with wrap-around) and hp
 * the ring position after the last tile; *mend receives the tile's running
 * end. */
__device__ __forceinline__ uint32_t ring_space(ZRing *r, uint32_t need, uint32_t R, uint32_t &H, uint32_t &hp,
                                               uint32_t &mend, uint32_t *err)
{
    const uint32_t H0 = H;
    uint32_t M = H, pos = hp;
    if (pos + need > R) { /* skip the ring's end */
        M += R - pos;
        pos = 0;
    }
    H = M + need;
    hp = pos + need;
    mend = H;
    /* the bytes' previous contents end at running byte M + need - R, but
     * nothing past H0 was ever written: after a skip the requirement is at
     * most that every earlier tile is out */
    uint32_t req = M + need - R;
    if ((int32_t)(req - H0) > 0) req = H0;
    ring_wait(&r->tail, req, err);
    return pos;
}

/* Thread 0, before its warp's `packed` arrival: where tile k lies. */
__device__ __forceinline__ void ring_where(ZRing *r, uint32_t k, uint32_t pos, uint32_t mend)
{
    r->slot[k % ZR_SLOTS].pos = pos;
    r->slot[k % ZR_SLOTS].mend = mend;
}

/* Thread 0, when there is no tile k: ends the placers. */
__device__ __forceinline__ void ring_end(ZRing *r, uint32_t k, uint32_t placers, uint32_t *err)
{
#pragma unroll 1
    for (uint32_t i = k; i < k + placers; i++) {
        ring_slot(r, i, err).ticket = ZP_NONE;
        mbar_arrive(&r->sized[i % ZR_SLOTS]);
    }
}

/* A placer warp, number p of N taking turns: for every N-th tile k its byte offset in its stream
 * (as soon as its size is known, from the scan of the tiles' sizes), then
 * the chunk offset in the header (a segment's first tile), the stream's size
 * (its last) and, once the tile is packed, its groups' offsets in the side
 * index and its bytes, with 16-byte vector stores realigned to that offset.
 * Its ring bytes are zeroed, so the packers find zeroed space, and
 * released. */
template <uint32_t N>
__device__ __forceinline__ void placer_loop(ZRing *r, uint8_t *ringb, uint64_t *status, uint64_t max_tiles,
                                            uint32_t p, uint32_t *err, uint32_t &bad, uint32_t spin)
{
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll 1
    for (uint64_t k = p; k <= max_tiles + N; k += N) {
        const uint32_t s = (uint32_t)k % ZR_SLOTS, par = (uint32_t)(k / ZR_SLOTS) & 1u;
        mbar_wait(&r->sized[s], par, err);
        const ZSlot &S = r->slot[s];
        const uint64_t t = S.ticket;
        if (t == ZP_NONE) break;
        const uint32_t total = S.total;
        /* after a wait that gave up, here or in the scan, a sum may be
         * missing or too small: nothing is written then */
        const uint64_t sum = scan_wait(status + t, total, spin, err), base = S.T8 + sum - total;
        const bool fits = sum != SCAN_NONE && sum >= total && S.T8 + sum <= S.cap;
        if (!fits) bad |= ZERR_CAPACITY;
        if (lane < 8 && fits && S.hdr) S.hdr[lane] = (uint8_t)((base - S.T8) >> (8u * lane));
        if (lane == 0 && S.size) *S.size = base + total;
        mbar_wait(&r->packed[s], par, err);
        if (lane < S.ngrp) S.grp_off[lane] = base + S.goff[lane];
        const uint32_t pos = S.pos, mend = S.mend;
        if (fits) store_realign(S.out + base, ringb + pos, total, lane, 32);
        __syncwarp(); /* every lane has read the tile and its slot */
        uint4 *zr = reinterpret_cast<uint4 *>(ringb + pos);
#pragma unroll 4
        for (uint32_t i = lane; i < zg_ring_need(total) / 16u; i += 32) zr[i] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        if (lane == 0) { /* in order */
            if (N > 1) ring_wait(&r->placed, (uint32_t)k, err);
            ring_set(&r->tail, mend);
            ring_set(&r->placed, (uint32_t)k + 1);
        }
    }
}

/* Thread 0: the job and local tile of batch ticket t. */
__device__ __forceinline__ uint32_t batch_job(const ZBatch &b, uint64_t t, uint64_t *local)
{
    if (!b.jobs) {
        *local = t;
        return 0;
    }
    const uint32_t j = b.tile_job[t];
    *local = t - b.job_tile0[j];
    return j;
}

/* All lanes: the words around the widths w[0, n) of a tile's blocks (n <=
 * 256), requested: blocks 8 lane .. 8 lane + 7 are the eight bytes of v from
 * bit widths_shift(w) on (those from n on are not 0).  Whole words around
 * them are read: the index has four bytes before its widths and sixteen
 * after. */
__device__ __forceinline__ void load_widths(const uint8_t *w, uint32_t n, uint32_t (&v)[3])
{
    const uint32_t lane = threadIdx.x & 31u;
    v[0] = v[1] = v[2] = 0;
    if (8u * lane < n) {
        const uint32_t *p = reinterpret_cast<const uint32_t *>((uintptr_t)(w + 8u * lane) & ~(uintptr_t)3u);
        v[0] = p[0];
        v[1] = p[1];
        v[2] = p[2];
    }
}
__device__ __forceinline__ uint32_t widths_shift(const uint8_t *w) { return ((uint32_t)(uintptr_t)w & 3u) * 8u; }

/* All lanes: the table entries (offset from the tile's first block << 8 |
 * width) of blocks 8 lane .. 8 lane + 7 of a tile of nblk blocks, the last of
 * nlast elements and the others of L, from their widths (load_widths); a
 * width above 32 counts as 0 and sets ZERR_CORRUPT.  Returns the blocks'
 * bytes. */
template <bool L32>
__device__ __forceinline__ uint32_t tile_entries(uint32_t L, uint32_t fmt, uint32_t nblk, uint32_t nlast, uint32_t w0,
                                                 uint32_t w1, uint4 (&e)[2], uint32_t &bad)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t mine = nblk > 8u * lane ? min(nblk - 8u * lane, 8u) : 0u; /* this lane's blocks */
    const bool f32 = L32 && fmt == ZG_FASTMODE1;
    uint32_t ent[8], sum = 0, blast = 0;
#pragma unroll
    for (uint32_t k = 0; k < 8; k++) {
        uint32_t b = k < mine ? ((k < 4 ? w0 : w1) >> (8 * (k & 3))) & 0xFFu : 0u;
        if (b > 32) {
            bad |= ZERR_CORRUPT;
            b = 0;
        }
        ent[k] = sum << 8 | b;
        blast = k + 1 == mine ? b : blast;
        if (k < mine) sum += f32 ? block32_bytes(b) : zg_block_bytes_f(fmt, b, L);
    }
    if (mine && 8u * lane + mine == nblk) /* the tile's last block may be short */
        sum += zg_block_bytes_f(fmt, blast, nlast) - zg_block_bytes_f(fmt, blast, L);
    const uint32_t incl = warp_incl_scan(sum), x = (incl - sum) << 8;
    e[0] = make_uint4(ent[0] + x, ent[1] + x, ent[2] + x, ent[3] + x);
    e[1] = make_uint4(ent[4] + x, ent[5] + x, ent[6] + x, ent[7] + x);
    return __shfl_sync(0xffffffffu, incl, 31);
}

/* All lanes: each lane's v maximised over its block's G lanes (its octet og
 * among them), then block `src / G`'s maximum from its first lane. */
__device__ __forceinline__ uint32_t octet_max(uint32_t v, uint32_t og, uint32_t G, uint32_t src)
{
#pragma unroll 1
    for (uint32_t s = 1; s < G; s <<= 1) {
        const uint32_t u = __shfl_down_sync(0xffffffffu, v, s);
        if (og + s < G) v = max(v, u);
    }
    return __shfl_sync(0xffffffffu, v, src);
}

/* Launchers; each returns the cudaError_t of the launch. */
cudaError_t launch_compress(const CompressArgs &a, cudaStream_t st);
cudaError_t launch_decompress(const DecompressArgs &a, cudaStream_t st);

/* The SZp 3-D codec (zk_szp3d.cu): scratch bytes (err words, block sizes and
 * offsets, and for compress the quantized volume), the largest stream, and
 * the two passes, enqueued on st.  *d_size (device) receives the stream size. */
size_t sz3_workspace_bytes(uint64_t d1, uint64_t d2, uint64_t d3, uint32_t bs, bool compress);
size_t sz3_max_stream_bytes(uint64_t d1, uint64_t d2, uint64_t d3, uint32_t bs);
cudaError_t sz3_compress(uint8_t *out, uint64_t cap, const float *x, uint64_t d1, uint64_t d2, uint64_t d3,
                         uint32_t bs, double eb, void *ws, uint64_t *d_size, cudaStream_t st);
cudaError_t sz3_decompress(float *y, const uint8_t *in, uint64_t avail, uint64_t d1, uint64_t d2, uint64_t d3,
                           uint32_t bs, double eb, void *ws, cudaStream_t st);

/* The OpenMP form of the SZp 3-D codec (zk_szp3d_split.cu): the thread
 * grid of T threads over a d1 x d2 x d3 volume, its sizes, and the two
 * passes (sub-volume after sub-volume through the serial-form kernels).
 * sz3_split_plan fails when T is out of range or an axis has fewer planes
 * than parts.  Decompression takes the T header offsets on the host. */
struct Sz3Split3 {
    uint32_t T;
    uint32_t parts[3]; /* thread grid, parts[0] >= parts[1] >= parts[2] */
    uint64_t dim[3];
};
bool sz3_split_plan(uint64_t d1, uint64_t d2, uint64_t d3, uint32_t T, Sz3Split3 *sp);
void sz3_split_origin(const Sz3Split3 &sp, uint32_t r, uint64_t o[3], uint64_t s[3]);
void sz3_split_extent(const Sz3Split3 &sp, uint32_t r, uint64_t s[3]);
size_t sz3_split_max_stream_bytes(const Sz3Split3 &sp, uint32_t bs);
size_t sz3_split_workspace_bytes(const Sz3Split3 &sp, uint32_t bs, bool compress);
cudaError_t sz3_split_compress(uint8_t *out, uint64_t cap, const float *x, const Sz3Split3 &sp, uint32_t bs, double eb,
                               void *ws, uint64_t *d_size, cudaStream_t st);
cudaError_t sz3_split_decompress(float *y, const uint8_t *in, uint64_t avail, const uint64_t *offs, const Sz3Split3 &sp,
                                 uint32_t bs, double eb, void *ws, cudaStream_t st);

/* Host: a 2-D TMA map of the floats p[0, n), from the 16-byte boundary at or
 * before p on, as rows of 32, boxes of 32 rows, 128-byte swizzle (16-byte
 * chunk k of row r lands at chunk k ^ (r & 7) of a 1024-byte-aligned box).
 * False when there are fewer than 256 whole rows or the driver's encoder is
 * unavailable. */
bool zk_rows_map(CUtensorMap *map, const void *p, uint64_t n);
cudaError_t launch_homadd(const HomAddArgs &a, cudaStream_t st);
cudaError_t launch_walk(const WalkArgs &a, cudaStream_t st);

#endif
