/*
 * zk_compress.cu -- fused single-pass compressor.
 *
 * Replaces ZCCL_float_openmp_threadblock_arg (ZCCL/src/ZCCL_float.c:501-807)
 * and produces the same bytes.  Persistent CTAs take tiles of blocks in
 * ticket order with three kinds of warps.  A loader warp claims a tile, finds
 * its geometry and starts the copy of its floats.  Eight compute warps take a
 * group of the tile's blocks each:
 *   1. quantize (truncation, ZCCL_float.c:580) and form the running deltas
 *      (ZCCL_float.c:581-582; the element before the block supplies the
 *      first one), sign mask, largest magnitude, width (ZCCL_float.c:606)
 *      and encoded size of every block;
 *   2. scan the block sizes for their offsets in the tile (the tile's one
 *      barrier) and publish the tile's size;
 *   3. pack the blocks into a ring in shared memory, while the loader
 *      already fetches the next tile.
 * One CTA of the grid scans the published sizes into the tiles' places
 * (zdev.cuh).  The placer warp waits for each tile's place, writes its bytes
 * with 16-byte vector stores realigned to it, records its groups' offsets
 * and zeroes the ring bytes it has written out (the ring starts zeroed, so
 * packing needs no zeroing pass), all while the compute warps work on the
 * next tiles (the reference's per-thread scan and second memcpy pass,
 * ZCCL_float.c:774-791, disappear).
 * With blocks of 32 elements a thread works on a block; other block lengths
 * go eight elements a thread (G = ceil(L / 8) lanes share a block).
 */
#include <cstring>

#include "zkern.cuh"

namespace {

constexpr uint32_t CMP_WARPS = ZG_SUB;                  /* compute warps */
constexpr uint32_t CMP_NC = 32 * CMP_WARPS;             /* compute threads */
constexpr uint32_t CMP_PLACERS = 2;                     /* placer warps */
constexpr uint32_t CMP_THREADS = CMP_NC + 32 * CMP_PLACERS + 32; /* and the placers and the loader */

/* A claimed tile, written by the loader before its floats' barriers fire. */
struct CTile {
    uint64_t ticket;    /* ZP_NONE: no more tiles */
    uint8_t *widths;    /* index: the tile's first block's width */
    int32_t *grp_qprev; /* index: the tile's first group's starting value */
    uint32_t nblk, nlast, has_head, first; /* first: tile 0 of its stream */
    float inv;
    uint32_t fmt;
    uint32_t box;       /* the floats came as swizzled rows (see load_floats) */
    uint32_t at;        /* box: column of a group's first float in its row 0; else unused */
};

struct CShared {
    uint64_t full[CMP_WARPS], empty[CMP_WARPS]; /* per compute warp: its floats arrived; it has read them */
    uint32_t ws[2][34];     /* scan scratch, by tile parity */
    CTile t[4];             /* by tile count: a record is written while the tile before is still being read */
    ZRing ring;
    uint32_t scanner;       /* this CTA scans */
};
constexpr uint32_t CMP_HEAD = (sizeof(CShared) + 1023u) / 1024u * 1024u;
constexpr uint32_t CMP_ROWS = 4096u;                    /* a group's 32 rows of 32 floats */
constexpr uint32_t CMP_IN = CMP_ROWS + 1024u;           /* and the row after; or 1025 + 3 floats (1024-byte multiples) */

/* Lane w < CMP_WARPS: the copy of its warp's floats (those of the tile's
 * group w, and the element before them) into its part of `in`.  A full tile
 * of 32-element blocks comes as rows of 32 floats, the rows of the whole
 * array counted from its 16-byte-aligned start: one TMA tensor load of 32
 * rows from the one that holds the first float on, with the 128-byte swizzle
 * (16-byte chunk k of row r at chunk k ^ (r & 7)), so that a thread reads
 * its block's row with vector loads that meet no bank conflict; the floats
 * past the last row follow as a plain copy.  Other tiles come as they lie. */
struct Floats {
    const float *src;  /* box: row 32; else the first float */
    int32_t row;       /* box: the first row, else -1 */
    uint32_t bytes;    /* from src on */
};

template <bool L32>
__device__ __forceinline__ Floats place_floats(const CompressJob &J, const ZTile &z, uint32_t box, uint32_t w)
{
    const uint32_t cnt = (uint32_t)(z.e_end - z.e_first), GL = J.g.GB * J.g.L, e0 = w * GL;
    Floats f;
    f.src = J.x + (z.e_first - 1) + e0;
    f.row = -1;
    if (L32 && box) {
        const uint64_t e = z.e_first - 1 + e0 + (((uintptr_t)J.x & 15u) >> 2); /* in the aligned array */
        const uint32_t c = (uint32_t)e & 31u;
        f.row = (int32_t)(e >> 5);
        f.src += 1024 - (int32_t)c; /* 128-byte aligned in the aligned array */
        f.bytes = (4u * (c + 1u) + 15u) & ~15u;
    } else {
        /* the element before the group, and its own; nothing for a group past the tile's end */
        f.bytes = 4u * (cnt > e0 ? min(cnt - e0, GL) + 1u : w == 0 ? 1u : 0u);
    }
    return f;
}

template <bool L32>
__device__ __forceinline__ void load_floats(const Floats &f, const void *map, uint8_t *in, uint64_t *bar)
{
    if (L32 && f.row >= 0) {
        fence_proxy_async_smem(); /* earlier generic accesses of the buffer before the async writes */
        mbar_expect_tx(bar, CMP_ROWS + f.bytes);
        tma_load_2d(smem_u32(in), map, 0, f.row, bar);
        bulk_g2s(in + CMP_ROWS, f.src, f.bytes, bar);
    } else {
        tma_load_superset(in, reinterpret_cast<const uint8_t *>(f.src), f.bytes, bar);
    }
}

template <bool L32, bool BATCH>
__device__ __forceinline__ void load_tiles(const CompressArgs &a, CShared *sh, uint8_t *in, const CUtensorMap *xmap)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t total = BATCH ? a.batch.ntiles : a.job.g.ntiles;
    uint32_t ticket = 0; /* lane 0: the next tile's, requested a tile ahead */
    if (lane == 0) ticket = atomicAdd(a.w.ticket, 1u);
#pragma unroll 1
    for (uint32_t it = 0;; it++) {
        const uint64_t t = __shfl_sync(0xffffffffu, ticket, 0);
        CTile &d = sh->t[it & 3u];
        if (t >= total) {
            if (it >= 1)
                for (uint32_t w = 0; w < CMP_WARPS; w++) mbar_wait(&sh->empty[w], (it - 1u) & 1u, a.w.err);
            if (lane == 0) {
                d.ticket = ZP_NONE;
            }
            __syncwarp();
            if (lane < CMP_WARPS) mbar_arrive(&sh->full[lane]);
            return;
        }
        if (lane == 0) ticket = atomicAdd(a.w.ticket, 1u);
        uint64_t local = t;
        uint32_t j = 0;
        if (BATCH) j = batch_job(a.batch, t, &local);
        const CompressJob &J = BATCH ? static_cast<const CompressJob *>(a.batch.jobs)[j] : a.job;
        ZTile z;
        zg_tile(&J.g, local, &z);
        const void *map = BATCH ? (J.boxed ? static_cast<const CUtensorMap *>(a.batch.maps) + j : nullptr)
                                : (a.rows_map ? xmap : nullptr);
        const uint32_t box = L32 && map && z.nblk == 256 && z.e_end - z.e_first == 8192;
        if (lane == 0) {
            ring_describe(ring_slot(&sh->ring, it, a.w.err), t, local, z, J.g, J.out, J.cap, J.idx);
            d.ticket = t;
            d.first = local == 0;
            d.widths = J.idx.widths + z.gblk0;
            d.grp_qprev = J.idx.grp_qprev + z.grp0;
            d.nblk = z.nblk;
            d.nlast = z.nblk ? (uint32_t)(z.e_end - z.e_first) - (z.nblk - 1u) * J.g.L : 0u;
            d.has_head = z.has_head;
            d.inv = J.inv;
            d.fmt = J.g.fmt;
            d.box = box;
            const uint32_t off = ((uint32_t)(uintptr_t)J.x & 15u) >> 2;
            d.at = box ? (uint32_t)(z.e_first - 1 + off) & 31u : (uint32_t)(z.e_first - 1 + off) & 3u;
        }
        __syncwarp();
        const Floats f = place_floats<L32>(J, z, box, lane);
        /* the warps have read the tile before */
        if (it >= 1)
#pragma unroll 1
            for (uint32_t w = 0; w < CMP_WARPS; w++) mbar_wait(&sh->empty[w], (it - 1u) & 1u, a.w.err);
        /* in every lane: a warp with nothing to read is done with this tile as soon as its lane here has sent for
         * it, and a lane that still waited for the tile before would not see that phase any more */
        __syncwarp();
        if (lane < CMP_WARPS) load_floats<L32>(f, map, in + lane * CMP_IN, sh->full + lane);
    }
}

/* A thread's block of 32 elements with the element before it, x[0] first,
 * from its warp's swizzled rows at box: floats c .. c + 32 counted from its
 * row's start (c < 32, the same for the whole tile). */
__device__ __forceinline__ void read_row(uint32_t box, uint32_t c, float (&x)[36])
{
    const uint32_t l = threadIdx.x & 31u;
    const uint32_t r0 = box + l * 128u, x0 = (l & 7u) << 4, r1 = r0 + 128u, x1 = ((l + 1u) & 7u) << 4;
    auto chunk = [&](int t, uint32_t at) {
        const float4 f = ld_shared_v4(at);
        x[4 * t] = f.x;
        x[4 * t + 1] = f.y;
        x[4 * t + 2] = f.z;
        x[4 * t + 3] = f.w;
    };
    if (c < 4u) { /* uniform, as all below; the usual case: segments start on a row */
#pragma unroll
        for (int t = 0; t < 8; t++) chunk(t, r0 | (((uint32_t)t << 4) ^ x0));
        chunk(8, r1 | x1);
    } else {
#pragma unroll
        for (int t = 0; t < 9; t++) {
            const uint32_t q = (c >> 2) + (uint32_t)t, k = (q & 7u) << 4;
            chunk(t, q < 8u ? r0 | (k ^ x0) : r1 | (k ^ x1));
        }
    }
    if (c & 1u) {
#pragma unroll
        for (int j = 0; j < 35; j++) x[j] = x[j + 1];
    }
    if (c & 2u) {
#pragma unroll
        for (int j = 0; j < 33; j++) x[j] = x[j + 2];
    }
}

template <bool L32, bool BATCH>
__global__ void __launch_bounds__(CMP_THREADS, 2) k_compress(const __grid_constant__ CompressArgs a,
                                                             const __grid_constant__ CUtensorMap xmap)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    CShared *sh = reinterpret_cast<CShared *>(smem);
    uint8_t *in = smem + CMP_HEAD;        /* 1024-byte aligned, as the swizzle wants */
    uint8_t *outs = in + CMP_WARPS * CMP_IN; /* the ring of packed tiles */
    const uint32_t R = a.ring;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint32_t bad = 0;

    if (tid == 0) {
#pragma unroll 1
        for (uint32_t w = 0; w < CMP_WARPS; w++) {
            mbar_init(&sh->full[w], 1);
            mbar_init(&sh->empty[w], 1);
        }
        ring_init(&sh->ring, CMP_WARPS);
        sh->scanner = gridDim.x > 1 && atomicAdd(a.w.role, 1u) == 0;
    }
    /* the ring starts zeroed, and the placer zeroes what it has written out */
#pragma unroll 1
    for (uint32_t i = tid; i < (R + 48u) / 16u; i += CMP_THREADS) reinterpret_cast<uint4 *>(outs)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();

    const uint64_t max_tiles = BATCH ? a.batch.ntiles : a.job.g.ntiles;
    if (sh->scanner) {
        if (warp == 0) scan_tiles(a.w.status, max_tiles, a.w.ticket, a.w.err, a.w.spin);
        return;
    }
    if (warp >= CMP_WARPS && warp < CMP_WARPS + CMP_PLACERS) {
        placer_loop<CMP_PLACERS>(&sh->ring, outs, a.w.status, max_tiles, warp - CMP_WARPS, a.w.err, bad, a.w.spin);
        if (bad) atomicOr(a.w.err, bad);
        return;
    }
    if (warp == CMP_WARPS + CMP_PLACERS) {
        load_tiles<L32, BATCH>(a, sh, in, &xmap);
        return;
    }

    /* the compute warps */
    const uint32_t L = L32 ? 32u : a.job.g.L, GB = L32 ? 32u : a.job.g.GB; /* one L for the whole batch */
    const uint32_t G = (L + 7u) / 8u, BPI = 32u / G, og = lane % G, bi = lane / G; /* octets (not L32) */
    const float *lin = reinterpret_cast<const float *>(in + warp * CMP_IN); /* this warp's floats */
    const uint32_t box = smem_u32(lin);
    uint32_t H = 0, hp = 0; /* ring bytes taken and the ring's next position (the same in every thread) */
#pragma unroll 1
    for (uint32_t it = 0; it <= max_tiles; it++) { /* bounded even if a wait gave up */
        mbar_wait(&sh->full[warp], it & 1u, a.w.err);
        const CTile &D = sh->t[it & 3u];
        if (D.ticket == ZP_NONE) {
            if (tid == 0) ring_end(&sh->ring, it, CMP_PLACERS, a.w.err); /* nothing more */
            break;
        }
        const uint32_t tb = D.nblk, b0 = warp * GB, nblk = tb > b0 ? min(GB, tb - b0) : 0u;
        const uint32_t fmt = D.fmt;
        const float inv = D.inv;
        /* lane k: block k of the warp's group */
        const bool own = lane < nblk;
        const uint32_t n = !own ? 0u : b0 + lane + 1u < tb ? L : D.nlast;
        uint32_t b = 0, smask = 0, m[32];
        uint32_t ints = 0; /* not L32, bit i: octet i's magnitudes are integers, without the float form's exponent above them */
        int32_t q0 = 0; /* lane 0: the value before the group */

        if (L32) {
            float x[36];
            uint32_t c = D.at;
            if (!D.box) {
                /* from where the floats lie into swizzled rows in the same
                 * buffer; past the group's last float its copies, whose
                 * deltas are 0 */
                const uint32_t last = nblk ? (nblk - 1u) * 32u + (b0 + nblk == tb ? D.nlast : 32u) : 0u;
#pragma unroll
                for (uint32_t r = 0; r < 33; r++) x[r] = nblk || warp == 0 ? lin[c + min(r < 32 ? lane + 32u * r : 1024u, last)] : 0.f;
                __syncwarp();
                const uint32_t w = box + (lane & 3u) * 4u, k = lane >> 2;
#pragma unroll
                for (uint32_t r = 0; r < 32; r++) st_shared_f32(w + 128u * r + ((k ^ (r & 7u)) << 4), x[r]);
                if (lane == 0) st_shared_f32(box + CMP_ROWS, x[32]);
                __syncwarp(); /* a row's last element is in the next row */
                c = 0;
            }
            read_row(box, c, x);
            uint32_t mx;
            if (__builtin_expect(!quantize_deltas<32>(x, inv, m, smask, mx, q0), 0)) {
                const uint32_t e0 = c;
                quantize_exact<32>(
                    [&](int j) { /* float e0 + j of this thread's rows */
                        const uint32_t q = e0 + (uint32_t)j, r = lane + (q >> 5);
                        return ld_shared_f32(box + r * 128u + ((((q >> 2) & 7u) ^ (r & 7u)) << 4) + (q & 3u) * 4u);
                    },
                    inv, m, smask, mx, q0, bad);
            }
            b = own ? width_of(mx, a.wt) : 0u;
        } else {
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) {
                if (i && i * BPI >= nblk) break; /* uniform: a group may fill fewer rounds */
                const uint32_t k = i * BPI + bi;
                const bool has = bi < BPI && k < nblk;
                const uint32_t nk = !has ? 0u : b0 + k + 1u < tb ? L : D.nlast;
                /* the octet's first element is float e + 1 of the group's, the block's last is float `end`: past
                 * it copies, no delta */
                const uint32_t end = has ? k * L + nk : 0u, e = min(k * L + 8u * og, end);
                float x[9];
#pragma unroll
                for (uint32_t j = 0; j < 9; j++) x[j] = nblk || warp == 0 ? lin[D.at + min(e + j, end)] : 0.f;
                uint32_t mi[8], s8, mx;
                int32_t qi;
                if (__builtin_expect(!quantize_deltas<8>(x, inv, mi, s8, mx, qi), 0)) {
                    quantize_exact<8>([&](int j) { return x[j]; }, inv, mi, s8, mx, qi, bad);
                    ints |= 1u << i;
                }
                if (!has) mx = 0;
                if (i == 0) q0 = qi;
#pragma unroll
                for (int j = 0; j < 8; j++) m[8 * i + j] = mi[j];
                smask |= s8 << (8 * i);
                /* the block's largest magnitude over its lanes, then to lane k */
                const uint32_t w = octet_max(mx, og, G, (lane % BPI) * G);
                if (own && lane / BPI == i) b = width_of(w, a.wt);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->empty[warp]); /* this warp is done with the floats */

        /* the blocks' offsets in the tile, the tile's size, the index entries */
        const uint32_t size = !own ? 0u : fmt == ZG_FASTMODE1 && n == 32u ? block32_bytes(b) : zg_block_bytes_f(fmt, b, n);
        const uint32_t headb = D.has_head ? 4u : 0u;
        uint32_t total;
        const uint32_t off = headb + grp_excl_scan1(size, sh->ws[it & 1u], &total, CMP_NC, 1);
        total += headb;
        if (tid == 0) {
            scan_publish(a.w.status, D.ticket, total, D.first);
            ring_sized(&sh->ring, it, total);
        }
        if (own) D.widths[b0 + lane] = (uint8_t)b;
        if (lane == 0 && (nblk || warp == 0)) D.grp_qprev[warp] = q0;

        /* room in the ring: every thread finds the same place and waits, if
         * need be, for the placer to have written out (and zeroed) what was
         * there */
        uint32_t mend;
        const uint32_t pos = ring_space(&sh->ring, zg_ring_need(total), R, H, hp, mend, a.w.err);
        const uint32_t pk = smem_u32(outs + pos);
        if (lane == 0) sh->ring.slot[it % ZR_SLOTS].goff[warp] = (uint16_t)(warp ? off : 0u);
        if (headb && tid == 0) *reinterpret_cast<int32_t *>(outs + pos) = q0;
        if (L32) {
            if (__builtin_expect(n == 32, 1))
                encode_block(pk, off, b, smask, m, fmt);
            else if (own)
                encode_any(
                    pk, off, b, n,
                    [&](uint32_t j, uint32_t &neg, uint32_t &mg) {
                        neg = (smask >> (31u - j)) & 1u;
                        mg = pick(m, j) & (b < 24 ? 0xFFFFFFu : 0xFFFFFFFFu);
                    },
                    fmt);
        } else {
            const uint32_t ent = off << 8 | b;
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) {
                if (i * BPI >= nblk) break;
                const uint32_t k = i * BPI + bi, e = __shfl_sync(0xffffffffu, ent, k & 31u);
                const bool has = bi < BPI && k < nblk;
                const uint32_t nk = !has ? 0u : b0 + k + 1u < tb ? L : D.nlast;
                if (8u * og < nk) {
                    uint32_t mi[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) mi[j] = 8u * og + (uint32_t)j < nk ? m[8 * i + j] : 0u;
                    /* another octet may have made the block so wide that bits from the 24th on are packed */
                    if (__builtin_expect((e & 0xFFu) >= 24u && !((ints >> i) & 1u), 0)) {
#pragma unroll
                        for (int j = 0; j < 8; j++) mi[j] &= 0x7FFFFFu;
                    }
                    encode_octet(pk, e >> 8, e & 0xFFu, nk, og, (smask >> (8 * i)) & 0xFFu, mi, fmt);
                }
            }
        }
        if (tid == 0) ring_where(&sh->ring, it, pos, mend);
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->ring.packed[it % ZR_SLOTS]); /* this warp's blocks are packed */
    }
    if (bad) atomicOr(a.w.err, bad);
}

} // namespace

cudaError_t launch_compress(const CompressArgs &a0, cudaStream_t st)
{
    CompressArgs a = a0;
    const bool batch = a.batch.jobs != nullptr, l32 = a.job.g.L == 32;
    /* two CTAs share an SM: the ring takes what they leave */
    const uint32_t fixed = CMP_HEAD + CMP_WARPS * CMP_IN + 48u;
    a.ring = ring_bytes(2, fixed, zg_ring_bytes(a.job.g.L, a.job.g.TB));
    const size_t smem = fixed + a.ring;
    void (*fn)(const CompressArgs, const CUtensorMap) =
        l32 ? (batch ? k_compress<true, true> : k_compress<true, false>)
            : (batch ? k_compress<false, true> : k_compress<false, false>);
    const cudaError_t e = set_max_smem((const void *)fn, smem);
    if (e != cudaSuccess) return e;
    const uint64_t tiles = batch ? a.batch.ntiles : a.job.g.ntiles;
    const unsigned grid = scanned_grid((const void *)fn, CMP_THREADS, smem, tiles, a.grid);
    alignas(64) CUtensorMap map;
    memset(&map, 0, sizeof map);
    a.rows_map = l32 && (batch ? a.batch.maps != nullptr : zk_rows_map(&map, a.job.x, a.job.g.n));
    fn<<<grid, CMP_THREADS, smem, st>>>(a, map);
    return cudaGetLastError();
}
