/*
 * zk_homadd.cu -- homomorphic add of P compressed streams in one pass.
 *
 * Replaces ZCCL_float_homomophic_add_openmp_threadblock
 * (ZCCL/src/ZCCLd_float.c:988-1679).  The reference result is the canonical
 * encoding of the summed int32 deltas with int32-added heads
 * (ZCCLd_float.c:1072, :1172-1219; a zero-width side is copied verbatim,
 * :1103-1153, which is the same bytes because every input block is itself
 * canonical).  Integer addition is associative modulo 2^32, so one pass over
 * P inputs equals the ring's pairwise fold in any order, bit for bit.
 *
 * Persistent CTAs take tiles in ticket order with three kinds of warps.  A
 * loader warp turns every input of every claimed tile into one TMA copy
 * into one of two buffers, with a table of each block's offset and width
 * found from the input's width index.  Eight adding warps, a group of the
 * tile's blocks each, decode every input as it arrives and add it into
 * registers (zero-width blocks are skipped without touching their bytes),
 * handing each buffer back through an mbarrier.  After the last input the
 * sum is re-encoded like the compressor does (width, scan, early publication
 * of its size, packing into a shared-memory ring), and the placer warp waits
 * for its place in the stream and writes it out while the adding warps go
 * on; one CTA of the grid scans the tiles' sizes into places (zdev.cuh).  The starting value per group is the sum of the inputs'
 * values.
 * With blocks of 32 elements a thread works on a block; other block lengths
 * go eight elements a thread (G = ceil(L / 8) lanes share a block).
 */
#include "zkern.cuh"

namespace {

constexpr uint32_t ADD_WARPS = ZG_SUB;           /* adding warps */
constexpr uint32_t ADD_NC = 32 * ADD_WARPS;      /* adding threads */
constexpr uint32_t ADD_THREADS = ADD_NC + 64;    /* and the placer and the loader */

constexpr uint32_t IN_SLOTS = 4; /* input copies in flight */

/* One staged input tile: where its bytes start within the input ring (the
 * TMA copy keeps the source's 16-byte phase). */
struct HStage {
    uint32_t none; /* no more tiles */
    uint32_t at;   /* the tile's first byte in the ring */
    uint32_t mend; /* the copy's end in running ring bytes */
};

/* What the adding warps need of a claimed tile, written by the loader with
 * the tile's first input so that the adders read shared memory instead of
 * the job in device or parameter memory.  TILE_RECS records, by tile count:
 * the loader runs at most IN_SLOTS input copies ahead of the adders, so with
 * IN_SLOTS + 2 records one is reused only after its tile is packed. */
struct HTile {
    uint8_t *widths;    /* the sum's width index, from the tile's first block on */
    int32_t *grp_qprev; /* the sum's starting values from the tile's first group on, or null */
    uint64_t ticket;
    uint32_t P, nblk;
    uint32_t nlast;     /* elements of the tile's last block */
    uint32_t has_head;  /* tile 0 of its segment */
    uint32_t first;     /* tile 0 of its stream */
    uint32_t qsum[ZG_SUB]; /* the inputs' starting values of the tile's groups, summed */
};
constexpr uint32_t TILE_RECS = 8;
static_assert(TILE_RECS >= IN_SLOTS + 2, "records outlast the copies in flight");

struct HShared {
    uint64_t full[IN_SLOTS], empty[IN_SLOTS]; /* input copy arrived; consumed */
    HStage stage[IN_SLOTS];
    HTile t[TILE_RECS];
    uint32_t ws[2][34];         /* scan scratch, by tile parity */
    ZRing ring;
    uint32_t scanner;           /* this CTA scans */
    alignas(16) uint32_t ent[IN_SLOTS][256];       /* per block of the staged input: offset << 8 | width */
};
constexpr uint32_t ADD_HEAD = (sizeof(HShared) + 127u) / 128u * 128u;

template <bool BATCH>
__device__ __forceinline__ const HomAddJob &job_of(const HomAddArgs &a, uint32_t j)
{
    return BATCH ? static_cast<const HomAddJob *>(a.batch.jobs)[j] : a.job;
}

/* The inputs' starting values of the tile's groups, as loads in flight: lane
 * 8p + k: group k of input p (and of p + 4, ...). */
__device__ __forceinline__ uint32_t group_starts(const HomAddJob &J, const ZTile &z, uint32_t lane)
{
    const uint32_t k = lane & 7u, p = lane >> 3;
    uint32_t q = 0;
    if (J.qprev_valid && p < J.P && (k == 0 || k * J.g.GB < z.nblk)) {
        q = (uint32_t)J.in[p].grp_qprev[z.grp0 + k];
#pragma unroll 1
        for (uint32_t i = p + 4u; i < J.P; i += 4u) q += (uint32_t)J.in[i].grp_qprev[z.grp0 + k];
    }
    return q;
}

/* The loader warp.  It claims tiles in ticket order and, for every input of
 * every claimed tile, finds each block's width and offset from the input's
 * width index (eight blocks per lane and a warp scan), writes them into a
 * block table (offset << 8 | width), takes room in the input ring and starts
 * one TMA copy of the tile's bytes; the copy's mbarrier tells the adding
 * warps.  Up to IN_SLOTS copies are in flight, as far as the ring has room
 * (it holds two of the largest, typically all).  After the last tile it
 * hands over a stage marked `none`.
 *
 * The ticket of the tile after next is requested early, and the next copy's
 * offset, widths and starting values before the current copy is handed over,
 * so that their latencies overlap that work instead of adding up.  A claimed
 * tile is always processed, in order, and the adding warps never wait on
 * another CTA before they publish their tile's size, so every wait for a
 * place ends. */
template <bool L32, bool BATCH>
__device__ __forceinline__ void load_inputs(const HomAddArgs &a, HShared *sh, uint8_t *in, uint32_t &bad)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t ntiles = BATCH ? a.batch.ntiles : a.job.g.ntiles;
    const uint32_t L = a.job.g.L, RB = a.in_ring;
    uint32_t ticket = 0; /* lane 0: the next tile's */
    uint64_t nt = 0, ntk = 0, nbase = 0;    /* the copy to hand over next: its tile, ticket, the tile's offset */
    uint32_t nj = 0, np = 0, nq = 0, nw[3]; /* its job, input, group starts (input 0), words around its widths */
    ZTile nz;
    bool have = true;
    auto request = [&](bool open) { /* open: the next tile's input 0, else the tile's next input */
        if (open) {
            const uint64_t tk = __shfl_sync(0xffffffffu, ticket, 0);
            if (tk >= ntiles) {
                have = false;
                return;
            }
            if (lane == 0) ticket = atomicAdd(a.w.ticket, 1u);
            nt = ntk = tk;
            if (BATCH) nj = batch_job(a.batch, tk, &nt);
            np = 0;
            zg_tile(&job_of<BATCH>(a, nj).g, nt, &nz);
            nq = group_starts(job_of<BATCH>(a, nj), nz, lane);
        } else {
            np++;
        }
        const HomInput &I = job_of<BATCH>(a, nj).in[np];
        nbase = I.grp_off[nz.grp0];
        load_widths(I.widths + nz.gblk0, nz.nblk, nw);
    };
    uint32_t seq = 0, ti = 0;              /* copies handed over, tiles opened */
    uint32_t old = 0, freed = 0;           /* copies known consumed, running ring bytes they end at */
    uint32_t H = 0, hp = 0;                /* running ring bytes taken, the ring's next position */
    auto reclaim = [&]() { /* wait for the oldest copy in flight */
        mbar_wait(&sh->empty[old % IN_SLOTS], (old / IN_SLOTS) & 1u, a.w.err);
        freed = sh->stage[old % IN_SLOTS].mend;
        old++;
    };
    if (lane == 0) ticket = atomicAdd(a.w.ticket, 1u);
    request(true);
    bool open = true;
    for (; have; seq++) {
        const uint64_t t = nt, tk = ntk;
        uint64_t base = nbase;
        const uint32_t j = nj, p = np, qv = nq;
        const uint32_t wsh = widths_shift(job_of<BATCH>(a, j).in[p].widths + nz.gblk0);
        const uint32_t w0 = __funnelshift_r(nw[0], nw[1], wsh), w1 = __funnelshift_r(nw[1], nw[2], wsh);
        const ZTile z = nz;
        const HomAddJob &J = job_of<BATCH>(a, j);
        open = p + 1 >= J.P;
        request(open);

        /* hand over this copy */
        const HomInput &I = J.in[p];
        const uint32_t nlast = z.nblk ? (uint32_t)(z.e_end - z.e_first) - (z.nblk - 1u) * L : 0u;
        uint4 e[2];
        const uint32_t total = tile_entries<L32>(L, ZG_FASTMODE1, z.nblk, nlast, w0, w1, e, bad) + (z.has_head ? 4u : 0u);
        uint32_t nload = total;
        /* overflow-safe: base comes from the index and is not trusted */
        if (base > I.avail || total > I.avail - base) {
            bad |= ZERR_BOUNDS;
            nload = base < I.avail ? (uint32_t)min((uint64_t)total, I.avail - base) : 0u;
            if (base > I.avail) base = 0;
        }
        const uint32_t ph = (uint32_t)((uintptr_t)(I.bytes + base) & 15u), need = (ph + total + 15u) & ~15u;
        /* room: the ring position, skipping its end when the copy would not
         * fit before it, once every byte it overwrites is consumed */
        uint32_t M = H, pos = hp;
        if (pos + need > RB) {
            M += RB - pos;
            pos = 0;
        }
        while (old < seq && (seq - old >= IN_SLOTS || (int32_t)(M + need - RB - freed) > 0)) reclaim();
        H = M + need;
        hp = pos + need;

        const uint32_t s = seq % IN_SLOTS;
        if (p == 0) { /* the tile's record, before its first copy is handed over */
            uint32_t q = qv + __shfl_xor_sync(0xffffffffu, qv, 8);
            q += __shfl_xor_sync(0xffffffffu, q, 16);
            HTile &d = sh->t[ti % TILE_RECS];
            if (lane < ZG_SUB) d.qsum[lane] = q;
            if (lane == 0) {
                ring_describe(ring_slot(&sh->ring, ti, a.w.err), tk, t, z, J.g, J.out, J.cap, J.idx);
                d.ticket = tk;
                d.first = t == 0;
                d.widths = J.idx.widths + z.gblk0;
                d.grp_qprev = J.qprev_valid ? J.idx.grp_qprev + z.grp0 : nullptr;
                d.P = J.P;
                d.nblk = z.nblk;
                d.nlast = nlast;
                d.has_head = z.has_head;
            }
            ti++;
        }
        uint4 *tab = reinterpret_cast<uint4 *>(&sh->ent[s][8u * lane]);
        tab[0] = e[0];
        tab[1] = e[1];
        __syncwarp();
        if (lane == 0) {
            sh->stage[s].none = 0;
            sh->stage[s].at = pos + ph;
            sh->stage[s].mend = H;
            tma_load_superset(in + pos, I.bytes + base, nload, &sh->full[s]);
        }
        __syncwarp();
    }
    /* no more tiles */
    while (seq - old >= IN_SLOTS) reclaim();
    if (lane == 0) {
        sh->stage[seq % IN_SLOTS].none = 1;
        mbar_arrive(&sh->full[seq % IN_SLOTS]);
    }
}

/* The adding warps meet at one barrier per tile (the scan of the sum's block
 * sizes); inputs arrive and buffers are returned through mbarriers, and
 * packed sums go to the placer through a per-slot mbarrier that every adding
 * warp arrives on. */
template <bool L32, bool BATCH>
__global__ void __launch_bounds__(ADD_THREADS, 2) k_homadd(const __grid_constant__ HomAddArgs a)
{
    extern __shared__ __align__(128) uint8_t smem[];
    HShared *sh = reinterpret_cast<HShared *>(smem);
    uint8_t *const in = smem + ADD_HEAD; /* the ring of input copies */
    uint8_t *outs = in + a.in_bytes;     /* the ring of packed sums */
    const uint32_t R = a.ring;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint32_t bad = 0;
    /* see k_decompress: a failed index walk stops every CTA alike */
    if (*(volatile const uint32_t *)a.w.walk_err) return;
    if (tid == 0) {
#pragma unroll 1
        for (uint32_t i = 0; i < IN_SLOTS; i++) {
            mbar_init(&sh->full[i], 1);
            mbar_init(&sh->empty[i], ADD_WARPS);
        }
        ring_init(&sh->ring, ADD_WARPS);
        sh->scanner = gridDim.x > 1 && atomicAdd(a.w.role, 1u) == 0;
    }
    /* the ring starts zeroed, and the placer zeroes what it has written out */
#pragma unroll 1
    for (uint32_t i = tid; i < (R + 48u) / 16u; i += ADD_THREADS) reinterpret_cast<uint4 *>(outs)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();

    const uint64_t max_tiles = BATCH ? a.batch.ntiles : a.job.g.ntiles;
    if (sh->scanner) {
        if (warp == 0) scan_tiles(a.w.status, max_tiles, a.w.ticket, a.w.err, a.w.spin);
        return;
    }
    if (warp == ADD_WARPS) { /* the placer warp */
        placer_loop<1>(&sh->ring, outs, a.w.status, max_tiles, 0, a.w.err, bad, a.w.spin);
        if (bad) atomicOr(a.w.err, bad);
        return;
    }
    if (warp == ADD_WARPS + 1) { /* the loader warp */
        load_inputs<L32, BATCH>(a, sh, in, bad);
        if (bad) atomicOr(a.w.err, bad);
        return;
    }

    /* the adding warps */
    const uint32_t L = L32 ? 32u : a.job.g.L, GB = L32 ? 32u : a.job.g.GB; /* one L for the whole batch */
    const uint32_t G = (L + 7u) / 8u, BPI = 32u / G, og = lane % G, bi = lane / G; /* octets (not L32) */
    uint32_t acc[32];
    uint32_t seq = 0;       /* input copies consumed */
    uint32_t H = 0, hp = 0; /* ring bytes taken and the ring's next position (the same in every thread) */
#pragma unroll 1
    for (uint32_t it = 0; it <= max_tiles; it++) { /* bounded even if a wait gave up */
        uint32_t s = seq % IN_SLOTS;
        mbar_wait(&sh->full[s], (seq / IN_SLOTS) & 1u, a.w.err);
        if (sh->stage[s].none) {
            if (tid == 0) ring_end(&sh->ring, it, 1, a.w.err); /* nothing more */
            break;
        }
        const HTile &D = sh->t[it % TILE_RECS];
        const uint32_t P = D.P, tb = D.nblk, b0 = warp * GB, nblk = tb > b0 ? min(GB, tb - b0) : 0u;
        /* lane k: block k of the warp's group */
        const bool own = lane < nblk;
        const uint32_t n = !own ? 0u : b0 + lane + 1u < tb ? L : D.nlast;
        const uint32_t headb = D.has_head ? 4u : 0u;
#pragma unroll
        for (int j = 0; j < 32; j++) acc[j] = 0;
        uint32_t hsum = 0, nzmask = 0;
        /* L32: sums as floats (see ZF_TWO23) while this lane's magnitudes,
         * below `most` in sum, stay exact integers; a warp with a block past
         * that goes on in integers */
        uint32_t most = 0;
        bool fl = L32; /* uniform over the warp */

#pragma unroll 1
        for (uint32_t p = 0; p < P; p++, seq++) { /* one copy of the decoders: the kernel lives by its instruction cache */
            s = seq % IN_SLOTS;
            if (p) mbar_wait(&sh->full[s], (seq / IN_SLOTS) & 1u, a.w.err);
            const uint32_t *sw = reinterpret_cast<const uint32_t *>(in);
            const uint32_t at = sh->stage[s].at, body = at + headb;
            if (headb && tid == 0) {
                uint32_t h = 0;
#pragma unroll
                for (int k = 0; k < 4; k++) h |= (uint32_t)in[at + k] << (8 * k);
                hsum += h;
            }
            const uint32_t e = own ? sh->ent[s][b0 + lane] : 0u, bp = e & 0xFFu, o = body + (e >> 8);
            if (own && in[o] != bp) bad |= ZERR_CORRUPT;
            if (bp) nzmask |= 1u << (p & 31);
            if (L32) {
                if (bp) most += bp < 24 ? 1u << bp : 1u << 25;
                if (fl && !__all_sync(0xffffffffu, most <= (1u << 24))) {
                    fl = false;
#pragma unroll
                    for (int j = 0; j < 32; j++) acc[j] = (uint32_t)__float2int_rn(__uint_as_float(acc[j]));
                }
                if (bp) {
                    auto each = [&](int j, float m, uint32_t sg) {
                        acc[j] = __float_as_uint(__uint_as_float(acc[j]) + with_sign(m, sg, j));
                    };
                    if (__builtin_expect(!fl, 0))
                        decode_add_any(sw, o, bp, n, acc);
                    else if (__builtin_expect(bp < 16, 1))
                        decode_small_f(sw, o, bp, n, each);
                    else
                        decode_mid_f(sw, o, bp, n, each);
                }
            } else {
#pragma unroll
                for (uint32_t i = 0; i < 4; i++) {
                    if (i * BPI >= nblk) break; /* uniform: a group may fill fewer rounds */
                    const uint32_t k = i * BPI + bi, ek = __shfl_sync(0xffffffffu, e, k & 31u);
                    const bool has = bi < BPI && k < nblk;
                    const uint32_t nk = !has ? 0u : b0 + k + 1u < tb ? L : D.nlast;
                    uint32_t d[8];
                    decode_octet(sw, body + (has ? ek >> 8 : 0u), has ? ek & 0xFFu : 0u, nk, og, ZG_FASTMODE1, d);
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[8 * i + j] += d[j];
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->empty[s]); /* this warp is done with the buffer */
        }

        /* branch-case counters of the two-input add (ZCCLd_float.c:2175-2764) */
        if (a.cases && P == 2) {
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) { /* both zero, first zero, second zero, both non-zero */
                const uint32_t want = k == 1 ? 2u : k == 2 ? 1u : k;
                const uint32_t c = __popc(__ballot_sync(0xffffffffu, own && nzmask == want));
                if (lane == 0) atomicAdd(a.cases + k, (unsigned long long)c);
            }
        }
        /* magnitudes, signs, widths of the sum */
        uint32_t b = 0, smask = 0;
        if (L32) {
            if (__builtin_expect(n < 32, 0)) { /* a short block (or none): its sums end at element n */
#pragma unroll
                for (int j = 0; j < 32; j++)
                    if ((uint32_t)j >= n) acc[j] = 0;
            }
            uint32_t mx = 0;
            if (__builtin_expect(fl, 1)) {
                float mf = 0.f;
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    smask = __funnelshift_l(acc[j], smask, 1); /* (smask << 1) | sign of element j */
                    if (j & 1) mf = max3_abs(mf, __uint_as_float(acc[j - 1]), __uint_as_float(acc[j]));
                }
                mx = (uint32_t)mf;
                if (__builtin_expect(mx < (1u << 22), 1)) { /* 2^23 + |sum|: the magnitude in the low 23 bits */
#pragma unroll
                    for (int j = 0; j < 32; j++) acc[j] = __float_as_uint(fabsf(__uint_as_float(acc[j])) + ZF_TWO23);
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++) acc[j] = (uint32_t)fabsf(__uint_as_float(acc[j]));
                }
            } else {
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    smask = __funnelshift_l(acc[j], smask, 1);
                    acc[j] = (uint32_t)abs((int32_t)acc[j]);
                    mx = max(mx, acc[j]);
                }
            }
            b = width_of(mx, a.wt);
        } else {
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) {
                if (i * BPI >= nblk) break;
                uint32_t mx = 0, s8 = 0;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    s8 = s8 << 1 | acc[8 * i + j] >> 31;
                    acc[8 * i + j] = (uint32_t)abs((int32_t)acc[8 * i + j]);
                    mx = max(mx, acc[8 * i + j]);
                }
                smask |= s8 << (8 * i);
                const uint32_t w = octet_max(mx, og, G, (lane % BPI) * G);
                if (own && lane / BPI == i) b = width_of(w, a.wt);
            }
        }

        /* the blocks' offsets in the tile, the tile's size, the index entries */
        const uint32_t size = !own ? 0u : n == 32u ? block32_bytes(b) : zg_block_bytes(b, n);
        uint32_t total;
        const uint32_t off = headb + grp_excl_scan1(size, sh->ws[it & 1u], &total, ADD_NC, 1);
        total += headb;
        if (tid == 0) {
            scan_publish(a.w.status, D.ticket, total, D.first);
            ring_sized(&sh->ring, it, total);
        }
        if (own) D.widths[b0 + lane] = (uint8_t)b;
        if (lane == 0 && D.grp_qprev && (nblk || warp == 0)) D.grp_qprev[warp] = (int32_t)D.qsum[warp];

        /* room for the packed sum in the ring: every thread finds the same
         * place and waits, if need be, for the placer to have written out
         * (and zeroed) what was there */
        uint32_t mend;
        const uint32_t pos = ring_space(&sh->ring, zg_ring_need(total), R, H, hp, mend, a.w.err);
        const uint32_t pk = smem_u32(outs + pos);
        if (lane == 0) sh->ring.slot[it % ZR_SLOTS].goff[warp] = (uint16_t)(warp ? off : 0u);
        if (headb && tid == 0) *reinterpret_cast<uint32_t *>(outs + pos) = hsum;
        if (L32) {
            if (__builtin_expect(n == 32, 1))
                encode_block(pk, off, b, smask, acc);
            else if (own)
                encode_any(pk, off, b, n, [&](uint32_t j, uint32_t &neg, uint32_t &mg) {
                    neg = (smask >> (31u - j)) & 1u;
                    mg = pick(acc, j) & (b < 24 ? 0xFFFFFFu : 0xFFFFFFFFu);
                });
        } else {
            const uint32_t ent = off << 8 | b;
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) {
                if (i * BPI >= nblk) break;
                const uint32_t k = i * BPI + bi, ek = __shfl_sync(0xffffffffu, ent, k & 31u);
                const bool has = bi < BPI && k < nblk;
                const uint32_t nk = !has ? 0u : b0 + k + 1u < tb ? L : D.nlast;
                if (8u * og < nk) {
                    uint32_t mi[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) mi[j] = acc[8 * i + j];
                    encode_octet(pk, ek >> 8, ek & 0xFFu, nk, og, (smask >> (8 * i)) & 0xFFu, mi, ZG_FASTMODE1);
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

cudaError_t launch_homadd(const HomAddArgs &a0, cudaStream_t st)
{
    HomAddArgs a = a0;
    const uint32_t L = a.job.g.L, TB = a.job.g.TB;
    const bool batch = a.batch.jobs != nullptr;
    /* two CTAs share an SM (registers allow no more): the ring takes the
     * shared memory they leave */
    a.in_ring = 2u * zg_a16(zg_tile_worst(L, TB) + 15u);
    a.in_bytes = zg_a16(a.in_ring + (L == 32 ? zg_lane_slack() : zg_octet_slack(L))); /* and room for reads past a block's end */
    const uint32_t fixed = ADD_HEAD + a.in_bytes + 48u;
    a.ring = ring_bytes(2, fixed, zg_ring_bytes(L, TB));
    const size_t smem = fixed + a.ring;
    void (*fn)(const HomAddArgs) = L == 32 ? (batch ? k_homadd<true, true> : k_homadd<true, false>)
                                           : (batch ? k_homadd<false, true> : k_homadd<false, false>);
    const cudaError_t e = set_max_smem((const void *)fn, smem);
    if (e != cudaSuccess) return e;
    const uint64_t tiles = batch ? a.batch.ntiles : a.job.g.ntiles;
    const unsigned grid = scanned_grid((const void *)fn, ADD_THREADS, smem, tiles, a.grid);
    fn<<<grid, ADD_THREADS, smem, st>>>(a);
    return cudaGetLastError();
}
