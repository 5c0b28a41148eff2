/*
 * zk_decompress.cu -- decompressor.
 *
 * Replaces ZCCL_float_decompress_openmp_threadblock_arg
 * (ZCCL/src/ZCCLd_float.c:538-754) and produces the same floats, for one
 * stream or a batch of them, written or added to the destination (the DOC
 * reduce step's decompress-then-add, ZCCL/src/ZCCL_ring.c:1074-1076, in one
 * pass with one rounding per sum).
 *
 * The side index holds, for every group of blocks, the quantized value
 * before it, so groups are independent.  CTA c takes tiles c, c + grid, ...
 * A producer warp does the work that is the same for a whole tile: its
 * geometry, its blocks' widths and offsets (from the width index, requested
 * a tile ahead), and one TMA bulk copy of its bytes.  Eight consumer warps
 * take a group of the tile each, with no barrier and no wait on each other:
 *   1. every lane decodes its block (sign bits, high bytes, low-bit stream,
 *      ZCCL/src/ZCCL_TypeManager.c:423-950) into running sums, and a warp
 *      scan of the blocks' sums restores the running values
 *      (ZCCLd_float.c:617-628);
 *   2. x = (float)q * eb (ZCCLd_float.c:624) goes through shared memory at
 *      the destination's 16-byte phase and out in whole vectors.
 * Groups with a short block, a block of another length than 32, the
 * fixed-byte layout or a width above 15 go eight elements a lane instead
 * (decode_octet).
 * A stream that arrived as bytes gets its groups' starting values first: the
 * same kernel in its SUMS form writes every group's delta sum into the
 * index, and k_qprev_scan turns them, segment by segment, into starting
 * values from the segment's raw head.
 */
#include <cudaTypedefs.h>

#include <mutex>

#include "zkern.cuh"

namespace {

constexpr uint32_t DEC_WARPS = ZG_SUB;            /* consumer warps */
constexpr uint32_t DEC_THREADS = 32 * DEC_WARPS + 32; /* and the producer */

/* A staged tile, written by the producer before its copy's barrier fires. */
struct DTile {
    uint64_t tile;    /* ZP_NONE: no more tiles */
    float *y;         /* the tile's first block's first element */
    int32_t *qout;    /* SUMS: the tile's groups' index entries */
    uint32_t nblk, nlast, head;
    uint32_t fmt, body; /* first block's place in shared memory, from the input buffer's start */
    float eb;
    uint32_t acc, pad;
    uint32_t q0[ZG_SUB]; /* the value before each group */
};

struct DShared {
    uint64_t full[2], empty[2];
    DTile t[2];
    uint32_t ent[2][256]; /* per block: offset from body << 8 | width */
};
constexpr uint32_t DEC_HEAD = (sizeof(DShared) + 127u) / 128u * 128u;

/* The producer warp.  The two tiles in flight share the input buffer, one
 * at its start and one at its end (typical tiles are far below the largest,
 * so two fit; one that does not waits for the other to be decoded). */
template <bool L32, bool BATCH, bool QPREV>
__device__ __forceinline__ void produce(const DecompressArgs &a, DShared *sh, uint8_t *buf, uint32_t room, uint32_t &bad)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t ntiles = BATCH ? a.batch.ntiles : a.job.g.ntiles;
    const DecompressJob *nj = nullptr; /* the requested tile: its job, geometry, index entries */
    ZTile nz;
    uint64_t nbase = 0;
    uint32_t nq = 0, nw[3] = {0, 0, 0};
    auto request = [&](uint64_t t) {
        uint64_t local = t;
        if (BATCH) nj = static_cast<const DecompressJob *>(a.batch.jobs) + batch_job(a.batch, t, &local);
        const DecompressJob &J = BATCH ? *nj : a.job;
        zg_tile(&J.g, local, &nz);
        nbase = J.idx.grp_off[nz.grp0];
        if (QPREV && (lane == 0 || (lane < ZG_SUB && lane * J.g.GB < nz.nblk))) nq = (uint32_t)J.idx.grp_qprev[nz.grp0 + lane];
        load_widths(J.idx.widths + nz.gblk0, nz.nblk, nw);
    };
    uint64_t t = blockIdx.x;
    if (t < ntiles) request(t);
    uint32_t ppos = 0, plen = 0; /* the previous tile's place */
    for (uint32_t seq = 0;; seq++, t += gridDim.x) {
        const uint32_t s = seq & 1u;
        if (t >= ntiles) {
            if (seq >= 2) mbar_wait(&sh->empty[s], ((seq >> 1) + 1u) & 1u, a.w.err);
            if (lane == 0) {
                sh->t[s].tile = ZP_NONE;
                mbar_arrive(&sh->full[s]);
            }
            return;
        }
        const DecompressJob &J = BATCH ? *nj : a.job;
        const ZTile z = nz;
        uint64_t base = nbase;
        const uint32_t wsh = widths_shift(J.idx.widths + nz.gblk0);
        const uint32_t q = nq, w0 = __funnelshift_r(nw[0], nw[1], wsh), w1 = __funnelshift_r(nw[1], nw[2], wsh);
        const uint32_t L = J.g.L;
        if (t + gridDim.x < ntiles) request(t + gridDim.x);

        const uint32_t nlast = z.nblk ? (uint32_t)(z.e_end - z.e_first) - (z.nblk - 1u) * L : 0u;
        const uint32_t fmt = J.g.fmt;
        uint4 e[2];
        const uint32_t total = tile_entries<L32>(L, fmt, z.nblk, nlast, w0, w1, e, bad) + (z.has_head ? 4u : 0u);
        const uint32_t len = ((uint32_t)((uintptr_t)(J.in + base) & 15u) + total + 15u) & ~15u; /* of the aligned superset */

        if (seq >= 2) mbar_wait(&sh->empty[s], ((seq >> 1) + 1u) & 1u, a.w.err); /* tile seq - 2 is decoded */
        uint32_t pos = 0;
        if (seq >= 1) {
            if (ppos == 0 ? plen + len <= room : len <= ppos)
                pos = ppos == 0 ? room - len : 0u;
            else /* no room beside it: wait for tile seq - 1 too */
                mbar_wait(&sh->empty[s ^ 1u], ((seq - 1u) >> 1) & 1u, a.w.err);
        }
        ppos = pos;
        plen = len;
        uint32_t nload = total;
        /* overflow-safe: base comes from the index and is not trusted */
        if (base > J.avail || total > J.avail - base) {
            bad |= ZERR_BOUNDS;
            nload = base < J.avail ? (uint32_t)min((uint64_t)total, J.avail - base) : 0u;
            if (base > J.avail) base = 0;
        }
        DTile &d = sh->t[s];
        if (lane < ZG_SUB) d.q0[lane] = q;
        uint4 *tab = reinterpret_cast<uint4 *>(&sh->ent[s][8u * lane]);
        tab[0] = e[0];
        tab[1] = e[1];
        if (lane == 0) {
            d.tile = t;
            d.y = J.y + z.e_first;
            d.qout = J.idx.grp_qprev + z.grp0;
            d.nblk = z.nblk;
            d.nlast = nlast;
            d.head = z.has_head;
            d.fmt = fmt;
            d.body = pos + (uint32_t)((uintptr_t)(J.in + base) & 15u) + (z.has_head ? 4u : 0u);
            d.eb = J.eb;
            d.acc = J.accumulate != 0;
        }
        __syncwarp();
        if (lane == 0) tma_load_superset(buf + pos, J.in + base, nload, &sh->full[s]);
    }
}

/* MODE 0: floats (or, by the job's flag, added floats); 1: only each
 * group's wrapped sum of deltas, into the index's grp_qprev. */
template <bool L32, int MODE, bool BATCH>
__global__ void __launch_bounds__(DEC_THREADS, 3) k_decompress(const __grid_constant__ DecompressArgs a)
{
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    DShared *sh = reinterpret_cast<DShared *>(smem);
    uint8_t *buf = smem + DEC_HEAD;
    const uint32_t L = L32 ? 32u : a.job.g.L, GB = L32 ? 32u : a.job.g.GB; /* one L for the whole batch */
    uint32_t bad = 0;
    /* The index walk ran to completion before this launch, so every CTA sees
     * the same word: after a failed walk no CTA touches the stream. */
    if (*(volatile const uint32_t *)a.w.walk_err) return;
    if (tid == 0) {
        mbar_init(&sh->full[0], 1);
        mbar_init(&sh->full[1], 1);
        mbar_init(&sh->empty[0], DEC_WARPS);
        mbar_init(&sh->empty[1], DEC_WARPS);
    }
    __syncthreads();
    if (warp == DEC_WARPS) {
        produce<L32, BATCH, MODE == 0>(a, sh, buf, a.room, bad);
        if (bad) atomicOr(a.w.err, bad);
        return;
    }

    float *stage = reinterpret_cast<float *>(buf + a.in_bytes) + warp * ((GB * L + 31u) / 32u * 32u);
    const uint32_t *sw = reinterpret_cast<const uint32_t *>(buf);
    const uint32_t rb = smem_u32(stage) + lane * 128u, x4 = (lane & 7u) << 4;
    const uint32_t sb = smem_u32(stage) + ((lane >> 3) << 7);
    const uint64_t max_tiles = BATCH ? a.batch.ntiles : a.job.g.ntiles;
    for (uint32_t seq = 0; seq <= max_tiles; seq++) { /* bounded even if a wait gave up */
        const uint32_t s = seq & 1u;
        mbar_wait(&sh->full[s], (seq >> 1) & 1u, a.w.err);
        const DTile &D = sh->t[s];
        if (D.tile == ZP_NONE) break;
        const uint32_t tb = D.nblk, b0 = warp * GB;
        const uint32_t nblk = tb > b0 ? min(GB, tb - b0) : 0u;
        const uint32_t nlast = b0 + nblk == tb ? D.nlast : L; /* elements of the group's last block */
        const uint32_t body = D.body, fmt = D.fmt, run0 = D.q0[warp];
        const bool head = warp == 0 && D.head, acc = D.acc != 0;
        const float eb = D.eb;
        int32_t *qout = MODE == 1 ? D.qout : nullptr;
        float *y = D.y + b0 * L;
        auto put = [&](float *at, float x) { *at = acc ? __fadd_rn(*at, x) : x; };
        uint32_t e = lane < nblk ? sh->ent[s][b0 + lane] : 0u;
        const uint32_t b = e & 0xFFu, o = body + (e >> 8);
        if (lane < nblk && buf[o] != b) bad |= ZERR_CORRUPT;
        uint32_t sum = 0;
        if (L32 && nblk == 32 && nlast == 32 && fmt == ZG_FASTMODE1 && __all_sync(0xffffffffu, b < 16)) {
            /* running values from the block's start, then one scan of the
             * blocks' sums.  In floats, which are exact while every value is
             * an integer below 2^24: the 32 magnitudes of a block move the
             * running value by less than 2^20, which leaves room for a
             * starting value below 2^23. */
            float v[32], f = 0.f;
            decode_small_f(sw, o, b, 32u, [&](int j, float m, uint32_t sg) {
                f += with_sign(m, sg, j);
                v[j] = f;
            });
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->empty[s]); /* this warp is done with the tile's bytes and entries */
            sum = (uint32_t)__float2int_rn(f);
            if (MODE == 0) {
                const uint32_t q0 = run0 + warp_incl_scan(sum) - sum;
                if (__all_sync(0xffffffffu, (uint32_t)abs((int32_t)q0) < (1u << 23))) {
                    const float f0 = __int2float_rn((int32_t)q0);
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] = __fmul_rn(__fadd_rn(v[j], f0), eb);
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        v[j] = __fmul_rn(__int2float_rn((int32_t)(q0 + (uint32_t)__float2int_rn(v[j]))), eb);
                }
                /* rows of 32 floats at the destination's phase p: the last p
                 * elements of the lane before, then this lane's; 16-byte
                 * chunk k of row r at chunk k ^ (r & 7), so neither these
                 * stores nor the reads below conflict */
                const uint32_t p = (uint32_t)((uintptr_t)y >> 2) & 3u;
                auto row = [&](int pc, float w0, float w1, float w2) {
                    auto u = [&](int j) { return j >= pc ? v[j - pc] : j == pc - 1 ? w0 : j == pc - 2 ? w1 : w2; };
#pragma unroll
                    for (int k = 0; k < 8; k++)
                        st_shared_v4(rb | (((uint32_t)k << 4) ^ x4), u(4 * k), u(4 * k + 1), u(4 * k + 2), u(4 * k + 3));
                };
                auto before = [&](float x) { return __shfl_up_sync(0xffffffffu, x, 1); };
                if (p == 1) /* uniform; first as the usual case: the element after a segment's head */
                    row(1, before(v[31]), 0.f, 0.f);
                else if (p == 0)
                    row(0, 0.f, 0.f, 0.f);
                else if (p == 2)
                    row(2, before(v[31]), before(v[30]), 0.f);
                else
                    row(3, before(v[31]), before(v[30]), before(v[29]));
                /* the first vector's elements from p on, and the p elements
                 * past the last vector */
                if (p && lane == 0) {
                    put(y, v[0]);
                    if (p < 3) put(y + 1, v[1]);
                    if (p < 2) put(y + 2, v[2]);
                }
                if (p && lane == 31) {
                    put(y + 1023, v[31]);
                    if (p > 1) put(y + 1022, v[30]);
                    if (p > 2) put(y + 1021, v[29]);
                }
                if (head && lane == 0) put(y - 1, __fmul_rn(__int2float_rn((int32_t)run0), eb));
                __syncwarp();
                float4 *y4 = reinterpret_cast<float4 *>(y - p) + lane;
                const bool first = !p || lane; /* vector 0 is ragged unless p == 0 */
                auto chunk = [&](uint32_t u) { /* vector lane + 32 u: chunk lane & 7 of row (lane >> 3) + 4 u */
                    return ld_shared_v4(sb + u * 512u + (((lane & 7u) ^ (((lane >> 3) + 4u * u) & 7u)) << 4));
                };
                if (!acc) {
#pragma unroll
                    for (uint32_t u = 0; u < 8; u++) {
                        const float4 x = chunk(u);
                        if (u || first) y4[32u * u] = x;
                    }
                } else {
#pragma unroll
                    for (uint32_t h = 0; h < 2; h++) {
                        float4 t[4];
#pragma unroll
                        for (uint32_t u = 0; u < 4; u++) /* the loads ahead of the stores */
                            t[u] = h || u || first ? y4[128u * h + 32u * u] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (uint32_t u = 0; u < 4; u++) {
                            const float4 x = chunk(4u * h + u);
                            t[u].x = __fadd_rn(t[u].x, x.x);
                            t[u].y = __fadd_rn(t[u].y, x.y);
                            t[u].z = __fadd_rn(t[u].z, x.z);
                            t[u].w = __fadd_rn(t[u].w, x.w);
                            if (h || u || first) y4[128u * h + 32u * u] = t[u];
                        }
                    }
                }
                __syncwarp(); /* the stage is free again */
            }
        } else {
            /* G = ceil(L / 8) lanes share a block, BPI blocks at a time */
            const uint32_t G = L32 ? 4u : (L + 7u) / 8u, BPI = 32u / G;
            const uint32_t og = lane % G, bi = lane / G;
            uint32_t run = run0;
#pragma unroll 1
            for (uint32_t k0 = 0; k0 < nblk; k0 += BPI) {
                const uint32_t k = k0 + bi;
                const bool has = bi < BPI && k < nblk;
                e = has ? sh->ent[s][b0 + k] : 0u;
                const uint32_t n = !has ? 0u : k + 1 < nblk ? L : nlast;
                uint32_t d[8];
                decode_octet(sw, body + (e >> 8), e & 0xFFu, n, og, fmt, d);
                uint32_t tot = 0;
#pragma unroll
                for (int j = 0; j < 8; j++) tot += d[j];
                if (MODE == 1) {
                    sum += tot;
                    continue;
                }
                const uint32_t incl = warp_incl_scan(tot);
                uint32_t q = run + incl - tot;
                run += __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    q += d[j];
                    if (8u * og + (uint32_t)j < n)
                        stage[k * L + 8u * og + (uint32_t)j] = __fmul_rn(__int2float_rn((int32_t)q), eb);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->empty[s]);
            if (MODE == 0) {
                if (head && lane == 0) put(y - 1, __fmul_rn(__int2float_rn((int32_t)run0), eb));
                const uint32_t cnt = nblk ? (nblk - 1u) * L + nlast : 0u;
                for (uint32_t i0 = lane; i0 < cnt; i0 += 256) { /* eight in flight */
                    float t[8];
#pragma unroll
                    for (uint32_t u = 0; u < 8; u++) t[u] = acc && i0 + 32u * u < cnt ? y[i0 + 32u * u] : 0.f;
#pragma unroll
                    for (uint32_t u = 0; u < 8; u++)
                        if (i0 + 32u * u < cnt) {
                            const float x = stage[i0 + 32u * u];
                            y[i0 + 32u * u] = acc ? __fadd_rn(t[u], x) : x;
                        }
                }
                __syncwarp();
            }
        }
        if (MODE == 1) {
            sum = __reduce_add_sync(0xffffffffu, sum);
            if (lane == 0 && (nblk || head)) qout[warp] = (int32_t)sum;
        }
    }
    if (bad) atomicOr(a.w.err, bad);
}

/* One CTA per segment: its groups' delta sums (from k_decompress in its SUMS
 * form) become the quantized value before each group, starting from the
 * segment's raw int32 head (the four bytes at its first group's offset) and
 * wrapping like the reference's int32 running value (ZCCLd_float.c:582-628).
 * Four groups a thread and one scan over the CTA a round: a segment of 64M
 * floats is 16 rounds (a warp per segment took 2048 steps of one load's
 * latency each). */
__global__ void __launch_bounds__(1024) k_qprev_scan(const __grid_constant__ DecompressArgs a)
{
    __shared__ uint32_t ws[33];
    const DecompressJob &J = a.job;
    const ZGeom &g = J.g;
    const uint64_t seg = blockIdx.x;
    if (*(volatile const uint32_t *)a.w.walk_err) return;
    const uint64_t g0 = seg * g.gr_reg;
    const uint64_t ng = seg < g.T ? g.gr_reg : g.ngroups - (uint64_t)g.T * g.gr_reg;
    const uint64_t off = J.idx.grp_off[g0];
    uint32_t run = 0;
    if (off <= J.avail && J.avail - off >= 4) {
#pragma unroll
        for (int k = 0; k < 4; k++) run |= (uint32_t)J.in[off + k] << (8 * k);
    } else if (threadIdx.x == 0) {
        atomicOr(a.w.err, ZERR_BOUNDS);
    }
    for (uint64_t k0 = 0; k0 < ng; k0 += 4ull * blockDim.x) {
        const uint64_t k = k0 + 4ull * threadIdx.x;
        uint32_t v[4], s = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            v[i] = k + i < ng ? (uint32_t)J.idx.grp_qprev[g0 + k + i] : 0u;
            s += v[i];
        }
        uint32_t tot;
        uint32_t pre = run + cta_excl_scan(s, ws, &tot);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (k + i < ng) J.idx.grp_qprev[g0 + k + i] = (int32_t)pre;
            pre += v[i];
        }
        run += tot;
    }
}

/* cuTensorMapEncodeTiled from the driver, looked up once. */
PFN_cuTensorMapEncodeTiled_v12000 encode_tiled()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        else
            cudaGetLastError();
    });
    return fn;
}

} // namespace

bool zk_rows_map(CUtensorMap *map, const void *p, uint64_t n)
{
    const uint64_t before = ((uintptr_t)p & 15u) / 4u, nrows = (n + before) / 32u;
    if (((uintptr_t)p & 3u) || nrows < 256u || nrows > 0x7fffffffull) return false;
    PFN_cuTensorMapEncodeTiled_v12000 enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t dim[2] = {32u, nrows};
    const cuuint64_t stride[1] = {128u};
    const cuuint32_t box[2] = {32u, 32u};
    const cuuint32_t estride[2] = {1u, 1u};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(static_cast<const float *>(p) - before), dim, stride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_decompress(const DecompressArgs &a0, cudaStream_t st)
{
    DecompressArgs a = a0;
    const uint32_t L = a.job.g.L, GB = a.job.g.GB;
    /* two typical tiles (at least one of the largest), room for the reads
     * past a tile's end, and the floats */
    a.room = zg_a16(zg_tile_worst(L, a.job.g.TB) + 15u);
    a.in_bytes = (a.room + zg_octet_slack(L) + 127u) / 128u * 128u;
    const size_t smem = DEC_HEAD + a.in_bytes + DEC_WARPS * ((GB * L + 31u) / 32u * 128u);
    const bool batch = a.batch.jobs != nullptr;
    const uint64_t tiles = batch ? a.batch.ntiles : a.job.g.ntiles;
    auto launch = [&](void (*k)(const DecompressArgs)) -> cudaError_t {
        const cudaError_t e = set_max_smem((const void *)k, smem);
        if (e != cudaSuccess) return e;
        unsigned grid = persistent_grid((const void *)k, DEC_THREADS, smem, tiles);
        if (a.grid && a.grid < grid) grid = a.grid;
        k<<<grid, DEC_THREADS, smem, st>>>(a);
        return cudaGetLastError();
    };
    /* a stream without starting values: group sums, then the scan per segment */
    if (!a.qprev_valid) {
        cudaError_t e = launch(L == 32 ? k_decompress<true, 1, false> : k_decompress<false, 1, false>);
        if (e != cudaSuccess) return e;
        const unsigned nseg = a.job.g.T + (a.job.g.rem ? 1u : 0u);
        const uint64_t most = a.job.g.gr_reg; /* groups of a segment (the extra one has fewer than T elements) */
        const unsigned threads = most >= 4096 ? 1024u : (unsigned)((most + 127) / 128 * 32);
        k_qprev_scan<<<nseg, threads < 32 ? 32 : threads, 0, st>>>(a);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (batch) return launch(L == 32 ? k_decompress<true, 0, true> : k_decompress<false, 0, true>);
    return launch(L == 32 ? k_decompress<true, 0, false> : k_decompress<false, 0, false>);
}
