/*
 * zk_walk.cu -- side-index builder for streams that arrive as bytes only
 * (written by the reference, or by any writer that did not keep the index).
 *
 * The wire format has no block index: inside a chunk, block k starts where
 * block k-1 ends, and only its 1-byte width header says how long it is
 * (ZCCL/src/ZCCLd_float.c:598-614).  Walking the headers is a chain of
 * dependent loads as long as the chunk, so it is split into windows of WW
 * bytes and done in parallel, exactly:
 *
 *   W0  chunk starts from the T-entry header; per segment its block region
 *       and window count; heads' tile offsets.
 *   W1  for every window and every possible entry offset e in [0, M) (M = the
 *       largest block): the exit offset into the next window and the blocks
 *       passed.  A byte above 32 cannot be a header, so a walk that meets one
 *       is dead, and of the walks that start inside a block nearly all are
 *       within a few steps: every entry is followed that far, the survivors
 *       are gathered and followed to the window's end.
 *   W2  compose the tables: per group of G windows (parallel), then per
 *       segment across groups, giving each group its true entry offset and
 *       first block number.
 *   W3  per window, one lane follows the path from its true entry and lists
 *       its blocks; all lanes write their widths and every group's offset;
 *       each chunk must end where the next starts.
 *   W4  the extra segment of the last chunk (N % T elements) and the total
 *       size.
 * Widths above 32, chunk ends that disagree with the header, and blocks past
 * the readable bytes set ZERR_CORRUPT / ZERR_BOUNDS instead of faulting.
 */
#include "zkern.cuh"

namespace {

constexpr uint32_t WARPS_W1 = 8;
constexpr uint32_t WARPS_W3 = 8; /* warps per CTA in W3, a window each at a time */
constexpr uint32_t DEAD = 0xFFFFFFFFu; /* an entry whose walk meets a byte that is no header */
constexpr uint64_t DEAD_GROUP = 1ull << 63; /* the same in a group's table, with the windows entered */

__device__ __forceinline__ uint64_t load_u64(const uint8_t *p)
{
    uint64_t v = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) v |= (uint64_t)p[k] << (8 * k);
    return v;
}

/* Size of a full block whose header byte is b <= 32. */
__device__ __forceinline__ uint32_t full_size(uint32_t b, uint32_t L, uint32_t fmt)
{
    return zg_block_bytes_f(fmt, b, L);
}

/* full_size on a walk's critical path: for 32-element fastmode1 blocks
 * (header, four sign bytes, 4 b bytes of magnitudes; a zero-width block is
 * its header alone) two operations instead of the general formula. */
struct Sizer {
    uint32_t L, fmt, fast;
    __device__ __forceinline__ Sizer(uint32_t L_, uint32_t fmt_)
        : L(L_), fmt(fmt_), fast(L_ == 32u && fmt_ == ZG_FASTMODE1) {}
    __device__ __forceinline__ uint32_t operator()(uint32_t b) const
    {
        if (fast) return b ? 4u * b + 5u : 1u;
        return full_size(b, L, fmt);
    }
};

/* Segment of a window / group index: last s with base[s] <= i, by all lanes,
 * 32 parts of what is left a step (131072 chunks of 64 floats, from wire bytes:
 * 4.5 ms; by halves 25, 32 bases a step from the first on 105). */
__device__ __forceinline__ uint32_t find_seg(const uint32_t *base, uint32_t T, uint32_t i)
{
    uint32_t lo = 0, n = T; /* base[lo] <= i; the last such is in [lo, lo + n) */
    while (n > 1) {
        const uint32_t part = (n + 31u) / 32u, at = (threadIdx.x & 31u) * part;
        const uint32_t k = __popc(__ballot_sync(0xffffffffu, at < n && base[lo + at] <= i)) - 1u; /* lane 0's is */
        lo += k * part;
        n = min(part, n - k * part);
    }
    return lo;
}

/* ---- W0 -------------------------------------------------------------- */
__global__ void k_walk_setup(const WalkArgs a)
{
    const ZGeom &g = a.g;
    const WalkScratch &w = a.ws;
    const uint64_t hdr = zg_header_bytes(&g);
    __shared__ uint32_t wsum[33];
    uint32_t carry_w = 0, carry_g = 0;
    for (uint32_t s0 = 0; s0 < g.T; s0 += blockDim.x) {
        const uint32_t s = s0 + threadIdx.x;
        uint32_t nwin = 0;
        if (s < g.T) {
            uint64_t P, R, rel = 0, next = 0;
            if (hdr <= a.avail) {
                rel = load_u64(a.in + 8ull * s);
                if (s + 1 < g.T) next = load_u64(a.in + 8ull * (s + 1));
            }
            const uint32_t bad = walk_chunk(&g, s, rel, next, a.avail, a.end_bound, &P, &R);
            bool ok = !bad;
            if (bad) atomicOr(a.err, bad);
            if (ok) a.idx.grp_off[(uint64_t)s * g.gr_reg] = hdr + rel;
            if (ok && g.nb_reg > 0) nwin = walk_windows(P, R);
            if (ok && g.nb_reg > 0 && nwin == 0) {
                atomicOr(a.err, ZERR_BOUNDS);
                ok = false;
            }
            w.seg_P[s] = P;
            w.seg_R[s] = R;
            w.seg_end[s] = (ok && g.nb_reg == 0) ? P : 0;
            w.seg_ok[s] = ok ? 1u : 0u;
            if (ok && g.nb_reg == 0 && s + 1 < g.T && P != R) atomicOr(a.err, ZERR_CORRUPT);
        }
        uint32_t tot_w, tot_g;
        uint32_t bw = cta_excl_scan(nwin, wsum, &tot_w);
        uint32_t bg = cta_excl_scan((nwin + a.G - 1) / a.G, wsum, &tot_g);
        if (s < g.T) {
            w.win_base[s] = carry_w + bw;
            w.grp_base[s] = carry_g + bg;
        }
        carry_w += tot_w;
        carry_g += tot_g;
    }
    if (threadIdx.x == 0) {
        w.win_base[g.T] = carry_w;
        w.grp_base[g.T] = carry_g;
    }
}

/* Bytes of a warp's window area: the window and the M bytes after it, with
 * alignment slack; and then a bit for every 16-byte line of it. */
__host__ __device__ inline uint32_t win_lines(uint32_t M) { return (WALK_WW + M + 32u + 15u) & ~15u; }
__host__ __device__ inline uint32_t win_area(uint32_t M) { return win_lines(M) + ((win_lines(M) / 512u + 1u) * 4u + 15u & ~15u); }

/* A window in a warp's area, loaded. */
struct Window {
    uint32_t at, buf; /* shared addresses of its first byte and of the area */
    uint32_t bits;    /* of the lines' bits, set where a line is not all zero; 0: no line is */
    bool zeros;       /* every line is zero (sparse data: zero-width blocks) */
};

/* The window [start, start + WW + M) of the stream into the 16-byte-aligned
 * area (bytes past avail read as 0xFF, no header), by aligned 16-byte loads that the
 * warp issues together. */
__device__ __forceinline__ Window load_window(const WalkArgs &a, uint64_t start, uint8_t *area)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uintptr_t base = reinterpret_cast<uintptr_t>(a.in), end = base + a.avail;
    const uintptr_t lo = (base + start) & ~(uintptr_t)15;
    const uint32_t ph = (uint32_t)(base + start - lo), nl = (ph + WALK_WW + a.M + 15u) / 16u;
    uint4 *d = reinterpret_cast<uint4 *>(area);
    uint32_t any = 0;
    bool gap = false; /* a zero line */
#pragma unroll 8
    for (uint32_t i = lane; i < nl; i += 32) {
        const uintptr_t p = lo + 16u * i;
        uint32_t o;
        if (p >= base && p + 16u <= end) {
            const uint4 v = *reinterpret_cast<const uint4 *>(p);
            d[i] = v;
            o = v.x | v.y | v.z | v.w;
        } else { /* a line across either end of the readable bytes */
            uint32_t v[4] = {~0u, ~0u, ~0u, ~0u};
            for (uint32_t k = 0; k < 16; k++) {
                const uintptr_t q = p + k;
                if (q >= base && q < end)
                    v[k >> 2] ^= (uint32_t)(uint8_t)~*reinterpret_cast<const uint8_t *>(q) << (8 * (k & 3));
            }
            d[i] = make_uint4(v[0], v[1], v[2], v[3]);
            o = v[0] | v[1] | v[2] | v[3];
        }
        any |= o;
        gap |= o == 0;
    }
    Window w;
    w.buf = smem_u32(area);
    w.at = w.buf + ph;
    w.zeros = !__any_sync(0xffffffffu, any != 0);
    w.bits = 0;
    if (__any_sync(0xffffffffu, gap) && !w.zeros) {
        uint32_t *bits = reinterpret_cast<uint32_t *>(area + win_lines(a.M));
        w.bits = smem_u32(bits);
        for (uint32_t i0 = 0; i0 < nl; i0 += 32) { /* each lane reads what it wrote */
            const uint4 v = i0 + lane < nl ? d[i0 + lane] : make_uint4(0, 0, 0, 0);
            const uint32_t m = __ballot_sync(0xffffffffu, (v.x | v.y | v.z | v.w) != 0);
            if (lane == 0) bits[i0 / 32u] = m;
        }
    }
    __syncwarp();
    return w;
}

/* One thread, at a zero byte, number pos of a window that has lines of zeros:
 * how many zeros they show from there on, up to byte `end`; 1 if its line is none. */
__device__ __forceinline__ uint32_t zero_run(const Window &w, uint32_t pos, uint32_t end)
{
    const uint32_t a = w.at + pos - w.buf, l = a >> 4, last = (w.at + end - w.buf + 15u) >> 4; /* lines that matter */
    uint32_t k = l >> 5, m = ld_shared_u32(w.bits + 4u * k) >> (l & 31u) << (l & 31u);
    while (!m && 32u * (k + 1u) < last) m = ld_shared_u32(w.bits + 4u * ++k);
    const uint32_t next = m ? 32u * k + (uint32_t)__ffs(m) - 1u : last; /* the next line that is not zero */
    return next == l ? 1u : min(16u * next - a, end - pos);
}

/* ---- W1 --------------------------------------------------------------
 * Per window, the walk of every entry offset e < M: where it leaves the
 * window (offset into the next) << 16 | blocks passed, or DEAD.  Walks from
 * inside a block die on the first byte above 32 (a random byte is a header
 * once in eight) or run into another walk's path.  So all entries first walk
 * to the end of their first HEAD bytes; one walk per distinct place where
 * they left goes on, a lane each, to the window's end.  A window of zeros
 * (sparse data: zero-width blocks) is its own answer.  What is left is the
 * chain of dependent shared loads of about as many steps as the window has
 * blocks, in few instructions each.  Per warp: the window, then per place a
 * flag and a result.
 * In windows that have lines of zeros, their blocks go at once: a field of 1M
 * zeros, whose windows end in such a stretch, 150 us for the whole walk with a
 * step a block here and in W3, 62 so (a pass over every position, 80).
 * 64M floats' 77 MB of signal data: 76 us, bound by issue (a window's few
 * long walks leave most lanes of their warp idle); a backward pass over every
 * position of every window, which this replaces, took 176.  A stream of 0.6 MB:
 * 15 us against 23; windows of 4096 bytes 64 / 23, four windows a warp in turn
 * 216 / 75. */
constexpr uint32_t HEAD = 128, HEAD_DEAD = WALK_WW - 1; /* HEAD + M - 1 < HEAD_DEAD */

__host__ __device__ inline uint32_t w1_warp_bytes(uint32_t M) { return win_area(M) + ((6u * M + 15u) & ~15u); }

/* One thread: the walk of a window from pos to its end: where it leaves it
 * (offset into the next) << 16 | its blocks, or DEAD. */
__device__ __forceinline__ uint32_t walk_out(uint32_t win, uint32_t pos, const Sizer &size)
{
    uint32_t cnt = 0;
    while (pos < WALK_WW) {
        const uint32_t b = ld_shared_u8(win + pos);
        if (b > 32u) return DEAD;
        pos += size(b);
        cnt++;
    }
    return (pos - WALK_WW) << 16 | cnt;
}

/* The same in a window that has lines of zeros: their zero-width blocks at once. */
__device__ __noinline__ uint32_t walk_out_runs(Window w, uint32_t pos, Sizer size)
{
    uint32_t cnt = 0;
    while (pos < WALK_WW) {
        const uint32_t b = ld_shared_u8(w.at + pos);
        if (b > 32u) return DEAD;
        const uint32_t n = b ? 1u : zero_run(w, pos, WALK_WW);
        pos += b ? size(b) : n;
        cnt += n;
    }
    return (pos - WALK_WW) << 16 | cnt;
}

__global__ void __launch_bounds__(32 * WARPS_W1) k_walk_tables(const WalkArgs a)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const ZGeom &g = a.g;
    const WalkScratch &w = a.ws;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t M = a.M;
    const Sizer size(g.L, g.fmt);
    uint8_t *area = smem + warp * a.w1_warp_bytes;
    uint32_t *fin = reinterpret_cast<uint32_t *>(area + win_area(M)); /* [M] */
    uint16_t *list = reinterpret_cast<uint16_t *>(fin + M);            /* [M] distinct places, less HEAD */
    const uint32_t nwin = w.win_base[g.T];
    /* persistent: the warps stride over the windows the header gives */
    for (uint32_t wg = blockIdx.x * WARPS_W1 + warp; wg < nwin; wg += gridDim.x * WARPS_W1) {
        const uint32_t s = find_seg(w.win_base, g.T, wg);
        const uint64_t start = w.seg_P[s] + (uint64_t)(wg - w.win_base[s]) * WALK_WW;
        const Window w1 = load_window(a, start, area);
        const uint32_t win = w1.at;
        uint32_t *tab = a.ws.wtab + (uint64_t)wg * M;
        if (w1.zeros) { /* a block a byte */
            for (uint32_t e = lane; e < M; e += 32) tab[e] = WALK_WW - e;
            continue;
        }
        for (uint32_t x = lane; x < M; x += 32) fin[x] = 0;
        __syncwarp();
        /* the first HEAD bytes, four entries a lane at a time so that their
         * loads overlap: entry e's place and count wait in its table word,
         * and the place is flagged */
        for (uint32_t e0 = lane; e0 < M; e0 += 128) {
            uint32_t pos[4], cnt[4], b[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t e = e0 + 32u * (uint32_t)k;
                pos[k] = e < M ? e : HEAD;
                cnt[k] = 0;
            }
            bool more = true;
            while (more) {
#pragma unroll
                for (int k = 0; k < 4; k++) b[k] = ld_shared_u8(win + pos[k]);
                more = false;
#pragma unroll
                for (int k = 0; k < 4; k++) { /* past HEAD, or DEAD (all ones, far past it): no step */
                    if (pos[k] < HEAD) {
                        pos[k] = b[k] > 32u ? HEAD_DEAD : pos[k] + size(b[k]);
                        cnt[k]++;
                        more |= pos[k] < HEAD;
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t e = e0 + 32u * (uint32_t)k;
                if (e < M) {
                    tab[e] = pos[k] == HEAD_DEAD ? DEAD : pos[k] << 16 | cnt[k];
                    if (pos[k] != HEAD_DEAD) fin[pos[k] - HEAD] = 1; /* < M: a block, or an entry, past HEAD - 1 */
                }
            }
        }
        __syncwarp();
        uint32_t n = 0;
        for (uint32_t x0 = 0; x0 < M; x0 += 32) {
            const uint32_t x = x0 + lane;
            const bool f = x < M && fin[x];
            const uint32_t m = __ballot_sync(0xffffffffu, f);
            if (f) list[n + __popc(m & ((1u << lane) - 1u))] = (uint16_t)x;
            n += __popc(m);
        }
        __syncwarp();
        if (w1.bits)
            for (uint32_t i = lane; i < n; i += 32) fin[list[i]] = walk_out_runs(w1, HEAD + list[i], size);
        else
            for (uint32_t i = lane; i < n; i += 32) fin[list[i]] = walk_out(win, HEAD + list[i], size);
        __syncwarp();
        for (uint32_t e = lane; e < M; e += 32) {
            const uint32_t t = tab[e];
            if (t != DEAD) {
                const uint32_t f = fin[(t >> 16) - HEAD];
                tab[e] = f == DEAD ? DEAD : f + (t & 0xFFFFu); /* the count in the low 16 bits stays below 2^16 */
            }
        }
        __syncwarp(); /* the area is reused for the next window */
    }
}

/* ---- W2a: compose the window tables of each group ----------------------
 * For every entry offset into the group, the walk through its windows'
 * tables; each step's entry offset and the blocks passed before it are kept
 * (gwin), so that once the group's true entry is known every window's is a
 * single load.  A walk that dies leaves the number of windows it entered.
 * From shared copies of the tables 15 us for 77 MB; from global memory, a
 * dependent load a step, 29. */
__global__ void __launch_bounds__(1024) k_walk_groups(const WalkArgs a)
{
    extern __shared__ __align__(16) uint32_t tabs[]; /* the group's window tables */
    const ZGeom &g = a.g;
    const WalkScratch &w = a.ws;
    const uint32_t gg = blockIdx.x;
    if (gg >= w.grp_base[g.T]) return;
    const uint32_t s = find_seg(w.grp_base, g.T, gg);
    const uint32_t nwin = w.win_base[s + 1] - w.win_base[s];
    const uint32_t w0 = (gg - w.grp_base[s]) * a.G;
    const uint32_t w1 = min(w0 + a.G, nwin);
    /* one coalesced copy, so that the walks' dependent steps read shared memory */
    const uint32_t *gt = w.wtab + (uint64_t)(w.win_base[s] + w0) * a.M;
#pragma unroll 8
    for (uint32_t i = threadIdx.x; i < (w1 - w0) * a.M; i += blockDim.x) tabs[i] = __ldg(gt + i);
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < a.M; e += blockDim.x) {
        uint32_t x = e, c = 0, k = 0;
        uint32_t *gw = w.gwin + ((uint64_t)gg * a.M + e) * a.G;
        for (; k < w1 - w0 && x != DEAD; k++) {
            gw[k] = c << 12 | x; /* c <= 64 windows x 2048 blocks; x < M < 4096 */
            const uint32_t t = tabs[k * a.M + x];
            x = t == DEAD ? DEAD : t >> 16;
            c += t & 0xFFFFu;
        }
        w.gtab[(uint64_t)gg * a.M + e] = x == DEAD ? DEAD_GROUP | k : (uint64_t)c << 32 | x;
    }
}

/* ---- W2b: per segment, carry the entry offset across its groups --------
 * A dead walk ends the segment's blocks (past its last block the bytes need
 * be no headers) or is a corrupt stream, which W3 and W4 tell apart: the
 * groups after it are marked as past every block. */
__global__ void __launch_bounds__(1024) k_walk_segments(const WalkArgs a)
{
    extern __shared__ __align__(16) uint8_t smem[];
    uint64_t *rows = reinterpret_cast<uint64_t *>(smem);
    __shared__ uint64_t s_base;
    __shared__ uint32_t s_x;
    const ZGeom &g = a.g;
    const WalkScratch &w = a.ws;
    const uint32_t s = blockIdx.x;
    if (!w.seg_ok[s]) return;
    const uint32_t g0 = w.grp_base[s], g1 = w.grp_base[s + 1];
    uint32_t x = 0;
    uint64_t base = 0;
    for (uint32_t b0 = g0; b0 < g1; b0 += a.seg_batch) {
        const uint32_t nb = min(a.seg_batch, g1 - b0);
        if (base < g.nb_reg) /* groups past the last block need no table */
            for (uint32_t i = threadIdx.x; i < nb * a.M; i += blockDim.x)
                rows[i] = w.gtab[(uint64_t)b0 * a.M + i];
        __syncthreads();
        if (threadIdx.x == 0) {
            for (uint32_t j = 0; j < nb; j++) {
                uint32_t enter = x | a.G << 16; /* and the windows of the group that the path enters */
                w.gbase[b0 + j] = base;
                if (base < g.nb_reg) {
                    const uint64_t t = rows[j * a.M + x];
                    if (t & DEAD_GROUP) {
                        enter = x | (uint32_t)t << 16;
                        base = ~0ull;
                    } else {
                        base += t >> 32;
                        x = (uint32_t)t;
                    }
                }
                w.gentry[b0 + j] = enter;
            }
            s_base = base;
            s_x = x;
        }
        __syncthreads();
        base = s_base;
        x = s_x;
    }
}

/* ---- W3: the true walk of every window -------------------------------
 * One warp per window: its true entry and first block are one load (gwin at
 * its group's true entry); lane 0 follows the headers from the entry and
 * lists where they are, PATH at a time, and all lanes write the blocks' widths
 * (neighbouring bytes) and group offsets.  Lines of zeros, one zero-width block a
 * byte, need no list.  Shared bytes per warp: the window,
 * the list.  64M floats' 77 MB: 66 us; a stream of 0.6 MB: 12 us, against 18
 * with a lane per 128-byte part of the window. */
constexpr uint32_t PATH = 256;

__host__ __device__ inline uint32_t w3_warp_bytes(uint32_t M) { return win_area(M) + 2u * PATH; }

/* One thread, in a window that has lines of zeros: the next headers, up to and
 * with a byte that is none or up to a line of zeros, at most PATH of them, into
 * the list: the position behind them and their number; or, where such a line
 * starts at pos, pos and 1 << 16 | the zeros from there on. */
__device__ __noinline__ uint2 list_runs(Window w, uint32_t pos, uint32_t list, Sizer size)
{
    uint32_t n = 0, b = 0;
    while (pos < WALK_WW && n < PATH && b <= 32u) {
        b = ld_shared_u8(w.at + pos);
        if (b == 0) {
            const uint32_t z = zero_run(w, pos, WALK_WW);
            if (z > 1u) return make_uint2(pos, n ? n : 1u << 16 | z);
        }
        st_shared_u16(list + 2u * n, pos);
        n++;
        pos += size(min(b, 32u));
    }
    return make_uint2(b > 32u ? WALK_WW : pos, n);
}

__global__ void __launch_bounds__(32 * WARPS_W3, 6) k_walk_final(const WalkArgs a)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const ZGeom &g = a.g;
    const WalkScratch &w = a.ws;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const Sizer size(g.L, g.fmt);
    const uint64_t nb = g.nb_reg;
    const uint64_t nfull = (g.tbs - 1) / g.L;
    const uint32_t ntail = (uint32_t)((g.tbs - 1) % g.L);
    uint8_t *area = smem + warp * w3_warp_bytes(a.M);
    const uint32_t list = smem_u32(area + win_area(a.M)); /* u16[PATH] */
    /* persistent: the warps stride over the windows the header gives */
    for (uint32_t wi = blockIdx.x * nw + warp; wi < w.win_base[g.T]; wi += gridDim.x * nw) {
        const uint32_t s = find_seg(w.win_base, g.T, wi);
        if (!w.seg_ok[s]) continue; /* uniform over the warp */
        const uint32_t k = wi - w.win_base[s]; /* the window within its segment */
        const uint32_t gg = w.grp_base[s] + k / a.G;
        const uint32_t enter = w.gentry[gg];
        const uint64_t gb = w.gbase[gg];
        if (gb >= nb || k % a.G >= enter >> 16) continue; /* uniform */
        const uint32_t v = w.gwin[((uint64_t)gg * a.M + (enter & 0xFFFFu)) * a.G + k % a.G];
        uint64_t blk0 = gb + (v >> 12); /* the window's first block, then the list's */
        if (blk0 >= nb) continue;
        const uint64_t gblk0 = (uint64_t)s * g.nb_reg, grp0 = (uint64_t)s * g.gr_reg;
        const uint64_t start = w.seg_P[s] + (uint64_t)k * WALK_WW;
        const Window win = load_window(a, start, area);
        uint32_t pos = v & 0xFFFu; /* lane 0's walk */
        while (blk0 < nb) {
            /* the next headers, up to and with a byte that is none; or a run of zeros, which needs no list */
            uint32_t n = 0; /* 1 << 16 | blocks: a run */
            if (win.zeros) {
                n = 1u << 16 | (WALK_WW - pos);
            } else if (lane == 0) {
                if (win.bits) {
                    const uint2 r = list_runs(win, pos, list, size);
                    pos = r.x;
                    n = r.y;
                } else {
                    uint32_t b = 0;
                    while (pos < WALK_WW && n < PATH && b <= 32u) {
                        b = ld_shared_u8(win.at + pos);
                        st_shared_u16(list + 2u * n, pos);
                        n++;
                        pos += size(min(b, 32u));
                    }
                    if (b > 32u) pos = WALK_WW;
                }
            }
            n = __shfl_sync(0xffffffffu, n, 0);
            const bool run = n >> 16;
            n &= 0xFFFFu;
            const uint32_t from = __shfl_sync(0xffffffffu, pos, 0); /* the run's first byte */
            __syncwarp();
            if (n == 0) break;
            const uint64_t q = (blk0 + lane) >> 32 ? (blk0 + lane) / g.GB : (uint32_t)(blk0 + lane) / g.GB;
            uint32_t in_grp = (uint32_t)(blk0 + lane - q * g.GB);
            uint64_t grp = grp0 + q;
            for (uint32_t i = lane; i < n; i += 32) {
                const uint64_t blk = blk0 + i;
                const uint32_t p = run ? from + i : ld_shared_u16(list + 2u * i);
                if (blk < nb) {
                    const uint64_t gpos = start + p;
                    const uint32_t b = ld_shared_u8(win.at + p);
                    if (gpos >= a.avail) {
                        atomicOr(a.err, ZERR_BOUNDS);
                    } else if (b > 32) {
                        atomicOr(a.err, ZERR_CORRUPT);
                    } else {
                        if (in_grp == 0 && blk) a.idx.grp_off[grp] = gpos;
                        a.idx.widths[gblk0 + blk] = (uint8_t)b;
                        if (blk + 1 == nb) {
                            const uint64_t end = gpos + zg_block_bytes_f(g.fmt, b, blk < nfull ? g.L : ntail);
                            if (end > a.avail) atomicOr(a.err, ZERR_BOUNDS);
                            w.seg_end[s] = end;
                            if (s + 1 < g.T && end != w.seg_R[s]) atomicOr(a.err, ZERR_CORRUPT);
                        }
                    }
                }
                for (in_grp += 32; in_grp >= g.GB; in_grp -= g.GB) grp++;
            }
            blk0 += n;
            if (run) pos += n;
            __syncwarp(); /* the list is reused */
        }
        __syncwarp();
    }
}

/* ---- W4: extra segment and total size -------------------------------- */
__global__ void k_walk_finish(const WalkArgs a)
{
    const ZGeom &g = a.g;
    const WalkScratch &w = a.ws;
    bool skip = false, cut = false;
    for (uint32_t s = threadIdx.x; s < g.T; s += blockDim.x) {
        skip |= !w.seg_ok[s];                     /* W0 already reported why */
        cut |= w.seg_ok[s] && w.seg_end[s] == 0;  /* the walk never reached this segment's last block */
    }
    const bool any_cut = __syncthreads_or(cut), any_skip = __syncthreads_or(skip);
    if (threadIdx.x != 0) return;
    if (any_cut) atomicOr(a.err, ZERR_CORRUPT);
    if (any_cut || any_skip) return;
    uint64_t pos = w.seg_end[g.T - 1];
    if (g.rem) {
        const uint64_t grp0 = (uint64_t)g.T * g.gr_reg, gblk0 = (uint64_t)g.T * g.nb_reg;
        if (pos + 4 > a.avail) {
            atomicOr(a.err, ZERR_BOUNDS);
            return;
        }
        a.idx.grp_off[grp0] = pos;
        pos += 4;
        for (uint64_t j = 0; j < g.nb_rm; j++) {
            if (j && j % g.GB == 0) a.idx.grp_off[grp0 + j / g.GB] = pos;
            if (pos >= a.avail) {
                atomicOr(a.err, ZERR_BOUNDS);
                return;
            }
            uint32_t b = a.in[pos];
            if (b > 32) {
                atomicOr(a.err, ZERR_CORRUPT);
                return;
            }
            a.idx.widths[gblk0 + j] = (uint8_t)b;
            pos += zg_block_bytes_f(g.fmt, b, zg_block_len(g.rem, g.L, j));
        }
        if (pos > a.avail) {
            atomicOr(a.err, ZERR_BOUNDS);
            return;
        }
    }
    *a.idx.size = pos;
}

} // namespace

/* Persistent grid: the CTAs that fit at once, at most `most`. */
static unsigned walk_grid(const void *fn, unsigned threads, size_t smem, unsigned most)
{
    const unsigned g = (unsigned)sm_count() * (unsigned)blocks_per_sm(fn, (int)threads, smem);
    return most < g ? (most ? most : 1) : g;
}

cudaError_t launch_walk(const WalkArgs &a0, cudaStream_t st)
{
    WalkArgs a = a0;
    a.M = zg_block_bytes(32, a.g.L);
    a.G = walk_group(a.M);
    a.w1_warp_bytes = w1_warp_bytes(a.M);
    cudaError_t e;
    k_walk_setup<<<1, 256, 0, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const uint32_t smem1 = WARPS_W1 * a.w1_warp_bytes;
    if ((e = set_max_smem((const void *)k_walk_tables, smem1)) != cudaSuccess) return e;
    const unsigned grid1 = walk_grid((const void *)k_walk_tables, 32 * WARPS_W1, smem1, (a.max_windows + WARPS_W1 - 1) / WARPS_W1);
    k_walk_tables<<<grid1, 32 * WARPS_W1, smem1, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const unsigned threads2 = std::max(512u, std::min(1024u, (a.M + 31u) / 32u * 32u)); /* a thread per entry offset, all to stage */
    const uint32_t smem2a = 4u * a.G * a.M;
    if ((e = set_max_smem((const void *)k_walk_groups, smem2a)) != cudaSuccess) return e;
    k_walk_groups<<<a.max_groups, threads2, smem2a, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    a.seg_batch = std::max(1u, (160u * 1024u) / (8u * a.M)); /* as many groups' tables at once as fit */
    const uint32_t smem2 = a.seg_batch * a.M * 8u;
    if ((e = set_max_smem((const void *)k_walk_segments, smem2)) != cudaSuccess) return e;
    k_walk_segments<<<a.g.T, 1024, smem2, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const uint32_t smem3 = WARPS_W3 * w3_warp_bytes(a.M);
    if ((e = set_max_smem((const void *)k_walk_final, smem3)) != cudaSuccess) return e;
    const unsigned grid3 = walk_grid((const void *)k_walk_final, 32 * WARPS_W3, smem3, (a.max_windows + WARPS_W3 - 1) / WARPS_W3);
    k_walk_final<<<grid3, 32 * WARPS_W3, smem3, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_walk_finish<<<1, 128, 0, st>>>(a);
    return cudaGetLastError();
}
