/*
 * zk_szp3d.cu -- the SZp 3-D Lorenzo codec, serial stream form.
 *
 * Replaces SZp_compress3D_fast / SZp_compress3D (ZCCL/src/ZCCL_float.c:1706-1860)
 * and SZp_decompress3D (ZCCL/src/ZCCLd_float.c:2801-2871) and produces the
 * same bytes and floats.  The reference walks the volume block by block and
 * carries its Lorenzo state from block to block; the quantity it encodes is
 * the 3-D mixed difference of the quantized values with zeros outside the
 * volume (ZCCL_float.h:63-73), which every element can form on its own, and
 * its inverse is the 3-D prefix sum.  So here every step is data parallel:
 *
 * quantization  q = (int)floor((double)x * (0.5 / eb) + 0.5) (ZCCL_float.h:57-61)
 *                with the reference's double rounding: float pairs where that
 *                is provably the same, FP64 for the rest;
 * compress   K1  the rate of every block (the bit length of its largest
 *                difference magnitude) into the rate table at the stream's
 *                start, and its payload size;
 *            K2  an exclusive scan of the payload sizes (three kernels);
 *            K3  every block packed at its offset: sign bits, then B =
 *                rate/8 high bytes per element, then the r = rate%8 low bits
 *                (the fastmode1 packers' layout,
 *                ZCCL/src/ZCCL_TypeManager.c:12-91,824-848);
 * decompress K1  payload sizes from the rate table, K2 the same scan,
 *            K3  every block's differences into the output buffer, viewed
 *                as int32;
 *            K4-K6 inclusive prefix sums along z (a warp per row), y and x
 *                (a thread per column, rows loaded in batches), the last one
 *                writing (float)((double)q * (2 eb)) in place
 *                (ZCCLd_float.c:2855-2857).
 *                For block sides 2, 4 and 8, K3 forms the z and y sums as it
 *                decodes, and the volume is passed over twice in all.
 * Block sides 2, 4 and 8: compress is one pass (K1-K3 together, quantizing as
 * it loads; the tiles' places in the stream come from one CTA's scan of their
 * sizes), decompress two.  Other block sides: a quantized volume, then a warp
 * (up to 512 elements) or a CTA per block.
 * Integer sums wrap modulo 2^32 like the reference's int.
 */
#include <algorithm>

#include "zkern.cuh"

namespace {

constexpr uint32_t SZ_THREADS = 256;
constexpr uint32_t SZ_CHUNK = 2048; /* sizes per CTA in the scan */
constexpr uint32_t SZ_SCAN_BATCH = 8; /* rows loaded together in the y and x prefix sums */

struct Sz3Dims {
    uint64_t d1, d2, d3;
    uint32_t bs;
    uint64_t nb1, nb2, nb3, nblocks;
};

__host__ __device__ inline Sz3Dims sz3_dims(uint64_t d1, uint64_t d2, uint64_t d3, uint32_t bs)
{
    Sz3Dims g;
    g.d1 = d1;
    g.d2 = d2;
    g.d3 = d3;
    g.bs = bs;
    g.nb1 = (d1 - 1) / bs + 1;
    g.nb2 = (d2 - 1) / bs + 1;
    g.nb3 = (d3 - 1) / bs + 1;
    g.nblocks = g.nb1 * g.nb2 * g.nb3;
    return g;
}

/* Block b's first element and extent on each axis. */
struct Sz3Block {
    uint64_t x0, y0, z0;
    uint32_t sx, sy, sz, n;
};

__device__ __forceinline__ Sz3Block sz3_block(const Sz3Dims &g, uint64_t b)
{
    Sz3Block k;
    const uint64_t bz = b % g.nb3, by = (b / g.nb3) % g.nb2, bx = b / (g.nb3 * g.nb2);
    k.x0 = bx * g.bs;
    k.y0 = by * g.bs;
    k.z0 = bz * g.bs;
    k.sx = (uint32_t)min((uint64_t)g.bs, g.d1 - k.x0);
    k.sy = (uint32_t)min((uint64_t)g.bs, g.d2 - k.y0);
    k.sz = (uint32_t)min((uint64_t)g.bs, g.d3 - k.z0);
    k.n = k.sx * k.sy * k.sz;
    return k;
}

/* Payload bytes of a block of n elements at rate b (0 for rate 0). */
__host__ __device__ inline uint32_t sz3_payload(uint32_t b, uint32_t n)
{
    if (!b) return 0;
    return (n + 7) / 8 + (b >> 3) * n + ((b & 7u) * n + 7) / 8;
}

/* A double as a pair of floats, hi = RN(d), lo = RN(d - hi), so that
 * hi + lo is within 2^-48 of d; ok only where both are normal floats
 * (2^-90 <= d <= 2^90), else the kernels take the double steps. */
struct Sz3Split {
    double d;
    float hi, lo;
    int ok;
    int mid; /* 2^-60 <= d <= 2^60: a product with an integer stays far from float's limits */
};

Sz3Split sz3_split(double d)
{
    Sz3Split s;
    s.d = d;
    s.hi = (float)d;
    s.lo = (float)(d - (double)s.hi);
    s.ok = d >= 0x1p-90 && d <= 0x1p90;
    s.mid = d >= 0x1p-60 && d <= 0x1p60;
    return s;
}

/* (int)floor((double)x * inv + 0.5), each step rounded as double
 * arithmetic rounds it (ZCCL_float.h:57-61).  FP64 is slow on this GPU, so
 * small products take one FMA (below); larger ones are first formed as a
 * float pair: hi = x*ih, its exact error
 * by FMA, plus x*il, within 2^-19 of x*inv + 0.5 when |x*ih| < 2^26.  When
 * the fractional part of that sum is more than 2^-12 from an integer, no
 * rounding of the exact product (at most 2^-27 here) can move it across
 * one, so its floor is the reference's; otherwise (about one element in
 * two thousand, or out of range, or not finite) the double steps run as
 * they are.  *bad is set where the reference is undefined. */
__device__ __forceinline__ int32_t sz3_quantize(float x, const Sz3Split &inv, uint32_t &bad)
{
    /* Below 2^11 one FMA suffices: x * ih + 0.5 rounded once is within
     * 2^-12.4 of x * inv + 0.5 (x * il and half an ulp), so a fraction more
     * than 2^-12 from an integer floors like the exact value. */
    const float t1 = __fmaf_rn(x, inv.hi, 0.5f);
    if (inv.ok && fabsf(t1) < 2048.0f) { /* NaN fails */
        const float n1 = floorf(t1), f1 = __fsub_rn(t1, n1);
        if (f1 > 2.44140625e-4f && f1 < 0.999755859375f) return (int32_t)n1;
    }
    const float th = __fmul_rn(x, inv.hi);
    if (inv.ok && fabsf(th) < 67108864.0f) { /* 2^26; NaN takes the double path */
        const float tl = __fmaf_rn(x, inv.lo, __fmaf_rn(x, inv.hi, -th));
        const float s = __fadd_rn(th, 0.5f); /* th + 0.5 = s + e exactly (TwoSum) */
        const float bb = __fsub_rn(s, th);
        const float e = __fadd_rn(__fsub_rn(th, __fsub_rn(s, bb)), __fsub_rn(0.5f, bb));
        const float n = floorf(s);
        float fr = __fadd_rn(__fsub_rn(s, n), __fadd_rn(e, tl));
        const float m = floorf(fr);
        fr = __fsub_rn(fr, m);
        if (fr > 2.44140625e-4f && fr < 0.999755859375f) return (int32_t)n + (int32_t)m;
    }
    const double v = floor(__dadd_rn(__dmul_rn((double)x, inv.d), 0.5));
    if (!(v >= -2147483648.0 && v < 2147483648.0)) { /* not finite, or outside int: undefined in the reference */
        bad = 1;
        return 0;
    }
    return (int32_t)v;
}

/* (float)((double)q * twice) (ZCCLd_float.c:2857), |q| < 2^24 (`sure` is false
 * beyond), with tw.mid.
 * EXACT: twice is a float (as where the caller's bound is one), so the double
 * product is exact and the float product rounds the same number once.  (Small
 * q often meet exact ties then, which no rounding test can settle.)
 * Else the product is formed as a float pair hi + lo, within 2^-46 of it;
 * r = hi + lo rounded, and d the exact rest (Fast2Sum).  r is the reference's
 * result unless the product lies so near the middle between r and a neighbour
 * that the double rounding could decide: if r + d (1 + 2^-17) still rounds to
 * r, the rest is below half an ulp by 2^-17 of it, far more than both
 * roundings and the pair's error (the test is exact at powers of two, where
 * the ulp changes). */
template <bool EXACT>
__device__ __forceinline__ float sz3_value(int32_t q, const Sz3Split &tw, bool &sure)
{
    const float qf = (float)q;
    const float hi = __fmul_rn(qf, tw.hi);
    sure = fabsf(qf) < 16777216.0f;
    if (EXACT) return hi;
    const float lo = __fmaf_rn(qf, tw.lo, __fmaf_rn(qf, tw.hi, -hi));
    const float r = __fadd_rn(hi, lo);
    const float d = __fsub_rn(lo, __fsub_rn(r, hi));
    sure = sure && __fmaf_rn(d, 1.00000762939453125f, r) == r; /* 1 + 2^-17 */
    return r;
}

/* N of them; the unsure ones (about one in 2^17) by the double steps, with
 * one branch for all. */
template <bool EXACT, uint32_t N>
__device__ __forceinline__ void sz3_values(const uint32_t (&q)[N], const Sz3Split &tw, float (&v)[N])
{
    bool all = true;
#pragma unroll
    for (uint32_t k = 0; k < N; k++) {
        bool sure;
        v[k] = sz3_value<EXACT>((int32_t)q[k], tw, sure);
        all &= sure;
    }
    if (!all) {
#pragma unroll
        for (uint32_t k = 0; k < N; k++) {
            bool sure;
            sz3_value<EXACT>((int32_t)q[k], tw, sure);
            if (!sure) v[k] = (float)__dmul_rn((double)(int32_t)q[k], tw.d);
        }
    }
}

template <uint32_t N>
__device__ __forceinline__ void sz3_values(const uint32_t (&q)[N], const Sz3Split &tw, float (&v)[N])
{
    if (tw.mid && tw.lo == 0.0f) { /* uniform over the grid */
        sz3_values<true>(q, tw, v);
    } else if (tw.mid) {
        sz3_values<false>(q, tw, v);
    } else {
#pragma unroll
        for (uint32_t k = 0; k < N; k++) v[k] = (float)__dmul_rn((double)(int32_t)q[k], tw.d);
    }
}

/* ---- K0: quantization -------------------------------------------------- */
__global__ void k_sz3_quant(const float *__restrict__ x, int32_t *__restrict__ q, uint64_t n, Sz3Split inv,
                            uint32_t *err)
{
    uint32_t bad = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        q[i] = sz3_quantize(x[i], inv, bad);
    if (bad) atomicOr(err, ZERR_RANGE);
}

/* The mixed difference at (i, j, k), zeros outside the volume. */
__device__ __forceinline__ uint32_t sz3_diff(const int32_t *q, const Sz3Dims &g, uint64_t i, uint64_t j, uint64_t k)
{
    const uint64_t s0 = g.d2 * g.d3, s1 = g.d3, p = i * s0 + j * s1 + k;
    auto at = [&](bool ok, uint64_t o) -> uint32_t { return ok ? (uint32_t)q[o] : 0u; };
    const bool bi = i > 0, bj = j > 0, bk = k > 0;
    return at(true, p) - at(bk, p - 1) - at(bj, p - s1) + at(bj && bk, p - s1 - 1) - at(bi, p - s0) +
           at(bi && bk, p - s0 - 1) + at(bi && bj, p - s0 - s1) - at(bi && bj && bk, p - s0 - s1 - 1);
}

/* Element t of a block (i slowest, k fastest), as in the reference. */
__device__ __forceinline__ void sz3_elem(const Sz3Block &k, uint32_t t, uint64_t &i, uint64_t &j, uint64_t &z)
{
    const uint32_t kz = t % k.sz, jy = (t / k.sz) % k.sy, ix = t / (k.sz * k.sy);
    i = k.x0 + ix;
    j = k.y0 + jy;
    z = k.z0 + kz;
}

__device__ __forceinline__ uint32_t mag(uint32_t v) { return (int32_t)v < 0 ? 0u - v : v; }

/* Blocks go to groups of G threads: a warp per block (G = 32) up to
 * 512 elements, the whole CTA (G = SZ_THREADS) above. */
template <uint32_t G>
__device__ __forceinline__ void group_sync()
{
    if (G == 32)
        __syncwarp();
    else
        __syncthreads();
}

/* ---- K1: rates and payload sizes (a group per block) -------------------- */
template <uint32_t G>
__global__ void __launch_bounds__(SZ_THREADS) k_sz3_rates(const int32_t *q, Sz3Dims g, uint8_t *out, uint32_t *sizes)
{
    __shared__ uint32_t wmax[SZ_THREADS / 32];
    const uint32_t per = SZ_THREADS / G, sub = threadIdx.x / G, gt = threadIdx.x % G;
    for (uint64_t b0 = (uint64_t)blockIdx.x * per; b0 < g.nblocks; b0 += (uint64_t)gridDim.x * per) {
        const uint64_t b = b0 + sub;
        const bool live = b < g.nblocks; /* uniform over the group */
        uint32_t m = 0;
        Sz3Block k = {};
        if (live) {
            k = sz3_block(g, b);
            for (uint32_t t = gt; t < k.n; t += G) {
                uint64_t i, j, z;
                sz3_elem(k, t, i, j, z);
                m = max(m, mag(sz3_diff(q, g, i, j, z)));
            }
        }
        m = __reduce_max_sync(0xffffffffu, m);
        if (G == 32) {
            if (live && gt == 0) {
                const uint32_t rate = 32u - __clz(m);
                out[b] = (uint8_t)rate;
                sizes[b] = sz3_payload(rate, k.n);
            }
        } else {
            if ((threadIdx.x & 31u) == 0) wmax[threadIdx.x >> 5] = m;
            __syncthreads();
            if (threadIdx.x == 0 && live) {
                for (uint32_t w = 0; w < blockDim.x / 32; w++) m = max(m, wmax[w]);
                const uint32_t rate = 32u - __clz(m);
                out[b] = (uint8_t)rate;
                sizes[b] = sz3_payload(rate, k.n);
            }
            __syncthreads();
        }
    }
}

/* ---- decompress K1: payload sizes from the rate table ------------------- */
__global__ void k_sz3_sizes(const uint8_t *in, uint64_t avail, Sz3Dims g, uint32_t *sizes, uint32_t *err)
{
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < g.nblocks; b += (uint64_t)gridDim.x * blockDim.x) {
        if (b >= avail) {
            atomicOr(err, ZERR_BOUNDS);
            sizes[b] = 0;
            continue;
        }
        const uint32_t rate = in[b];
        if (rate > 32) atomicOr(err, ZERR_CORRUPT);
        const Sz3Block k = sz3_block(g, b);
        sizes[b] = rate > 32 ? 0 : sz3_payload(rate, k.n);
    }
}

/* ---- K2: exclusive scan of the sizes into 64-bit offsets ---------------- */
__global__ void __launch_bounds__(1024) k_sz3_chunk_sums(const uint32_t *sizes, uint64_t nb, uint64_t *sums)
{
    __shared__ uint64_t ws[32];
    const uint64_t c = blockIdx.x, lo = c * SZ_CHUNK;
    uint64_t s = 0;
    for (uint64_t i = lo + threadIdx.x; i < nb && i < lo + SZ_CHUNK; i += blockDim.x) s += sizes[i];
    for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31u) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint64_t t = 0;
        for (uint32_t w = 0; w < blockDim.x / 32; w++) t += ws[w];
        sums[c] = t;
    }
}

/* One CTA: exclusive scan of the chunk sums in place; *total = all bytes. */
__global__ void __launch_bounds__(1024) k_sz3_scan_sums(uint64_t *sums, uint64_t nchunks, uint64_t head, uint64_t *total)
{
    __shared__ uint64_t ws[33];
    uint64_t carry = 0;
    for (uint64_t c0 = 0; c0 < nchunks; c0 += blockDim.x) {
        const uint64_t c = c0 + threadIdx.x;
        const uint64_t v = c < nchunks ? sums[c] : 0;
        uint64_t inc = v;
        const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= (uint32_t)o) inc += u;
        }
        if (lane == 31) ws[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            const uint64_t t = lane < blockDim.x / 32 ? ws[lane] : 0;
            uint64_t ti = t;
            for (int o = 1; o < 32; o <<= 1) {
                const uint64_t u = __shfl_up_sync(0xffffffffu, ti, o);
                if (lane >= (uint32_t)o) ti += u;
            }
            ws[lane] = ti - t;
            if (lane == 31) ws[32] = ti;
        }
        __syncthreads();
        if (c < nchunks) sums[c] = carry + ws[warp] + inc - v;
        carry += ws[32];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = head + carry;
}

/* sums: the chunks' exclusive sums; null for a single chunk, whose *total (all
 * bytes, with the rate table's `head`) is found here. */
__global__ void __launch_bounds__(1024) k_sz3_offsets(const uint32_t *sizes, uint64_t nb, const uint64_t *sums,
                                                      uint64_t *offs, uint64_t head, uint64_t *total)
{
    __shared__ uint64_t ws[33];
    const uint64_t c = blockIdx.x, lo = c * SZ_CHUNK;
    const uint32_t per = SZ_CHUNK / blockDim.x; /* consecutive sizes per thread */
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint64_t v[SZ_CHUNK / 1024 > 0 ? SZ_CHUNK / 1024 : 1];
    uint64_t s = 0;
    for (uint32_t r = 0; r < per; r++) {
        const uint64_t i = lo + (uint64_t)threadIdx.x * per + r;
        v[r] = i < nb ? sizes[i] : 0;
        s += v[r];
    }
    uint64_t inc = s;
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += u;
    }
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const uint64_t t = lane < blockDim.x / 32 ? ws[lane] : 0;
        uint64_t ti = t;
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t u = __shfl_up_sync(0xffffffffu, ti, o);
            if (lane >= (uint32_t)o) ti += u;
        }
        ws[lane] = ti - t;
    }
    __syncthreads();
    uint64_t run = (sums ? sums[c] : 0) + ws[warp] + inc - s;
    if (!sums && threadIdx.x == blockDim.x - 1) *total = head + run + s;
    for (uint32_t r = 0; r < per; r++) {
        const uint64_t i = lo + (uint64_t)threadIdx.x * per + r;
        if (i < nb) offs[i] = run;
        run += v[r];
    }
}

/* One block's n differences e[] (element order) packed at o with rate
 * `rate` > 0: sign bits (bit 7 - t % 8 of byte t / 8), B = rate/8 high
 * bytes per element (little-endian), then the r = rate%8 low bits, eight
 * elements to r bytes, MSB first; every byte by one of G threads (gt). */
template <uint32_t G>
__device__ __forceinline__ void sz3_pack_block(const uint32_t *e, uint32_t n, uint32_t rate, uint8_t *o, uint32_t gt)
{
    const uint32_t B = rate >> 3, r = rate & 7u, ns = (n + 7) / 8;
    for (uint32_t c = gt; c < ns; c += G) {
        uint32_t v = 0;
        for (uint32_t u = 0; u < 8 && 8 * c + u < n; u++) v |= ((e[8 * c + u] >> 31) & 1u) << (7 - u);
        o[c] = (uint8_t)v;
    }
    uint8_t *h = o + ns;
    if (B == 1) {
        for (uint32_t t = gt; t < n; t += G) h[t] = (uint8_t)(mag(e[t]) >> r);
    } else {
        for (uint32_t c = gt; c < B * n; c += G) {
            const uint32_t t = c / B, byte = c % B;
            h[c] = (uint8_t)((mag(e[t]) >> r) >> (8 * byte));
        }
    }
    if (r) {
        uint8_t *l = h + B * n;
        const uint32_t mask = (1u << r) - 1u, ng = (n + 7) / 8, tail = (r * n + 7) / 8;
        for (uint32_t gi = gt; gi < ng; gi += G) {
            uint64_t acc = 0;
            for (uint32_t u = 0; u < 8; u++) {
                const uint32_t t = 8 * gi + u;
                acc = (acc << r) | (t < n ? (mag(e[t]) & mask) : 0u);
            }
            for (uint32_t m = 0; m < r; m++) {
                const uint32_t at = gi * r + m;
                if (at < tail) l[at] = (uint8_t)(acc >> (8 * (r - 1 - m)));
            }
        }
    }
}

/* Element t of a block packed at `sg` with rate <= 32 (0: all zero). */
__device__ __forceinline__ uint32_t sz3_unpack_elem(const uint8_t *sg, uint32_t rate, uint32_t n, uint32_t t)
{
    if (!rate) return 0u;
    const uint32_t B = rate >> 3, r = rate & 7u, ns = (n + 7) / 8;
    const uint8_t *h = sg + ns, *l = h + B * n;
    uint32_t v = 0;
    for (uint32_t byte = 0; byte < B; byte++) v |= (uint32_t)h[t * B + byte] << (8 * byte);
    v <<= r;
    if (r) { /* bits [t r, t r + r) of the low section, MSB first */
        const uint64_t bit = (uint64_t)t * r;
        const uint64_t by = bit >> 3;
        const uint32_t w = ((uint32_t)l[by] << 8) | (by + 1 < (r * (uint64_t)n + 7) / 8 ? l[by + 1] : 0u);
        v |= (w >> (16 - (uint32_t)(bit & 7u) - r)) & ((1u << r) - 1u);
    }
    if ((sg[t >> 3] >> (7 - (t & 7u))) & 1u) v = 0u - v;
    return v;
}

/* ---- compress K3: pack every block at its offset (a group per block) ---- */
template <uint32_t G>
__global__ void __launch_bounds__(SZ_THREADS) k_sz3_pack(const int32_t *q, Sz3Dims g, uint8_t *out, uint64_t cap,
                                                         const uint64_t *offs, uint32_t *err)
{
    extern __shared__ uint32_t e_all[]; /* bs^3 differences per group */
    const uint32_t per = SZ_THREADS / G, sub = threadIdx.x / G, gt = threadIdx.x % G;
    uint32_t *e = e_all + sub * (g.bs * g.bs * g.bs);
    for (uint64_t b0 = (uint64_t)blockIdx.x * per; b0 < g.nblocks; b0 += (uint64_t)gridDim.x * per) {
        const uint64_t b = b0 + sub;
        /* every exit below is uniform over the group; a CTA-wide group meets
         * its barriers in every case */
        uint32_t rate = b < g.nblocks ? out[b] : 0u;
        const Sz3Block k = rate ? sz3_block(g, b) : Sz3Block{};
        const uint32_t n = k.n;
        const uint64_t base = rate ? g.nblocks + offs[b] : 0;
        if (rate && base + sz3_payload(rate, n) > cap) {
            if (gt == 0) atomicOr(err, ZERR_CAPACITY);
            rate = 0;
        }
        if (rate) {
            for (uint32_t t = gt; t < n; t += G) {
                uint64_t i, j, z;
                sz3_elem(k, t, i, j, z);
                e[t] = sz3_diff(q, g, i, j, z);
            }
        }
        group_sync<G>();
        if (rate) sz3_pack_block<G>(e, n, rate, out + base, gt);
        group_sync<G>();
    }
}

/* ---- decompress K3: every block's differences into the volume (a group per block) */
template <uint32_t G>
__global__ void __launch_bounds__(SZ_THREADS) k_sz3_unpack(const uint8_t *in, uint64_t avail, Sz3Dims g,
                                                           const uint64_t *offs, uint32_t *vol, uint32_t *err)
{
    const uint64_t s0 = g.d2 * g.d3, s1 = g.d3;
    const uint32_t per = SZ_THREADS / G, sub = threadIdx.x / G, gt = threadIdx.x % G;
    for (uint64_t b0 = (uint64_t)blockIdx.x * per; b0 < g.nblocks; b0 += (uint64_t)gridDim.x * per) {
        const uint64_t b = b0 + sub;
        if (b >= g.nblocks) continue; /* no barrier below */
        const Sz3Block k = sz3_block(g, b);
        uint32_t rate = b < avail ? in[b] : 0u;
        const uint64_t base = g.nblocks + offs[b];
        const uint32_t n = k.n;
        if (rate > 32 || base + sz3_payload(rate, n) > avail) { /* uniform over the CTA */
            if (gt == 0) atomicOr(err, rate > 32 ? ZERR_CORRUPT : ZERR_BOUNDS);
            rate = 0;
        }
        const uint8_t *sg = in + base;
        for (uint32_t t = gt; t < n; t += G) {
            const uint32_t v = sz3_unpack_elem(sg, rate, n, t);
            uint64_t i, j, z;
            sz3_elem(k, t, i, j, z);
            vol[i * s0 + j * s1 + z] = v;
        }
    }
}

/* ---- block sides 2, 4 and 8: compress ------------------------------------
 * A unit is U = 32 / BS consecutive blocks along z with the same block row
 * and plane: lane l owns z = z0 + l, in block l / BS.  A warp takes the unit's
 * rows plane by plane, quantizes them and forms the mixed difference from
 * neighbours it holds: the z neighbour by a shuffle (lane r takes row r's
 * element before z0), the previous row's z-difference and the previous plane's
 * 2-D differences in registers.  The row and plane before the
 * unit come in once more for that (zeros outside the volume). */
struct Sz3Unit {
    uint64_t bi, bj, bk0, i0, j0, z0;
    uint32_t sx, sy;
};

template <uint32_t BS>
__host__ __device__ inline uint64_t sz3_units(const Sz3Dims &g)
{
    return g.nb1 * g.nb2 * ((g.nb3 + 32 / BS - 1) / (32 / BS));
}

/* Extent along z of the unit's block c (0 past the volume). */
template <uint32_t BS>
__device__ __forceinline__ uint32_t sz3_unit_sz(const Sz3Dims &g, const Sz3Unit &k, uint32_t c)
{
    const uint64_t bk = k.bk0 + c;
    return bk < g.nb3 ? (uint32_t)min((uint64_t)BS, g.d3 - bk * BS) : 0u;
}

constexpr float SZ_MAGIC = 12582912.0f;         /* 1.5 * 2^23: a float m + this holds the integer m in its low bits, */
constexpr uint32_t SZ_ZERO = 0x4B400000u;       /* as this + m */

/* The unit's rows again, from memory: planes i0 - 1 .. and rows j0 - 1 .. of
 * each, z0 + lane, and in lane r the element before z0 of row r, zeros outside
 * the volume; plane(pl, v, l) for all BS + 1 planes, by the whole warp.  Sides 2
 * and 4 have all rows on their way at once, side 8 (81 rows) a plane ahead. */
template <uint32_t BS, class Plane>
__device__ __forceinline__ void sz3_reload(const float *__restrict__ x, const Sz3Dims &g, const Sz3Unit &k, Plane plane)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t s0 = g.d2 * g.d3, s1 = g.d3, z = k.z0 + lane;
    const bool zin = z < g.d3;
    auto load = [&](uint32_t pl, float (&v)[BS + 1], float &l) {
        const bool in = pl ? pl <= k.sx : k.i0 > 0 && k.sx > 0; /* (no unit: sx = 0) */
        const uint64_t o = (k.i0 + pl - 1) * s0; /* wraps only where not read */
#pragma unroll
        for (uint32_t r = 0; r <= BS; r++) v[r] = in && zin && (r ? r <= k.sy : k.j0 > 0) ? x[o + (k.j0 + r - 1) * s1 + z] : 0.0f;
        l = in && k.z0 && lane <= BS && (lane ? lane <= k.sy : k.j0 > 0) ? x[o + (k.j0 + lane - 1) * s1 + k.z0 - 1] : 0.0f;
    };
    if constexpr (BS == 8) {
        float v[BS + 1], nv[BS + 1], l, nl;
        load(0, v, l);
#pragma unroll 1
        for (uint32_t pl = 0; pl <= BS; pl++) {
            load(pl + 1, nv, nl); /* (zeros past the last) */
            plane(pl, v, l);
#pragma unroll
            for (uint32_t r = 0; r <= BS; r++) v[r] = nv[r];
            l = nl;
        }
    } else {
        float v[BS + 1][BS + 1], l[BS + 1];
#pragma unroll
        for (uint32_t pl = 0; pl <= BS; pl++) load(pl, v[pl], l[pl]);
#pragma unroll
        for (uint32_t pl = 0; pl <= BS; pl++) plane(pl, v[pl], l[pl]);
    }
}

/* sz3_quantize out of line. */
__device__ __noinline__ int32_t sz3_quantize_far(float x, const Sz3Split &inv, uint32_t &bad) { return sz3_quantize(x, inv, bad); }

/* The same: n is the integer next to the float x * hi and d the rest, x * (hi +
 * lo) - n, |d| < 2, which moves n on to the integer next to x * inv.  For |n| < 2^24
 * d's roundings (2^-25, 2^-24), lo's error (2^-24) and the reference's are together
 * below 2^-22.5; the others, and what lies within 2^-22 of a middle, go the long
 * way. */
__device__ __forceinline__ uint32_t sz3_quantize_wide(float x, const Sz3Split &inv, uint32_t &bad)
{
    const float p = __fmul_rn(x, inv.hi), n = rintf(p);
    const float d = __fmaf_rn(x, inv.lo, __fmaf_rn(x, inv.hi, -n)), c = __fsub_rn(__fadd_rn(d, SZ_MAGIC), SZ_MAGIC);
    if (inv.mid && fabsf(p) < 16777200.0f && fabsf(__fsub_rn(d, c)) < 0.499999761581420898f) /* NaN is not */
        return (uint32_t)__float2int_rn(__fadd_rn(n, c));
    return (uint32_t)sz3_quantize_far(x, inv, bad);
}

/* The unit's differences from integers, whatever their size: SZ_ZERO + difference
 * at w[di * BS + dj] (outside the volume: any), the largest magnitude to mx.
 * True, for the whole warp, if values or differences pass 2^22. */
template <uint32_t BS>
__device__ __forceinline__ bool sz3_walk_any(const float *x, const Sz3Dims &g, const Sz3Split &inv, const Sz3Unit &k, uint32_t *w,
                                          uint32_t &mx, uint32_t &bad)
{
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t dp[BS]; /* the plane's 2-D differences, row by row */
#pragma unroll
    for (uint32_t dj = 0; dj < BS; dj++) dp[dj] = 0;
    uint32_t far = 0;
    mx = 0;
    sz3_reload<BS>(x, g, k, [&](uint32_t pl, const float (&v)[BS + 1], float l) {
        const uint32_t ql = sz3_quantize_wide(l, inv, bad); /* 0 where l is */
        uint32_t rp = 0;
#pragma unroll
        for (uint32_t r = 0; r <= BS; r++) {
            const uint32_t q = sz3_quantize_wide(v[r], inv, bad);
            far = max(far, mag(q));
            const uint32_t up = __shfl_up_sync(0xffffffffu, q, 1), l0 = __shfl_sync(0xffffffffu, ql, r);
            const uint32_t rc = q - (lane ? up : l0); /* q(z) - q(z - 1) */
            if (r) {
                if (pl) {
                    const uint32_t e = rc - rp - dp[r - 1];
                    w[(pl - 1) * BS + r - 1] = SZ_ZERO + e;
                    mx = max(mx, mag(e));
                }
                dp[r - 1] = rc - rp;
            }
            rp = rc;
        }
    });
    return __any_sync(0xffffffffu, max(far, mx) >= 1u << 22) || !inv.mid;
}

/* (int)floor((double)x * inv + 0.5) on the float pipe.  n is the integer next
 * to x * hi, d = x * (hi + lo) - n: two roundings of 2^-25 at most, lo's own
 * error and the reference's two double roundings are together below 2^-23.5
 * for |n| < 2^22, so n is the reference's result if |d| < SZ_SURE, 1/2 - 2^-22.
 * If x * lo moves it past n's middle (one value in 2^25 / |n|), n + round(d)
 * is, unless a value lies next to a middle all the same (one in 2^21). */
constexpr float SZ_SURE = 0.499999761581420898f;
__device__ __forceinline__ float sz3_quantize_f(float x, const Sz3Split &inv, float &d)
{
    const float n = __fsub_rn(__fmaf_rn(x, inv.hi, SZ_MAGIC), SZ_MAGIC);
    d = __fmaf_rn(x, inv.lo, __fmaf_rn(x, inv.hi, -n));
    return n;
}

/* The same for any value: n moves on to the integer next to x * (hi + lo), and
 * what then still lies next to a middle takes the double steps.  Past 2^22, or
 * not finite: something past 2^22. */
__device__ __forceinline__ float sz3_quantize_any(float x, const Sz3Split &inv)
{
    float d;
    const float n = sz3_quantize_f(x, inv, d), c = __fsub_rn(__fadd_rn(d, SZ_MAGIC), SZ_MAGIC);
    if (!(fabsf(n) < 4194304.0f)) return 8388608.0f; /* NaN too */
    if (fabsf(__fsub_rn(d, c)) < SZ_SURE) return __fadd_rn(n, c);
    return (float)floor(__dadd_rn(__dmul_rn((double)x, inv.d), 0.5));
}
/* Four at a time, out of line. */
__device__ __noinline__ float4 sz3_quantize_any4(float4 x, const Sz3Split &inv)
{
    return make_float4(sz3_quantize_any(x.x, inv), sz3_quantize_any(x.y, inv), sz3_quantize_any(x.z, inv), sz3_quantize_any(x.w, inv));
}

/* One plane of a unit in floats, from its quantized rows q and, in lane r, the
 * element before row r's first: its differences to w (from the second plane on)
 * as SZ_ZERO + d, and the largest magnitudes of the values (far) and of the
 * differences (top). */
template <uint32_t BS>
__device__ __forceinline__ void sz3_plane_f(uint32_t pl, const float (&q)[BS + 1], float ql, float (&dp)[BS], uint32_t *w,
                                            float &far, float &top)
{
    const uint32_t lane = threadIdx.x & 31u;
    far = max3_abs(far, ql, q[0]);
#pragma unroll
    for (uint32_t r = 1; r < BS; r += 2) far = max3_abs(far, q[r], q[r + 1]);
    float rp = 0.0f, ep = 0.0f;
#pragma unroll
    for (uint32_t r = 0; r <= BS; r++) {
        const float up = __shfl_up_sync(0xffffffffu, q[r], 1), l0 = __shfl_sync(0xffffffffu, ql, r);
        const float rc = q[r] - (lane ? up : l0); /* q(z) - q(z - 1) */
        if (r) {
            const float d = rc - rp;
            if (pl) {
                const float e = d - dp[r - 1];
                w[(pl - 1) * BS + r - 1] = __float_as_uint(e + SZ_MAGIC);
                if (r % 2 == 0) top = max3_abs(top, ep, e);
                ep = e;
            }
            dp[r - 1] = d;
        }
        rp = rc;
    }
}

/* The unit once more from memory, every value by sz3_quantize_any; false (for
 * the whole warp) if values or differences pass 2^22. */
template <uint32_t BS>
__device__ __forceinline__ bool sz3_walk_again(const float *x, const Sz3Dims &g, const Sz3Split &inv, const Sz3Unit &k, uint32_t *w,
                                            uint32_t &mx)
{
    float dp[BS], far = 0.0f, top = 0.0f;
    sz3_reload<BS>(x, g, k, [&](uint32_t pl, const float (&v)[BS + 1], float l) {
        float q[BS + 1];
#pragma unroll
        for (uint32_t r = 0; r <= BS; r++) q[r] = sz3_quantize_any(v[r], inv);
        sz3_plane_f<BS>(pl, q, sz3_quantize_any(l, inv), dp, w, far, top);
    });
    mx = (uint32_t)top;
    return __all_sync(0xffffffffu, far < 4194304.0f && top < 4194304.0f);
}

/* A unit that sz3_walk_f leaves, with the most that it returned.  True if its
 * values or differences pass 2^22. */
template <uint32_t BS>
__device__ __noinline__ bool sz3_walk_slow(const float *x, const Sz3Dims &g, const Sz3Split &inv, const Sz3Unit &k, uint32_t left,
                                           uint32_t *w, uint32_t &mx, uint32_t &bad)
{
    if (BS < 8 && left == 1u && sz3_walk_again<BS>(x, g, inv, k, w, mx)) return false;
    return sz3_walk_any<BS>(x, g, inv, k, w, mx, bad);
}

/* A warp's rows on their way, plane by plane through its units, into PD
 * buffers in turn (a unit's BS + 1 planes are whole rounds of them): row r of a
 * plane is y = j0 - 1 + r, from the element before z0 on, in the 16-byte chunks
 * that hold it (160 bytes at any phase).  A lane copies NI chunks a plane;
 * rows outside the volume are zeros. */
constexpr uint32_t SZ_ROW = 160, SZ_CH = SZ_ROW / 16;
template <uint32_t BS>
struct Sz3Feed {
    static constexpr uint32_t N = SZ_CH * (BS + 1), NI = (N + 31) / 32, PLANE = SZ_ROW * (BS + 1), PD = BS == 4 ? 5 : 3;
    uint64_t at[NI]; /* this lane's chunks of the next plane: the element at their start, at any phase */
    int32_t lim[NI], top[NI]; /* a chunk is wanted where its row's phase is in [lim, top] */
    uint32_t planes; /* bit pl: plane pl is in the volume */
    __device__ __forceinline__ void set(const float *x, const Sz3Dims &g, const Sz3Unit &k)
    {
        const uint64_t a = reinterpret_cast<uintptr_t>(x) + 4u * ((k.i0 - 1) * (g.d2 * g.d3) + (k.j0 - 1) * g.d3 + k.z0 - 1);
        const int32_t nz = (int32_t)min((uint64_t)32, g.d3 - k.z0);
        planes = k.sx ? ((2u << k.sx) - 1u) & (k.i0 ? ~0u : ~1u) : 0u;
#pragma unroll
        for (uint32_t s = 0; s < NI; s++) {
            const uint32_t idx = (threadIdx.x & 31u) + 32u * s, r = idx / SZ_CH, ch = idx % SZ_CH;
            at[s] = a + 4u * g.d3 * r + 16u * ch; /* wraps only where not read */
            lim[s] = r >= (k.j0 ? 0u : 1u) && r <= k.sy ? (int32_t)(4u * ch) - nz : 4;
            top[s] = k.z0 == 0 && ch == 0 ? 2 : 3; /* nothing before the row's first element */
        }
    }
    /* the next plane, number pl of its unit; one group of copies, in any case */
    __device__ __forceinline__ void send(uint32_t buf, uint32_t pl, uint64_t stride)
    {
        const bool in = (planes >> pl) & 1u;
#pragma unroll
        for (uint32_t s = 0; s < NI; s++) {
            const uint32_t idx = (threadIdx.x & 31u) + 32u * s;
            if (32u * (s + 1) <= N || idx < N) {
                const int32_t ph = (int32_t)(((uint32_t)at[s] >> 2) & 3u);
                cp_async16_or_zero(buf + idx * 16u, reinterpret_cast<const void *>(at[s] & ~(uint64_t)15u),
                                   in && ph >= lim[s] && ph <= top[s]);
            }
            at[s] += stride;
        }
        cp_async_commit();
    }
};

/* The unit's differences, SZ_ZERO + d at w[di * BS + dj] (rows and planes
 * outside the volume: any), and this lane's largest magnitude; the next
 * unit's rows are sent for meanwhile, into the buffers that this one leaves.
 * In floats, which hold every step exactly while the quantized values and the
 * differences are below 2^22 (a difference of such values that passes 2^24, and
 * may be rounded, shows as one past 2^22).  Returns 0; or, by the lane, 2 if they
 * are not, and 1 where sz3_quantize_f leaves a value open: any w then.
 * Values of some 10^5 steps leave one open in nearly every unit: 256^3, side 4,
 * 150000 steps from zero, 282 us with integer steps for them, 131 with
 * sz3_walk_again (188 with integers for all).  A test after every plane keeps such units to their second form
 * for the plane alone (79 us), but parts the planes' code: 512^3, side 4, 413 and
 * 423 us, side 2 834 and 858.
 * Side 8 takes the planes in a loop, with w in local memory, and has that test: as
 * straight code for its 81 rows, a volume of 57 x 51 x 306 took 63 us, most of it
 * the code's way from L2, and 36 so; 512^3 489 us and 382. */
template <uint32_t BS>
__device__ __forceinline__ uint32_t sz3_walk_f(uint32_t sbuf, const float *__restrict__ x, const Sz3Dims &g, const Sz3Split &inv,
                                               const Sz3Unit &k, const Sz3Unit &next, Sz3Feed<BS> &feed, uint32_t (&w)[BS * BS],
                                               uint32_t &mx)
{
    using F = Sz3Feed<BS>;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t d3 = (uint32_t)g.d3, dpl = (uint32_t)(g.d2 * g.d3); /* phases: low bits are enough */
    const uint32_t a0 = ((uint32_t)reinterpret_cast<uintptr_t>(x) >> 2) + ((uint32_t)k.i0 - 1u) * dpl + ((uint32_t)k.j0 - 1u) * d3 +
                        (uint32_t)k.z0 - 1u;
    const bool lin = k.z0 && lane <= BS;
    const uint64_t stride = 4u * g.d2 * g.d3;
    float dp[BS], far = 0.0f, top = 0.0f, open = 0.0f; /* open: the widest rest */
    uint32_t slot = 0; /* pl % PD */
#pragma unroll(BS == 8 ? 1 : BS + 1)
    for (uint32_t pl = 0; pl <= BS; pl++, slot = slot + 1 == F::PD ? 0 : slot + 1) {
        cp_async_wait<F::PD - 1>(); /* all but the PD - 1 planes after this one */
        __syncwarp();
        const uint32_t buf = sbuf + slot * F::PLANE, ap = a0 + pl * dpl;
        float cv[BS + 1], cl;
#pragma unroll
        for (uint32_t r = 0; r <= BS; r++) cv[r] = ld_shared_f32(buf + r * SZ_ROW + 4u * (((ap + r * d3) & 3u) + 1u + lane));
        cl = lin ? ld_shared_f32(buf + lane * SZ_ROW + 4u * ((ap + lane * d3) & 3u)) : 0.0f; /* lane r: before row r */
        __syncwarp();
        if (pl + F::PD == BS + 1) feed.set(x, g, next);
        feed.send(buf, pl + F::PD <= BS ? pl + F::PD : pl + F::PD - BS - 1, stride);
        float q[BS + 1], d[BS + 1], dl, ql = sz3_quantize_f(cl, inv, dl);
#pragma unroll
        for (uint32_t r = 0; r <= BS; r++) q[r] = sz3_quantize_f(cv[r], inv, d[r]);
        open = max3_abs_nan(open, dl, d[0]);
#pragma unroll
        for (uint32_t r = 1; r < BS; r += 2) open = max3_abs_nan(open, d[r], d[r + 1]);
        if (BS == 8 && __any_sync(0xffffffffu, !(open < SZ_SURE))) { /* the plane again */
            open = 0.0f;
            auto at = [&](uint32_t r) { return r == 0 ? cl : cv[r <= BS + 1 ? r - 1 : 0]; };
#pragma unroll
            for (uint32_t r = 0; r < BS + 2; r += 4) {
                const float4 a = sz3_quantize_any4(make_float4(at(r), at(r + 1), at(r + 2), at(r + 3)), inv);
                if (r == 0) ql = a.x;
                else q[r - 1] = a.x;
                if (r < BS + 1) q[r < BS + 1 ? r : 0] = a.y;
                if (r + 1 < BS + 1) q[r + 1 < BS + 1 ? r + 1 : 0] = a.z;
                if (r + 2 < BS + 1) q[r + 2 < BS + 1 ? r + 2 : 0] = a.w;
            }
        }
        sz3_plane_f<BS>(pl, q, ql, dp, w, far, top);
    }
    mx = (uint32_t)top;
    return !(far < 4194304.0f && top < 4194304.0f) ? 2u : BS < 8 && !(open < SZ_SURE) ? 1u : 0u;
}

/* In sz3_walk_f's place, for a warp whose last unit it could not take: the feed
 * moves on.  (Side 8, 256^3, 6 million steps from zero, 252 us without and 216;
 * sides 2 and 4 lose 4 % of every volume by it.) */
template <uint32_t BS>
__device__ __forceinline__ void sz3_pass(uint32_t sbuf, const float *__restrict__ x, const Sz3Dims &g, const Sz3Unit &next,
                                         Sz3Feed<BS> &feed)
{
    using F = Sz3Feed<BS>;
#pragma unroll 1
    for (uint32_t pl = 0; pl <= BS; pl++) {
        cp_async_wait<F::PD - 1>();
        __syncwarp();
        if (pl + F::PD == BS + 1) feed.set(x, g, next);
        feed.send(sbuf + pl % F::PD * F::PLANE, pl + F::PD <= BS ? pl + F::PD : pl + F::PD - BS - 1, 4u * g.d2 * g.d3);
    }
}

/* Octet g of a block of n elements at byte o of the zeroed buffer: w[k] =
 * SZ_ZERO + difference (0 past the block's end). */
__device__ __forceinline__ void sz3_put_octet(uint32_t sbase, uint32_t o, uint32_t rate, uint32_t n, uint32_t g,
                                              const uint32_t (&w)[8])
{
    if (!rate) return;
    const uint32_t B = rate >> 3, r = rate & 7u, h = o + ((n + 7u) >> 3), at = o + g;
    uint32_t m[8], s8 = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const uint32_t v = w[k] - SZ_ZERO;
        s8 = __funnelshift_l(v, s8, 1);
        m[k] = (uint32_t)abs((int32_t)v);
    }
    if (s8) sh_or(sbase + (at & ~3u), s8 << (8u * (at & 3u)));
    put_octet(sbase, h, n, g, B, r, m);
}

/* One pass.  Tiles of NW * UPW units in stream order, handed out by tickets:
 * each of NW compute warps takes UPW units, keeps their differences in
 * registers while the blocks' rates, sizes and places in the tile are found
 * (the tile's one barrier), and packs them into a ring in shared memory, an
 * octet of 8 consecutive elements a lane: 256 elements at a time change from
 * rows to octets through a small buffer.  The ring, its placer warps (which
 * write the tiles out) and the scan of the tiles' sizes by one CTA are the
 * 1-D compressor's.
 * Bound by issue, 85 instructions per 32 elements at side 4 (252 with exact
 * integer quantization, byte-wise packing and a look-back per warp).  512^3:
 * side 8 388 us, 4 410, 2 820, against 706, 1216 and 3662.  At side 4, from
 * 407, two units a warp took 440, three CTAs an SM 470 (spills), 10 or 12
 * compute warps the same 408. */
template <uint32_t BS, uint32_t NW> /* NW: compute warps */
struct Sz3Cm {
    static constexpr uint32_t U = 32 / BS, NB = BS * BS * BS, UPW = BS == 2 ? 2 : 1;
    static constexpr uint32_t BPW = U * UPW;                                 /* blocks per warp, at most 32 */
    static constexpr uint32_t ROWS = BS * BS < 8 ? BS * BS : 8;              /* rows of a unit changed at a time */
    static constexpr uint32_t PER = ROWS * BS, BST = PER + (BS == 2 ? 4 : BS); /* a block's elements in them, its stride */
    static constexpr uint32_t WORST = NW * BPW * ((NB + 7) / 8 + 4 * NB);    /* a tile's bytes */
    static constexpr uint32_t THREADS = 32 * (NW + 2);                       /* and the placer and the one that claims */
    static constexpr uint32_t FEED = Sz3Feed<BS>::PLANE * Sz3Feed<BS>::PD;   /* a warp's rows */
    static constexpr uint32_t OWN = FEED + 4 * U * BST;                      /* a warp's shared bytes */
};
constexpr uint32_t SZ_CM_PLACERS = 1;

struct Sz3CmShared {
    uint64_t full[2], empty[2];
    uint64_t ticket[2];
    uint4 place[2][16]; /* compute warps' first units: z chunk, block row, block plane */
    uint32_t ws[2][34];
    ZRing ring;
    uint32_t scanner;
};
constexpr uint32_t SZ_CM_HEAD = (sizeof(Sz3CmShared) + 15u) / 16u * 16u;

template <uint32_t BS, uint32_t NW>
__global__ void __launch_bounds__(Sz3Cm<BS, NW>::THREADS, 2) k_sz3_compress_rows(const float *__restrict__ x, Sz3Dims g, Sz3Split inv,
                                                                        uint8_t *out, uint64_t cap, uint64_t *status,
                                                                        uint32_t *ticket, uint64_t *total_out, uint32_t R,
                                                                        uint32_t *err)
{
    using C = Sz3Cm<BS, NW>;
    constexpr uint32_t U = C::U, UPW = C::UPW;
    extern __shared__ __align__(16) uint8_t sm[];
    Sz3CmShared *sh = reinterpret_cast<Sz3CmShared *>(sm);
    uint8_t *outs = sm + SZ_CM_HEAD + NW * C::OWN;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t nzc = (uint32_t)((g.nb3 + U - 1) / U), nb2 = (uint32_t)g.nb2;
    const uint32_t units = (uint32_t)sz3_units<BS>(g), ntiles = (units + NW * UPW - 1u) / (NW * UPW);
    uint32_t bad = 0;
    if (tid == 0) {
        for (uint32_t i = 0; i < 2; i++) {
            mbar_init(&sh->full[i], 1);
            mbar_init(&sh->empty[i], NW);
        }
        ring_init(&sh->ring, NW);
        sh->scanner = gridDim.x > 1 && atomicAdd(ticket + 1, 1u) == 0;
    }
#pragma unroll 1
    for (uint32_t i = tid; i < (R + 48u) / 16u; i += C::THREADS) reinterpret_cast<uint4 *>(outs)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    if (sh->scanner) {
        if (warp == 0) scan_tiles(status, ntiles, ticket, err, SCAN_SPIN_LIMIT);
        return;
    }
    if (warp >= NW && warp < NW + SZ_CM_PLACERS) {
        placer_loop<SZ_CM_PLACERS>(&sh->ring, outs, status, ntiles, warp - NW, err, bad, SCAN_SPIN_LIMIT);
        if (bad) atomicOr(err, bad);
        return;
    }
    if (warp == NW + SZ_CM_PLACERS) { /* claims the tiles */
        for (uint32_t it = 0;; it++) {
            uint32_t t = lane ? 0u : atomicAdd(ticket, 1u);
            t = __shfl_sync(0xffffffffu, t, 0);
            const uint32_t s = it & 1u, u = t * (NW * UPW) + lane * UPW, strip = u / nzc;
            if (it >= 2) mbar_wait(&sh->empty[s], (it / 2u - 1u) & 1u, err);
            if (lane < NW)
                sh->place[s][lane] = make_uint4(u - strip * nzc, strip % nb2, t < ntiles ? strip / nb2 : (uint32_t)g.nb1, 0u);
            __syncwarp();
            if (lane == 0) {
                if (t < ntiles) {
                    ZSlot &S = ring_slot(&sh->ring, it, err);
                    S.ticket = t;
                    S.out = out;
                    S.cap = cap;
                    S.hdr = nullptr;
                    S.size = t == ntiles - 1u ? total_out : nullptr;
                    S.T8 = g.nblocks; /* the rate table */
                    S.ngrp = 0;
                }
                sh->ticket[s] = t < ntiles ? t : ZP_NONE;
                mbar_arrive(&sh->full[s]);
            }
            if (t >= ntiles) return;
        }
    }

    uint8_t *own = sm + SZ_CM_HEAD + warp * C::OWN;
    uint32_t *st = reinterpret_cast<uint32_t *>(own + C::FEED);
    const uint32_t sbuf = smem_u32(own);
    const uint32_t c = lane / BS, dz = lane % BS; /* this lane's block and place in a unit */
    uint32_t H = 0, hp = 0;
    /* tile number it's ticket (once for each it) and this warp's first unit of it */
    uint4 at;
    auto claim = [&](uint32_t it) {
        mbar_wait(&sh->full[it & 1u], (it / 2u) & 1u, err);
        const uint64_t t = sh->ticket[it & 1u];
        at = sh->place[it & 1u][warp];
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->empty[it & 1u]);
        return t;
    };
    auto unit = [&]() { /* the unit at `at` (no rows or planes where there is none), which moves on */
        Sz3Unit K;
        K.bk0 = (uint64_t)at.x * U;
        K.bj = at.y;
        K.bi = at.z;
        K.i0 = K.bi * BS;
        K.j0 = K.bj * BS;
        K.z0 = K.bk0 * BS;
        K.sx = at.z < (uint32_t)g.nb1 ? (uint32_t)min((uint64_t)BS, g.d1 - K.i0) : 0u;
        K.sy = K.sx ? (uint32_t)min((uint64_t)BS, g.d2 - K.j0) : 0u;
        if (++at.x == nzc) {
            at.x = 0;
            if (++at.y == nb2) {
                at.y = 0;
                at.z++;
            }
        }
        return K;
    };
    uint64_t t = claim(0);
    bool far = !inv.mid; /* side 8: sz3_walk_f would not take the next unit, as it seems (uniform over the warp) */
    Sz3Unit nextu = unit();
    Sz3Feed<BS> feed;
    feed.set(x, g, nextu);
#pragma unroll 1
    for (uint32_t pl = 0; pl < Sz3Feed<BS>::PD; pl++) feed.send(sbuf + pl * Sz3Feed<BS>::PLANE, pl, 4u * g.d2 * g.d3);
#pragma unroll 1
    for (uint32_t it = 0; it <= ntiles; it++) {
        if (t == ZP_NONE) {
            if (tid == 0) ring_end(&sh->ring, it, SZ_CM_PLACERS, err);
            break;
        }
        uint64_t tn = ZP_NONE;
        uint32_t w[UPW][BS * BS];
        Sz3Unit k[UPW];
        uint32_t rate = 0, n = 0; /* lane b: block b of the warp's */
#pragma unroll
        for (uint32_t i = 0; i < UPW; i++) {
            Sz3Unit &K = k[i];
            K = nextu;
            if (i + 1 == UPW) tn = claim(it + 1);
            nextu = unit();
            uint32_t mx = 0;
            uint32_t left = 2;
            if (BS == 8 && far)
                sz3_pass<BS>(sbuf, x, g, nextu, feed);
            else
                left = sz3_walk_f<BS>(sbuf, x, g, inv, K, nextu, feed, w[i], mx);
            if (BS < 8 && !inv.mid) left = 2;
            if (__any_sync(0xffffffffu, left != 0u)) {
                left = __reduce_max_sync(0xffffffffu, left);
                if constexpr (BS == 8) {
                    far = sz3_walk_slow<BS>(x, g, inv, K, left, w[i], mx, bad);
                } else {
                    uint32_t d[BS * BS];
                    sz3_walk_slow<BS>(x, g, inv, K, left, d, mx, bad);
#pragma unroll
                    for (uint32_t e = 0; e < BS * BS; e++) w[i][e] = d[e];
                }
            }
            if (K.sx < BS || K.sy < BS) { /* rows outside the volume count for nothing */
                mx = 0;
#pragma unroll(BS == 8 ? 1 : BS)
                for (uint32_t di = 0; di < BS; di++)
                    if (di < K.sx)
#pragma unroll
                        for (uint32_t dj = 0; dj < BS; dj++)
                            if (dj < K.sy) mx = max(mx, mag(w[i][di * BS + dj] - SZ_ZERO));
            }
            if (K.z0 + lane >= g.d3) mx = 0;
#pragma unroll
            for (uint32_t o = 1; o < BS; o <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const uint32_t mc = __shfl_sync(0xffffffffu, mx, (lane % U) * BS);
            if (lane / U == i && K.sx) {
                n = K.sx * K.sy * sz3_unit_sz<BS>(g, K, lane % U);
                rate = n ? 32u - __clz(mc) : 0u;
                if (n) out[(K.bi * g.nb2 + K.bj) * g.nb3 + K.bk0 + lane % U] = (uint8_t)rate;
            }
        }
        uint32_t total;
        const uint32_t off = grp_excl_scan1(sz3_payload(rate, n), sh->ws[it & 1u], &total, 32u * NW, 1);
        if (tid == 0) {
            scan_publish(status, t, total, t == 0);
            ring_sized(&sh->ring, it, total);
        }
        uint32_t mend;
        const uint32_t pos = ring_space(&sh->ring, zg_ring_need(total), R, H, hp, mend, err);
        const uint32_t pk = smem_u32(outs + pos);
#pragma unroll
        for (uint32_t i = 0; i < UPW; i++) {
            const Sz3Unit &K = k[i];
            if constexpr (BS == 8) {
                /* blocks whole along z go plane by plane, an octet a row; the last one of a unit, from `whole` on,
                 * where it is not, in its own order, 256 elements at a time */
                const uint32_t zleft = (uint32_t)min((uint64_t)32, g.d3 - K.z0);
                const uint32_t there = K.sx ? (zleft + 7u) / 8u : 0u, whole = K.sx ? zleft / 8u : 0u;
#pragma unroll 1
                for (uint32_t di = 0; whole && di < K.sx; di++) {
                    __syncwarp();
#pragma unroll
                    for (uint32_t e = 0; e < 8; e++) st[c * C::BST + e * 8u + dz] = w[i][di * 8u + e];
                    __syncwarp();
                    const uint32_t b = lane / 8u, at = __shfl_sync(0xffffffffu, off, b), rb = __shfl_sync(0xffffffffu, rate, b);
                    if (b < whole && lane % 8u < K.sy) {
                        const uint4 *p = reinterpret_cast<const uint4 *>(st + b * C::BST + 8u * (lane % 8u));
                        const uint4 lo = p[0], hi = p[1];
                        const uint32_t v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                        sz3_put_octet(pk, at, rb, K.sx * K.sy * 8u, di * K.sy + lane % 8u, v);
                    }
                }
                const uint32_t sz = K.z0 + lane < g.d3 ? sz3_unit_sz<BS>(g, K, c) : 0u;
#pragma unroll 1
                for (uint32_t lot = 2u * whole; lot < 2u * there; lot++) {
                    const uint32_t b = lot / 2u, e0 = (lot & 1u) * 256u; /* its block, and first element of it */
                    if (e0 >= K.sx * K.sy * 8u) continue;
                    __syncwarp();
                    if (sz && c == b)
#pragma unroll 1
                        for (uint32_t di = 0; di < K.sx; di++) {
                            const uint32_t at = di * K.sy * sz + dz - e0; /* its row 0 */
                            if ((int32_t)at >= 256 || (int32_t)(at + K.sy * sz) <= 0) continue;
#pragma unroll
                            for (uint32_t dj = 0; dj < 8; dj++)
                                if (dj < K.sy && at + dj * sz < 256u) st[at + dj * sz] = w[i][di * 8u + dj];
                        }
                    __syncwarp();
                    const uint32_t at = __shfl_sync(0xffffffffu, off, b), rb = __shfl_sync(0xffffffffu, rate, b), nb = __shfl_sync(0xffffffffu, n, b);
                    if (e0 + 8u * lane < nb) {
                        uint32_t v[8];
#pragma unroll
                        for (uint32_t e = 0; e < 8; e++) v[e] = e0 + 8u * lane + e < nb ? st[8u * lane + e] : SZ_ZERO;
                        sz3_put_octet(pk, at, rb, nb, e0 / 8u + lane, v);
                    }
                }
            } else if (K.sx == BS && K.sy == BS && K.z0 + 32 <= g.d3) { /* whole blocks: rows are octets, or halves or quarters */
#pragma unroll
                for (uint32_t e0 = 0; e0 < BS * BS; e0 += C::ROWS) {
                    __syncwarp();
#pragma unroll
                    for (uint32_t e = 0; e < C::ROWS; e++) st[c * C::BST + e * BS + dz] = w[i][e0 + e];
                    __syncwarp();
                    constexpr uint32_t OCT = C::PER / 8; /* octets of a block in this lot */
                    const uint32_t b = lane / OCT, go = lane % OCT;
                    const uint32_t at = __shfl_sync(0xffffffffu, off, (i * U + b) & 31u), rb = __shfl_sync(0xffffffffu, rate, (i * U + b) & 31u);
                    if (b < U) {
                        const uint4 *p = reinterpret_cast<const uint4 *>(st + b * C::BST + 8u * go);
                        const uint4 lo = p[0], hi = p[1];
                        const uint32_t v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                        sz3_put_octet(pk, at, rb, C::NB, e0 * BS / 8u + go, v);
                    }
                }
            } else if (K.sx) { /* at the volume's end: 256 elements at a time in their blocks' own order */
                constexpr uint32_t NB = C::NB, LB = NB > 256 ? 256 : NB, LOTS = U * NB > 256 ? U * NB / 256 : 1; /* a lot's elements of a block */
                const uint32_t sz = K.z0 + lane < g.d3 ? sz3_unit_sz<BS>(g, K, c) : 0u;
#pragma unroll 1
                for (uint32_t lot = 0; lot < LOTS; lot++) {
                    const uint32_t b0 = lot * 256u / NB, e0 = lot * 256u % NB; /* its first block, and first element of it */
                    __syncwarp();
                    if (sz && c - b0 < 256u / LB)
#pragma unroll
                        for (uint32_t e = 0; e < BS * BS; e++) {
                            const uint32_t di = e / BS, dj = e % BS, at = (di * K.sy + dj) * sz + dz - e0;
                            if (di < K.sx && dj < K.sy && at < LB) st[(c - b0) * LB + at] = w[i][e];
                        }
                    __syncwarp();
                    const uint32_t b = b0 + lane / (LB / 8u), go = lane % (LB / 8u), ln = (i * U + b) & 31u;
                    const uint32_t at = __shfl_sync(0xffffffffu, off, ln), rb = __shfl_sync(0xffffffffu, rate, ln), nb = __shfl_sync(0xffffffffu, n, ln);
                    if (b < U && e0 + 8u * go < nb) {
                        uint32_t v[8];
#pragma unroll
                        for (uint32_t e = 0; e < 8; e++) v[e] = e0 + 8u * go + e < nb ? st[(b - b0) * LB + 8u * go + e] : SZ_ZERO;
                        sz3_put_octet(pk, at, rb, nb, e0 / 8u + go, v);
                    }
                }
            }
        }
        if (tid == 0) ring_where(&sh->ring, it, pos, mend);
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->ring.packed[it % ZR_SLOTS]);
        t = tn;
    }
    cp_async_wait<0>();
    if (bad) atomicOr(err, ZERR_RANGE);
}

/* ---- block sides 2, 4 and 8: decompress ---------------------------------
 * The inverse of the mixed difference is a prefix sum along each axis, in any
 * order, so the decoder sums along y and z what it decodes and one pass along
 * x finishes: the volume is written as integers, read and written as floats
 * (12 bytes of traffic an element instead of the 28 of a pass per axis).
 * 301 x 450 x 517, side 8: 858 us before (decode 347, z 93, y 120, x 406
 * alone), 258 now (decode and sums 118, x 103, the carries 15).
 * 512^3: side 8 408 us, 4 425, 2 590.
 *
 * A strip is a row of blocks along z; its bytes are consecutive in the stream.
 * A part is PARTS strips along y.  Consumer warps take one layer of a part's
 * blocks each (BS = 8: one plane, 4: one plane, 2: both), a chunk of up to 32
 * blocks of a strip at a time, a lane per block: a lane decodes octets (8
 * consecutive elements of its block: one row of 8, two of 4, or the four of 2
 * with both planes), adds them to its columns' running y sums (registers), and
 * a warp scan makes the z sums, whose carry along the row sits in shared
 * memory.  Rows leave through shared memory, coalesced.
 * A producer warp copies the chunks' bytes into a ring of slots.  Blocks of 512 elements take whole
 * multiples of 64 bytes, so side by side the lanes' reads would meet in one
 * bank 16 times over (512^3: 239 us, 94 % of the cycles on shared memory);
 * they are placed one bank apart, by 4-byte asynchronous copies.  Where a
 * chunk does not fit a slot (side 8, rates above about 10) it goes in pieces
 * of 16 or 8 blocks; pieces of up to 16 blocks have 2, 4 or 8 rows decoded
 * side by side, summed along y by shuffles.
 * The parts' y sums start at zero; each part's last row is kept (`carry`), and
 * the pass along x adds the sums of the parts before it. */
template <uint32_t BS>
struct Sz3Un {
    static constexpr uint32_t PI = BS == 2 ? 2 : 1, PJ = BS == 8 ? 1 : 2; /* planes and rows of an octet */
    static constexpr uint32_t PW = BS / PI, STRIPS = 8 / PW;              /* warps per strip, strips per CTA (along x) */
    static constexpr uint32_t PARTS = BS == 8 ? 1 : 16 / BS;              /* strips per part: 8 or 16 rows */
    static constexpr uint32_t ROWS = PARTS * BS, NB = BS * BS * BS;
    static constexpr uint32_t CAP = BS == 8 ? 24u * 1024u : 32u * ((NB + 7) / 8 + 4 * NB); /* bytes of a chunk in a slot */
    static constexpr uint32_t AREA = (CAP + 32u + NB / 8 + NB + 24u + 15u) & ~15u; /* phase, rounding, what decode_octet reads on */
    static constexpr uint32_t SLOTS = BS == 8 ? 2 : 3;
    static constexpr uint32_t SLOT = 16u + STRIPS * (128u + AREA);        /* blocks in it | block descriptors | bytes */
    static constexpr uint32_t OUT = 4u * 288u;                            /* a warp's rows on their way out */
    static constexpr uint32_t SMEM = SLOTS * SLOT + 8u * (OUT + 4u * PI * ROWS) + 4096u; /* margin: reads stay inside whatever a slot holds */
};
constexpr uint32_t SZ_UN_THREADS = 9 * 32;

/* Chunks of 32 blocks of the strips, in stream order: their payload bytes (a
 * warp per chunk). */
__global__ void __launch_bounds__(SZ_THREADS) k_sz3_chunk_sizes(const uint8_t *__restrict__ in, uint64_t avail, Sz3Dims g,
                                                                uint64_t nchunks, uint32_t *__restrict__ sizes, uint32_t *err)
{
    constexpr uint32_t C = 4; /* chunks at a time */
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t nzc = (g.nb3 + 31) / 32;
    uint32_t flag = 0;
    for (uint64_t c0 = C * (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); c0 < nchunks;
         c0 += C * (((uint64_t)gridDim.x * blockDim.x) >> 5)) {
        uint32_t rate[C], n[C];
        uint64_t strip = c0 / nzc, zc = c0 % nzc;
#pragma unroll
        for (uint32_t u = 0; u < C; u++) {
            const uint64_t bk = zc * 32 + lane, b = strip * g.nb3 + bk;
            const bool in_vol = c0 + u < nchunks && bk < g.nb3;
            const uint64_t bj = strip % g.nb2, bi = strip / g.nb2;
            rate[u] = in_vol && b < avail ? in[b] : 0u;
            if (in_vol && b >= avail) flag |= ZERR_BOUNDS;
            n[u] = in_vol ? (uint32_t)(min((uint64_t)g.bs, g.d1 - bi * g.bs) * min((uint64_t)g.bs, g.d2 - bj * g.bs) *
                                       min((uint64_t)g.bs, g.d3 - bk * g.bs))
                          : 0u;
            if (++zc == nzc) {
                zc = 0;
                strip++;
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < C; u++) {
            if (rate[u] > 32) {
                flag |= ZERR_CORRUPT;
                rate[u] = 0;
            }
            const uint32_t size = __reduce_add_sync(0xffffffffu, sz3_payload(rate[u], n[u]));
            if (lane == 0 && c0 + u < nchunks) sizes[c0 + u] = size;
        }
    }
    if (flag) atomicOr(err, flag);
}

/* How a volume's chunks go to CTAs: a task is a part of STRIPS strips and one
 * of nseg pieces of it along z. */
struct Sz3Tasks {
    uint64_t ntasks, nparts, nbg, nseg;
    uint64_t seg; /* blocks along z in a piece: a multiple of 32 */
};

/* Where a CTA is in its chunks: one of every strip of it at a time.  PIECES:
 * the strips are cut along z. */
template <uint32_t BS, bool PIECES>
struct Sz3Pos {
    Sz3Tasks t;
    uint64_t task;
    uint64_t cb, cb1, bj, bj1, bi0;
    __device__ __forceinline__ uint64_t strips() const { return PIECES ? task / t.nseg : task; } /* the task's, in all */
    __device__ __forceinline__ uint64_t first() const { return strips() % t.nparts * Sz3Un<BS>::PARTS; }
    __device__ __forceinline__ void begin(const Sz3Dims &g)
    {
        if (task >= t.ntasks) return;
        bi0 = (t.nbg - 1 - strips() / t.nparts) * Sz3Un<BS>::STRIPS;
        bj = first();
        bj1 = min(bj + Sz3Un<BS>::PARTS, g.nb2);
        cb = PIECES ? task % t.nseg * t.seg : 0;
        cb1 = PIECES ? min(cb + t.seg, g.nb3) : g.nb3;
    }
    __device__ __forceinline__ void advance(const Sz3Dims &g)
    {
        if (++bj < bj1) return;
        cb += 32;
        if (cb < (PIECES ? cb1 : g.nb3)) {
            bj = first();
            return;
        }
        task += gridDim.x;
        begin(g);
    }
};

/* Producer, sides 2 and 4: lane s sends strip s's chunk and lane STRIPS + s
 * its rates, from which the strip's consumers place its blocks; the next
 * chunk's place is on its way meanwhile. */
template <uint32_t BS, bool PIECES>
__device__ __forceinline__ void sz3_produce_small(const uint8_t *__restrict__ in, uint64_t avail, const Sz3Dims &g,
                                                  const uint64_t *__restrict__ offs, const uint32_t *__restrict__ sizes,
                                                  uint8_t *slots, uint64_t *full, uint64_t *empty, Sz3Pos<BS, PIECES> p, uint32_t *err)
{
    using U = Sz3Un<BS>;
    const uint32_t lane = threadIdx.x & 31u, s = lane % U::STRIPS;
    const uint64_t nzc = (g.nb3 + 31) / 32;
    if (lane >= 2 * U::STRIPS) return;
    auto fetch = [&](uint64_t &at, uint32_t &bytes) {
        const uint64_t bi = p.bi0 + s, strip = bi * g.nb2 + p.bj;
        at = avail;
        bytes = 0;
        if (p.task >= p.t.ntasks || bi >= g.nb1) return;
        if (lane < U::STRIPS) {
            at = g.nblocks + offs[strip * nzc + p.cb / 32];
            bytes = sizes[strip * nzc + p.cb / 32];
        } else {
            at = strip * g.nb3 + p.cb;
            bytes = (uint32_t)min((uint64_t)32, g.nb3 - p.cb);
        }
    };
    uint64_t nat;
    uint32_t nbytes, it = 0;
    fetch(nat, nbytes);
    for (; p.task < p.t.ntasks; it++) {
        const uint64_t at = nat;
        const uint32_t bytes = at >= avail ? 0u : (uint32_t)min((uint64_t)nbytes, avail - at);
        p.advance(g);
        fetch(nat, nbytes);
        const uint32_t slot = it % U::SLOTS;
        uint8_t *sl = slots + slot * U::SLOT, *head = sl + 16u + 128u * s;
        if (it >= U::SLOTS) mbar_wait(empty + slot, (it / U::SLOTS - 1u) & 1u, err);
        reinterpret_cast<uint64_t *>(head)[lane / U::STRIPS] = at;
        tma_load_superset(lane < U::STRIPS ? sl + 16u + 128u * U::STRIPS + s * U::AREA : head + 16u, in + at, bytes, full + slot);
    }
}

/* Producer, side 8 (one strip): block c at word c (mod 32) of the slot, in as
 * many pieces as it takes. */
template <bool PIECES>
__device__ __forceinline__ void sz3_produce8(const uint8_t *__restrict__ in, uint64_t avail, const Sz3Dims &g,
                                             const uint64_t *__restrict__ offs, uint8_t *slots, uint64_t *full,
                                             uint64_t *empty, Sz3Pos<8, PIECES> p, uint32_t *err)
{
    using U = Sz3Un<8>;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t nzc = (g.nb3 + 31) / 32;
    uint32_t flag = 0, it = 0, nrate = 0;
    uint64_t nbase = 0;
    auto fetch = [&]() { /* the next chunk's rates and place */
        if (p.task >= p.t.ntasks) return;
        const uint64_t strip = p.bi0 * g.nb2 + p.bj, at = strip * g.nb3 + p.cb + lane;
        nrate = p.cb + lane < g.nb3 && at < avail ? in[at] : 0u;
        nbase = g.nblocks + offs[strip * nzc + p.cb / 32];
    };
    fetch();
    while (p.task < p.t.ntasks) {
        const uint32_t kb = (uint32_t)min((uint64_t)32, g.nb3 - p.cb);
        const uint32_t sx = (uint32_t)min((uint64_t)8, g.d1 - p.bi0 * 8), sy = (uint32_t)min((uint64_t)8, g.d2 - p.bj * 8);
        const uint32_t sz = lane < kb ? (uint32_t)min((uint64_t)8, g.d3 - (p.cb + lane) * 8) : 0u;
        uint32_t rate = nrate > 32u ? 0u : nrate; /* reported with the sizes */
        const uint32_t pay = sz3_payload(rate, sx * sy * sz), inc = warp_incl_scan(pay);
        const uint64_t at = nbase + (inc - pay);
        if (rate && at + pay > avail) {
            flag |= ZERR_BOUNDS;
            rate = 0;
        }
        p.advance(g);
        fetch();
        const uint32_t phase = (uint32_t)(reinterpret_cast<uintptr_t>(in) + at) & 3u;
        const uint32_t words = rate ? (phase + pay + 3u) / 4u : 0u, room = ((words + 31u) & ~31u) + 1u;
        const uint32_t rinc = warp_incl_scan(room);
        const uint32_t half = __shfl_sync(0xffffffffu, rinc, 15), all = __shfl_sync(0xffffffffu, rinc, 31);
        uint32_t kk = 32;
        if (4u * all > U::CAP) kk = 4u * half <= U::CAP && 4u * (all - half) <= U::CAP ? 16 : 8;
        const uint8_t *mine = in + (at - phase); /* this lane's block */
        for (uint32_t sb = 0; sb < kb; sb += kk, it++) {
            const uint32_t slot = it % U::SLOTS;
            uint8_t *sl = slots + slot * U::SLOT;
            if (it >= U::SLOTS) mbar_wait(empty + slot, (it / U::SLOTS - 1u) & 1u, err);
            const uint32_t lo = __shfl_sync(0xffffffffu, rinc - room, sb), pos = rinc - room - lo;
            if (lane >= sb && lane < sb + kk)
                reinterpret_cast<uint32_t *>(sl + 16)[lane - sb] = (4u * pos + phase) | rate << 24;
            if (lane == 0) *reinterpret_cast<uint32_t *>(sl) = min(kk, kb - sb);
            const uint32_t area = smem_u32(sl + 16u + 128u) + 4u * lane;
            const uint32_t last = min(sb + kk, kb);
#pragma unroll 2
            for (uint32_t c = sb; c < last; c++) {
                const uint32_t nw = __shfl_sync(0xffffffffu, words, c), d = area + 4u * __shfl_sync(0xffffffffu, pos, c);
                const uint8_t *src =
                    reinterpret_cast<const uint8_t *>(__shfl_sync(0xffffffffu, reinterpret_cast<uintptr_t>(mine), c)) + 4u * lane;
                for (uint32_t t = 0; t < nw; t += 128) {
#pragma unroll
                    for (uint32_t q = 0; q < 128; q += 32)
                        if (lane + t + q < nw) cp_async4(d + 4u * (t + q), src + 4u * (t + q));
                }
            }
            cp_async_arrive(full + slot); /* every lane, when its copies have landed */
            __syncwarp();
            if (lane == 0) mbar_arrive(full + slot); /* and the descriptors */
        }
    }
    if (flag) atomicOr(err, flag);
}

/* What a warp decodes at a time: k blocks of one strip, from block c0 on, in
 * the planes from i0 on. */
struct Sz3Piece {
    const uint8_t *area;
    uint32_t dsc; /* lane c: block c's place in the area and its rate << 24 (0: no block) */
    uint32_t *outw, *zc; /* the warp's row buffer; its rows' z sums */
    uint32_t *o;         /* the volume at (i0, the strip's first row, the first block's z + lane) */
    uint32_t *co;        /* the same place in the part's kept rows; null if none of these rows is kept */
    uint64_t s0, s1;     /* strides of the volume along x and y */
    uint64_t cs;         /* stride of the kept rows along x */
    uint32_t k, sx, sy, di0, row0, zlim, zleft;
    bool first;          /* the rows begin here */
};

/* LK: 2^LK lanes a row (side 8 may take fewer than 32, and 32 >> LK rows side
 * by side).  WHOLE: the blocks are whole along y and z. */
template <uint32_t BS, uint32_t LK, bool WHOLE>
__device__ __forceinline__ void sz3_strip(const Sz3Piece &w, uint32_t (&y)[Sz3Un<BS>::PI * BS])
{
    using U = Sz3Un<BS>;
    constexpr uint32_t PJ = U::PJ, NR = 8 / BS, kk = 1u << LK, RJ = 32u >> LK;
    const uint32_t lane = threadIdx.x & 31u, c = lane & (kk - 1u), rj = lane >> LK;
    const uint32_t sy = WHOLE ? BS : w.sy, NJ = (sy + PJ - 1) / PJ;
    const uint32_t dsc = LK == 5 ? w.dsc : __shfl_sync(0xffffffffu, w.dsc, c);
    const uint32_t rate = min(dsc >> 24, 32u), off = min(dsc & 0xFFFFFFu, U::CAP + 16u);
    const uint32_t sz = WHOLE ? BS : c < w.k ? min(BS, w.zleft - c * BS) : 0u, n = w.sx * sy * sz;
    const bool octets = WHOLE || (sz == BS && sy % PJ == 0); /* every octet is 8 consecutive elements */
    const uint32_t g0 = BS == 2 ? 0u : (w.di0 * sy) / PJ;
    uint32_t *o = w.o;
    uint32_t *src = w.outw + (BS == 8 ? (lane >> 3) * 4u + (lane & 3u) + ((lane >> 2) & 1u) * 144u : lane);
    constexpr uint32_t STEP = BS == 8 ? 16 : 32; /* words of src per 32 elements */
#pragma unroll(LK == 5 && BS < 8 ? 4 : 1)
    for (uint32_t j = 0; j < NJ; j += RJ, o += RJ * PJ * w.s1) {
        const uint32_t jj = j + rj;
        uint32_t v[8];
        if (WHOLE) {
            decode_octet<true>(reinterpret_cast<const uint32_t *>(w.area), off - 1u, rate, n, g0 + jj, ZG_FASTMODE1, v);
        } else {
#pragma unroll
            for (uint32_t e = 0; e < 8; e++) v[e] = 0;
            if (jj < NJ && sz) {
                if (octets) {
                    decode_octet<true>(reinterpret_cast<const uint32_t *>(w.area), off - 1u, rate, n, g0 + jj, ZG_FASTMODE1, v);
                } else { /* at the volume's end: an element at a time */
#pragma unroll
                    for (uint32_t e = 0; e < 8; e++) {
                        const uint32_t r = e / BS, di = w.di0 + r / PJ, dj = jj * PJ + r % PJ, dz = e % BS;
                        if (di < w.sx && dj < sy && dz < sz)
                            v[e] = sz3_unpack_elem(w.area + off, rate, n, (di * sy + dj) * sz + dz);
                    }
                }
            }
        }
        /* y sums */
        if (BS == 8) {
#pragma unroll
            for (uint32_t t = kk; t < 32; t <<= 1)
#pragma unroll
                for (uint32_t e = 0; e < 8; e++) {
                    const uint32_t u = __shfl_up_sync(0xffffffffu, v[e], t);
                    if (lane >= t) v[e] += u;
                }
#pragma unroll
            for (uint32_t e = 0; e < 8; e++) v[e] += y[e % (U::PI * BS)];
#pragma unroll
            for (uint32_t e = 0; e < 8; e++)
                y[e % (U::PI * BS)] = RJ == 1 ? v[e] : __shfl_sync(0xffffffffu, v[e], 32u - kk + c);
        } else {
#pragma unroll
            for (uint32_t r = 0; r < NR; r++)
#pragma unroll
                for (uint32_t e = 0; e < BS; e++) y[(r / PJ) * BS + e] = v[r * BS + e] += y[(r / PJ) * BS + e];
        }
        /* z sums */
#pragma unroll
        for (uint32_t r = 0; r < NR; r++) {
            uint32_t tot = v[r * BS];
#pragma unroll
            for (uint32_t e = 1; e < BS; e++) tot += v[r * BS + e];
            uint32_t run = tot;
#pragma unroll
            for (uint32_t t = 1; t < kk; t <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, run, t);
                if (c >= t) run += u;
            }
            uint32_t *z = w.zc + (r / PJ) * U::ROWS + w.row0 + jj * PJ + r % PJ;
            const uint32_t before = w.first ? 0u : *z;
            __syncwarp();
            if (c == kk - 1u) *z = before + run;
            v[r * BS] += before + run - tot;
#pragma unroll
            for (uint32_t e = 1; e < BS; e++) v[r * BS + e] += v[r * BS + e - 1];
        }
        /* out, whole rows: word e of the warp's 256 in row order is element e (side 8: the halves of a
         * block's row 144 words apart, so that neither side meets bank conflicts).  The barriers above
         * part this from the last row's reads. */
        if (BS == 8) {
            *reinterpret_cast<uint4 *>(w.outw + 4u * lane) = make_uint4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<uint4 *>(w.outw + 144u + 4u * lane) = make_uint4(v[4], v[5], v[6], v[7]);
        } else if (BS == 4) {
            *reinterpret_cast<uint4 *>(w.outw + 4u * lane) = make_uint4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<uint4 *>(w.outw + 128u + 4u * lane) = make_uint4(v[4], v[5], v[6], v[7]);
        } else {
#pragma unroll
            for (uint32_t r = 0; r < NR; r++)
                *reinterpret_cast<uint2 *>(w.outw + 64u * r + 2u * lane) = make_uint2(v[2 * r], v[2 * r + 1]);
        }
        __syncwarp();
        if (LK == 5) {
#pragma unroll
            for (uint32_t r = 0; r < NR; r++)
                if ((U::PI == 1 || w.di0 + r / PJ < w.sx) && (WHOLE || j * PJ + r % PJ < sy)) { /* uniform */
                    uint32_t *p = o + (r / PJ) * w.s0 + (r % PJ) * w.s1;
                    if (WHOLE && w.zlim == 32u * BS) {
#pragma unroll
                        for (uint32_t q = 0; q < BS; q++) p[32u * q] = src[(r * BS + q) * STEP];
                    } else {
#pragma unroll
                        for (uint32_t q = 0; q < BS; q++)
                            if (lane + 32u * q < w.zlim) p[32u * q] = src[(r * BS + q) * STEP];
                    }
                    if (w.co && j * PJ + r % PJ + 1u == sy) { /* the part's last row */
                        uint32_t *cp = w.co + (r / PJ) * w.cs;
#pragma unroll
                        for (uint32_t q = 0; q < BS; q++)
                            if (lane + 32u * q < w.zlim) cp[32u * q] = src[(r * BS + q) * STEP];
                    }
                }
        } else { /* side 8, RJ rows of kk blocks */
#pragma unroll
            for (uint32_t q = 0; q < 8; q++) {
                const uint32_t r = q / (kk / 4u), z = 32u * (q % (kk / 4u));
                if ((WHOLE || j + r < sy) && lane + z < w.zlim) {
                    const uint32_t x = src[q * STEP];
                    o[r * w.s1 + z] = x;
                    if (w.co && j + r + 1u == sy) w.co[z] = x;
                }
            }
        }
    }
    __syncwarp();
}

template <uint32_t BS, bool PIECES>
__global__ void __launch_bounds__(SZ_UN_THREADS, 3) k_sz3_unpack_sum(const uint8_t *__restrict__ in, uint64_t avail, Sz3Dims g, Sz3Tasks tk,
                                                                     const uint64_t *__restrict__ offs,
                                                                     const uint32_t *__restrict__ sizes,
                                                                     uint32_t *__restrict__ vol, uint32_t *__restrict__ carry,
                                                                     uint32_t *err)
{
    using U = Sz3Un<BS>;
    constexpr uint32_t PI = U::PI;
    extern __shared__ __align__(16) uint8_t sm[];
    __shared__ uint64_t full[U::SLOTS], empty[U::SLOTS];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0)
        for (uint32_t i = 0; i < U::SLOTS; i++) {
            mbar_init(full + i, BS == 8 ? 33 : 2 * U::STRIPS);
            mbar_init(empty + i, 8);
        }
    __syncthreads();
    if (warp == 8) {
        Sz3Pos<BS, PIECES> p;
        p.t = tk;
        p.task = blockIdx.x;
        p.begin(g);
        if constexpr (BS == 8)
            sz3_produce8<PIECES>(in, avail, g, offs, sm, full, empty, p, err);
        else
            sz3_produce_small<BS, PIECES>(in, avail, g, offs, sizes, sm, full, empty, p, err);
        return;
    }
    const uint32_t s = warp / U::PW;
    Sz3Piece w;
    w.outw = reinterpret_cast<uint32_t *>(sm + U::SLOTS * U::SLOT + warp * (U::OUT + 4u * PI * U::ROWS));
    w.zc = w.outw + U::OUT / 4u; /* [PI][ROWS] */
    w.di0 = (warp % U::PW) * PI;
    w.s0 = g.d2 * g.d3;
    w.s1 = g.d3;
    w.cs = g.d3;
    uint32_t it = 0, flag = 0;
    for (uint64_t task = blockIdx.x; task < tk.ntasks; task += gridDim.x) {
        const uint64_t strips = PIECES ? task / tk.nseg : task, z0 = PIECES ? task % tk.nseg * tk.seg : 0;
        const uint64_t part = strips % tk.nparts, bi = (tk.nbg - 1 - strips / tk.nparts) * U::STRIPS + s;
        const uint64_t bj0 = part * U::PARTS, bj1 = min(bj0 + U::PARTS, g.nb2), i0 = bi * BS + w.di0;
        const uint64_t z1 = PIECES ? min(z0 + tk.seg, g.nb3) : g.nb3;
        w.sx = bi < g.nb1 ? (uint32_t)min((uint64_t)BS, g.d1 - bi * BS) : 0u;
        for (uint64_t c0 = z0; c0 < z1; c0 += w.k) {
            uint32_t y[PI * BS]; /* the columns' y sums */
#pragma unroll
            for (uint32_t e = 0; e < PI * BS; e++) y[e] = 0;
            w.first = c0 == z0;
            for (uint64_t bj = bj0; bj < bj1; bj++, it++) {
                const uint32_t slot = it % U::SLOTS;
                const uint8_t *sl = sm + slot * U::SLOT;
                mbar_wait(full + slot, (it / U::SLOTS) & 1u, err);
                const uint8_t *head = sl + 16u + 128u * s;
                if (BS == 8)
                    w.k = min(max(*reinterpret_cast<const uint32_t *>(sl), 1u), 32u);
                else
                    w.k = (uint32_t)min((uint64_t)32, g.nb3 - c0);
                if (w.di0 < w.sx) {
                    w.area = sl + 16u + 128u * U::STRIPS + s * U::AREA;
                    w.sy = (uint32_t)min((uint64_t)BS, g.d2 - bj * BS);
                    if (BS == 8) {
                        w.dsc = lane < w.k ? reinterpret_cast<const uint32_t *>(head)[lane] : 0u;
                    } else { /* the blocks' places, from their rates */
                        const uint64_t at = reinterpret_cast<const uint64_t *>(head)[0], rat = reinterpret_cast<const uint64_t *>(head)[1];
                        uint32_t rate = lane < w.k && rat + lane < avail
                                            ? head[16u + ((uint32_t)(reinterpret_cast<uintptr_t>(in) + rat) & 15u) + lane]
                                            : 0u;
                        if (rate > 32u) rate = 0; /* reported with the sizes */
                        const uint32_t zl = (uint32_t)min(g.d3 - c0 * BS, (uint64_t)(32u * BS));
                        const uint32_t pay = sz3_payload(rate, w.sx * w.sy * min(BS, zl - min(zl, lane * BS)));
                        const uint32_t inc = warp_incl_scan(pay);
                        if (rate && at + inc > avail) {
                            flag |= ZERR_BOUNDS;
                            rate = 0;
                        }
                        w.dsc = (inc - pay + ((uint32_t)(reinterpret_cast<uintptr_t>(in) + at) & 15u)) | rate << 24;
                    }
                    w.row0 = (uint32_t)(bj - bj0) * BS;
                    w.zleft = (uint32_t)min(g.d3 - c0 * BS, (uint64_t)(32u * BS));
                    w.zlim = min(w.zleft, w.k * BS);
                    w.o = vol + i0 * w.s0 + bj * BS * w.s1 + c0 * BS + lane;
                    w.co = part + 1 < tk.nparts && bj + 1 == bj1 ? carry + (part * g.d1 + i0) * g.d3 + c0 * BS + lane : nullptr;
                    const bool whole = w.sy == BS && w.zlim == w.k * BS;
                    if (BS < 8 || w.k > 16) {
                        if (whole) sz3_strip<BS, 5, true>(w, y);
                        else sz3_strip<BS, 5, false>(w, y);
                    } else if constexpr (BS == 8) {
                        if (w.k > 8) {
                            if (whole) sz3_strip<8, 4, true>(w, y);
                            else sz3_strip<8, 4, false>(w, y);
                        } else if (w.k > 4) {
                            if (whole) sz3_strip<8, 3, true>(w, y);
                            else sz3_strip<8, 3, false>(w, y);
                        } else {
                            if (whole) sz3_strip<8, 2, true>(w, y);
                            else sz3_strip<8, 2, false>(w, y);
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(empty + slot);
            }
        }
    }
    if (flag) atomicOr(err, flag);
}

/* The parts' last rows summed over the parts, in place: a thread per (plane,
 * z), batches of rows loaded together. */
__global__ void __launch_bounds__(256) k_sz3_carry(uint32_t *__restrict__ carry, uint64_t columns, uint64_t parts)
{
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= columns) return;
    uint32_t run = 0;
    for (uint64_t p0 = 0; p0 < parts; p0 += SZ_SCAN_BATCH) {
        uint32_t v[SZ_SCAN_BATCH];
#pragma unroll
        for (uint32_t u = 0; u < SZ_SCAN_BATCH; u++) v[u] = p0 + u < parts ? carry[(p0 + u) * columns + t] : 0u;
#pragma unroll
        for (uint32_t u = 0; u < SZ_SCAN_BATCH; u++) {
            run += v[u];
            if (p0 + u < parts) carry[(p0 + u) * columns + t] = run;
        }
    }
}

/* Rows whose z sums start anew in each of nseg pieces of `seg` elements: what is
 * still to be added to each (pre[row * nseg + s]), the sums at the ends of the
 * pieces before it, of the row and of the carry's row that belongs to it; a
 * warp per row of the volume. */
__global__ void __launch_bounds__(256) k_sz3_piece_sums(const uint32_t *__restrict__ vol, const uint32_t *__restrict__ carry,
                                                        uint64_t d1, uint64_t d2, uint64_t d3, uint32_t part_rows, uint64_t seg,
                                                        uint64_t nseg, uint32_t *__restrict__ pre)
{
    const uint64_t row = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (row >= d1 * d2) return;
    const uint64_t i = row / d2, part = row % d2 / part_rows;
    const uint32_t *v = vol + row * d3, *c = part ? carry + ((part - 1) * d1 + i) * d3 : nullptr;
    uint32_t run = 0;
    for (uint64_t s0 = 0; s0 < nseg; s0 += 32) {
        const uint64_t s = s0 + (threadIdx.x & 31u), z = (s + 1) * seg - 1;
        const uint32_t e = s + 1 < nseg ? v[z] + (c ? c[z] : 0u) : 0u, inc = warp_incl_scan(e);
        if (s < nseg) pre[row * nseg + s] = run + inc - e;
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
}

/* The last pass: x sums of the volume and the parts' carries, floats in place.
 * A CTA takes a run of up to FQ * 288 consecutive elements of a plane (R whole
 * rows of one part, or a piece of a long row) and walks along x, FQ columns'
 * sums a thread.  A producer warp keeps a ring of stages of FP planes on their
 * way (the run, and the carry's row that its rows share).  Bound by memory:
 * 512^3 176 us (6.1 TB/s), against 351 with the threads themselves loading 4
 * planes ahead into registers.  Small planes leave an SM few warps, and a
 * stage's chain of waits, sums and stores sets the pace: eight planes a stage
 * and one column a thread then. */
constexpr uint32_t FTH = 288; /* summing threads at most */

struct Sz3Run {
    uint32_t R;      /* rows in a run */
    uint32_t pieces; /* runs per row where rows are longer than a run */
    uint32_t cols;   /* elements of a full run */
    uint32_t cz;     /* carry elements of a full run */
    uint32_t pb, cb; /* bytes of their places in a stage */
    uint32_t stages;
    const uint32_t *pre; /* PIECES: what the rows' pieces along z lack (k_sz3_piece_sums) */
    uint64_t seg, nseg;
};

template <uint32_t FQ, uint32_t FP, bool PIECES>
__global__ void __launch_bounds__(FTH + 32) k_sz3_finish(uint32_t *vol, const uint32_t *carry, uint64_t d1,
                                                                uint64_t d2, uint64_t d3, uint32_t rows, Sz3Run f,
                                                                Sz3Split twice, uint32_t *err)
{
    extern __shared__ __align__(16) uint8_t ring[]; /* per stage: FP runs, FP carries */
    __shared__ uint64_t full[8], empty[8];
    const uint32_t nth = blockDim.x - 32u, stage = FP * (f.pb + f.cb);
    const uint64_t j0 = blockIdx.x / f.pieces * f.R, z0 = (uint64_t)(blockIdx.x % f.pieces) * f.cols, plane = d2 * d3;
    const uint64_t part = j0 / rows; /* parts are whole multiples of R rows */
    const uint32_t cols = f.pieces > 1 ? (uint32_t)min((uint64_t)f.cols, d3 - z0) : (uint32_t)(min((uint64_t)f.R, d2 - j0) * d3);
    const bool more = part > 0;
    const uint64_t nst = (d1 + FP - 1) / FP;
    uint32_t *p0 = vol + j0 * d3 + z0;
    const uint32_t *c0 = more ? carry + (part - 1) * d1 * d3 + z0 : nullptr;
    if (threadIdx.x == 0)
        for (uint32_t i = 0; i < f.stages; i++) {
            mbar_init(full + i, 2 * FP);
            mbar_init(empty + i, nth / 32u);
        }
    __syncthreads();
    if (threadIdx.x >= nth) {
        const uint32_t l = threadIdx.x - nth, pl = l % FP, c = l / FP;
        if (c >= 2) return;
        uint32_t slot = 0, round = 0;
        for (uint64_t st = 0; st < nst; st++) {
            const uint64_t i = FP * st + pl;
            if (round) mbar_wait(empty + slot, (round - 1u) & 1u, err);
            const uint32_t *g = c ? c0 + i * d3 : p0 + i * plane;
            const uint32_t bytes = i < d1 && (!c || more) ? 4u * (c ? min(cols, f.cz) : cols) : 0u;
            tma_load_superset(ring + slot * stage + pl * f.pb + c * (FP * f.pb - pl * f.pb + pl * f.cb),
                              reinterpret_cast<const uint8_t *>(g), bytes, full + slot);
            if (++slot == f.stages) {
                slot = 0;
                round++;
            }
        }
        return;
    }
    uint32_t run[FQ], at[FQ], cz[FQ]; /* the columns' sums; their places in the run and in the carry's row */
#pragma unroll
    for (uint32_t q = 0; q < FQ; q++) { /* past the run's end: a column again, so that no value is out of the way */
        run[q] = 0;
        at[q] = min(threadIdx.x + nth * q, cols - 1u);
        cz[q] = at[q] % f.cz;
    }
    /* where a copy's first element lies in its 16 bytes: the low bits of its address */
    const uint32_t pv = (uint32_t)(reinterpret_cast<uintptr_t>(p0) >> 2), pc = (uint32_t)(reinterpret_cast<uintptr_t>(c0) >> 2);
    float *o = reinterpret_cast<float *>(p0) + threadIdx.x;
    const uint32_t *zp[FQ]; /* PIECES: the columns' places in f.pre, in the next plane */
    if (PIECES) {
#pragma unroll
        for (uint32_t q = 0; q < FQ; q++) zp[q] = f.pre + (j0 + at[q] / f.cz) * f.nseg + (z0 + cz[q]) / f.seg;
    }
    uint32_t slot = 0, round = 0;
    for (uint64_t st = 0; st < nst; st++, o += FP * plane) {
        uint32_t zv[FP * FQ];
        if (PIECES) {
#pragma unroll
            for (uint32_t pl = 0; pl < FP; pl++)
#pragma unroll
                for (uint32_t q = 0; q < FQ; q++) {
                    zv[pl * FQ + q] = FP * st + pl < d1 ? *zp[q] : 0u;
                    zp[q] += d2 * f.nseg;
                }
        }
        mbar_wait(full + slot, round & 1u, err);
        uint32_t v[FP * FQ];
#pragma unroll
        for (uint32_t pl = 0; pl < FP; pl++) {
            const uint32_t i = (uint32_t)st * FP + pl; /* its low bits are enough */
            const uint32_t *s = reinterpret_cast<const uint32_t *>(ring + slot * stage + pl * f.pb) +
                                ((pv + i * (uint32_t)plane) & 3u);
            const uint32_t *e = reinterpret_cast<const uint32_t *>(ring + slot * stage + FP * f.pb + pl * f.cb) +
                                ((pc + i * (uint32_t)d3) & 3u);
#pragma unroll
            for (uint32_t q = 0; q < FQ; q++) /* (a plane that is not there: any value, not written) */
                v[pl * FQ + q] = run[q] += (more ? e[cz[q]] : 0u) + s[at[q]] + (PIECES ? zv[pl * FQ + q] : 0u);
        }
        __syncwarp();
        if ((threadIdx.x & 31u) == 0) mbar_arrive(empty + slot);
        if (++slot == f.stages) {
            slot = 0;
            round++;
        }
        float x[FP * FQ];
        sz3_values(v, twice, x);
#pragma unroll
        for (uint32_t pl = 0; pl < FP; pl++)
            if (FP * st + pl < d1) {
#pragma unroll
                for (uint32_t q = 0; q < FQ; q++)
                    if (threadIdx.x + nth * q < cols) o[pl * plane + nth * q] = x[pl * FQ + q];
            }
    }
}

/* ---- decompress K4-K6: the 3-D prefix sum ------------------------------ */
__global__ void k_sz3_scan_z(uint32_t *vol, uint64_t rows, uint64_t d3)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t row = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (row >= rows) return;
    uint32_t *p = vol + row * d3;
    uint32_t run = 0;
    for (uint64_t k0 = 0; k0 < d3; k0 += 32) {
        const uint64_t k = k0 + lane;
        const uint32_t v = k < d3 ? p[k] : 0u;
        const uint32_t inc = warp_incl_scan(v);
        if (k < d3) p[k] = run + inc;
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
}

/* y: a thread per (i, k), j sequential */
__global__ void k_sz3_scan_y(uint32_t *vol, uint64_t d1, uint64_t d2, uint64_t d3)
{
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= d1 * d3) return;
    const uint64_t i = t / d3, k = t % d3;
    uint32_t *p = vol + i * d2 * d3 + k;
    uint32_t run = 0;
    for (uint64_t j0 = 0; j0 < d2; j0 += SZ_SCAN_BATCH) { /* the loads of a batch ahead of its stores */
        uint32_t v[SZ_SCAN_BATCH];
#pragma unroll
        for (uint32_t u = 0; u < SZ_SCAN_BATCH; u++) v[u] = j0 + u < d2 ? p[(j0 + u) * d3] : 0u;
#pragma unroll
        for (uint32_t u = 0; u < SZ_SCAN_BATCH; u++) {
            run += v[u];
            if (j0 + u < d2) p[(j0 + u) * d3] = run;
        }
    }
}

/* x: a thread per (j, k), i sequential; writes the floats in place */
__global__ void k_sz3_scan_x(uint32_t *vol, uint64_t d1, uint64_t plane, Sz3Split twice)
{
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= plane) return;
    uint32_t run = 0;
    for (uint64_t i0 = 0; i0 < d1; i0 += SZ_SCAN_BATCH) {
        uint32_t v[SZ_SCAN_BATCH];
#pragma unroll
        for (uint32_t u = 0; u < SZ_SCAN_BATCH; u++) v[u] = i0 + u < d1 ? vol[(i0 + u) * plane + t] : 0u;
#pragma unroll
        for (uint32_t u = 0; u < SZ_SCAN_BATCH; u++) v[u] = run += v[u];
        float f[SZ_SCAN_BATCH];
        sz3_values(v, twice, f);
#pragma unroll
        for (uint32_t u = 0; u < SZ_SCAN_BATCH; u++)
            if (i0 + u < d1) reinterpret_cast<float *>(vol)[(i0 + u) * plane + t] = f[u];
    }
}

unsigned grid_for(uint64_t items, unsigned per_cta)
{
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    uint64_t g = (items + per_cta - 1) / per_cta, cap = (uint64_t)(nsm > 0 ? nsm : 1) * 16;
    return (unsigned)(g < 1 ? 1 : (g > cap ? cap : g));
}

/* Scratch layout: err[4] | sizes[nb] | offs[nb] | sums[nchunks] | total |
 * quantized volume (compress, other block sides) or the parts' carries
 * (decompress, sides 2, 4 and 8). */
struct Sz3Ws {
    uint32_t *err, *sizes;
    uint64_t *offs, *sums, *total;
    int32_t *q;
};

Sz3Ws sz3_bind(void *ws, const Sz3Dims &g)
{
    uint8_t *p = static_cast<uint8_t *>(ws);
    const uint64_t nch = (g.nblocks + SZ_CHUNK - 1) / SZ_CHUNK;
    Sz3Ws w;
    w.err = reinterpret_cast<uint32_t *>(p);
    size_t o = 16;
    w.sizes = reinterpret_cast<uint32_t *>(p + o);
    o = (o + 4 * g.nblocks + 15) & ~(size_t)15;
    w.offs = reinterpret_cast<uint64_t *>(p + o);
    o += 8 * g.nblocks;
    w.sums = reinterpret_cast<uint64_t *>(p + o);
    o += 8 * nch;
    w.total = reinterpret_cast<uint64_t *>(p + o);
    o = (o + 8 + 255) & ~(size_t)255;
    w.q = reinterpret_cast<int32_t *>(p + o);
    return w;
}

/* Offsets of `count` payload sizes; *total includes the rate table. */
cudaError_t sz3_scan(const Sz3Dims &g, const Sz3Ws &w, uint64_t count, cudaStream_t st)
{
    const uint64_t nch = (count + SZ_CHUNK - 1) / SZ_CHUNK;
    if (nch == 1) {
        k_sz3_offsets<<<1, 1024, 0, st>>>(w.sizes, count, nullptr, w.offs, g.nblocks, w.total);
        return cudaGetLastError();
    }
    k_sz3_chunk_sums<<<(unsigned)nch, 1024, 0, st>>>(w.sizes, count, w.sums);
    k_sz3_scan_sums<<<1, 1024, 0, st>>>(w.sums, nch, g.nblocks, w.total);
    k_sz3_offsets<<<(unsigned)nch, 1024, 0, st>>>(w.sizes, count, w.sums, w.offs, g.nblocks, w.total);
    return cudaGetLastError();
}

/* Block sides with the row-mapped kernels. */
bool sz3_rows(uint32_t bs) { return bs == 2 || bs == 4 || bs == 8; }

/* ... and what their decoder takes: not wide flat volumes in blocks of 4^3, one
 * or two along z, which leave 30 of its lanes idle.  Side 4, with it and with a
 * warp a block: 2000 x 2000 x 3 1482 and 775 us, 1500 x 1500 x 6 916 and 572,
 * 1000 x 1000 x 12 298 and 343, but 100 x 3000 x 3 144 and 297 (few columns to
 * sum); sides 2 and 8, 2000 x 2000 x 3: 1095 and 1347, 568 and 713. */
bool sz3_decode_rows(const Sz3Dims &g)
{
    return sz3_rows(g.bs) && !(g.bs == 4 && g.nb3 <= 2 && std::min(g.d1, g.d2) * g.d3 >= 3000);
}

/* One pass; the tiles' sizes and places use the offsets array (8 bytes a
 * block, at least 8 a tile), and the ticket and the scanner's word the last
 * two of the four scratch words before it (the first two are error words the
 * status check reads), all zeroed first. */
template <uint32_t BS, uint32_t NW = 8>
cudaError_t sz3_compress_rows(uint8_t *out, uint64_t cap, const float *x, const Sz3Dims &g, const Sz3Ws &w,
                              const Sz3Split &inv, cudaStream_t st)
{
    using C = Sz3Cm<BS, NW>;
    const uint64_t units = sz3_units<BS>(g);
    if ((units + 16) >> 32) return cudaErrorInvalidValue; /* units are counted in 32 bits */
    if constexpr (BS == 8 && NW == 8) { /* too few units for tiles of eight on every SM: 57 x 51 x 306 36 us, with four 33 */
        if (units < 8 * (uint64_t)sm_count()) return sz3_compress_rows<8, 4>(out, cap, x, g, w, inv, st);
    }
    const uint64_t ntiles = (units + NW * C::UPW - 1) / (NW * C::UPW);
    cudaError_t e = cudaMemsetAsync(w.offs, 0, 8 * ntiles, st);
    if (e != cudaSuccess) return e;
    const uint32_t fixed = SZ_CM_HEAD + NW * C::OWN + 48u, R = ring_bytes(2, fixed, zg_ring_need(C::WORST));
    const size_t smem = fixed + R;
    const void *fn = (const void *)k_sz3_compress_rows<BS, NW>;
    if ((e = set_max_smem(fn, smem)) != cudaSuccess) return e;
    const unsigned grid = scanned_grid(fn, C::THREADS, smem, ntiles, 0);
    k_sz3_compress_rows<BS, NW><<<grid, C::THREADS, smem, st>>>(x, g, inv, out, cap, w.offs, w.err + 2, w.total, R, w.err);
    return cudaGetLastError();
}

/* The tasks of a volume: strips are cut along z where there are fewer than half
 * of SZ_TASKS of them, into pieces that make at most SZ_TASKS tasks (three CTAs
 * on each of 152 SMs).  Otherwise a task goes along the whole row, and a few long
 * rows leave the device idle: 8 x 8 x 100000, side 8, 2247 us in whole rows, 54
 * in pieces; 64 x 64 x 3000, side 4, 193 and 80 (with a pass per axis
 * 345 and 113). */
constexpr uint64_t SZ_TASKS = 456;
template <uint32_t BS>
Sz3Tasks sz3_tasks(const Sz3Dims &g)
{
    using U = Sz3Un<BS>;
    Sz3Tasks t;
    t.nparts = (g.nb2 + U::PARTS - 1) / U::PARTS;
    t.nbg = (g.nb1 + U::STRIPS - 1) / U::STRIPS;
    const uint64_t strips = t.nparts * t.nbg, chunks = (g.nb3 + 31) / 32;
    const uint64_t want = strips < SZ_TASKS ? std::min(chunks, SZ_TASKS / strips) : 1;
    const uint64_t per = (chunks + want - 1) / want; /* chunks of a piece */
    t.seg = 32 * per;
    t.nseg = (chunks + per - 1) / per;
    t.ntasks = strips * t.nseg;
    return t;
}

/* Bytes of the parts' carries, and of what the pieces of the volume's rows
 * lack: no less than any smaller volume's (the sub-volumes of the OpenMP form
 * share one scratch), so there are as many pieces as any volume's rows have. */
template <uint32_t BS>
size_t sz3_carry_bytes(const Sz3Dims &g)
{
    using U = Sz3Un<BS>;
    const uint64_t crows = ((g.nb2 + U::PARTS - 1) / U::PARTS - 1) * g.d1, chunks = (g.nb3 + 31) / 32;
    const uint64_t most = SZ_TASKS * U::STRIPS * BS * U::ROWS; /* rows of a task, all tasks' */
    return 4 * (size_t)(crows * g.d3 + (chunks > 1 ? std::min(g.d1 * g.d2 * chunks, most) : 0));
}

size_t sz3_carry_bytes(const Sz3Dims &g)
{
    return g.bs == 8 ? sz3_carry_bytes<8>(g) : g.bs == 4 ? sz3_carry_bytes<4>(g) : sz3_carry_bytes<2>(g);
}

template <uint32_t FQ, uint32_t FP>
cudaError_t sz3_finish(const Sz3Dims &g, uint32_t *vol, const uint32_t *carry, uint32_t rows, Sz3Run f, const Sz3Split &twice,
                       uint64_t sms, uint32_t *err, cudaStream_t st)
{
    constexpr uint32_t FCOLS = FQ * FTH;
    /* the most rows a run (they share the carry's row) that leave no SM short of
     * runs: 384^3 with two rows, 192 runs on 152 SMs, 107 us, with one 89; 512^3
     * with two, 256 runs, 176, with one 193 */
    auto even = [&](uint64_t runs) { return runs >= 8 * sms || 5 * runs >= 4 * sms * ((runs + sms - 1) / sms); };
    for (f.R = 8; f.R > 1; f.R /= 2) /* a power of two: rows of one part */
        if (f.R * g.d3 <= FCOLS && even((g.d2 + f.R - 1) / f.R)) break;
    f.pieces = (uint32_t)((g.d3 + FCOLS - 1) / FCOLS);
    f.cz = (uint32_t)((g.d3 + f.pieces - 1) / f.pieces);
    if (f.pieces > 1) f.cz = (f.cz + 31u) & ~31u; /* <= FCOLS, a multiple of 32 */
    f.pieces = (uint32_t)((g.d3 + f.cz - 1) / f.cz);
    f.cols = f.R * f.cz;
    f.pb = (4u * f.cols + 47u) & ~15u;
    f.cb = (4u * f.cz + 47u) & ~15u;
    const uint32_t nth = (f.cols + 32u * FQ - 1) / (32u * FQ) * 32u, stage = FP * (f.pb + f.cb);
    const uint64_t runs = (g.d2 + f.R - 1) / f.R * f.pieces;
    /* three CTAs an SM, or four where that takes them all at once */
    f.stages = std::min(8u, std::max(2u, (runs > 3 * sms && runs <= 4 * sms ? 54u : 72u) * 1024u / stage));
    const uint32_t smem = f.stages * stage; /* at most 72 KB; the limit is the same in every call, from any thread */
    auto *k = f.pre ? k_sz3_finish<FQ, FP, true> : k_sz3_finish<FQ, FP, false>;
    const cudaError_t e = set_max_smem((const void *)k, 72u * 1024u);
    if (e != cudaSuccess) return e;
    k<<<(unsigned)runs, nth + 32u, smem, st>>>(vol, carry, g.d1, g.d2, g.d3, rows, f, twice, err);
    return cudaGetLastError();
}

template <uint32_t BS>
cudaError_t sz3_decompress_rows(const uint8_t *in, uint64_t avail, const Sz3Dims &g, const Sz3Ws &w, uint32_t *vol,
                                const Sz3Split &twice, cudaStream_t st)
{
    using U = Sz3Un<BS>;
    cudaError_t e;
    const uint64_t nchunks = g.nb1 * g.nb2 * ((g.nb3 + 31) / 32); /* at most nblocks: sizes and offs hold them */
    k_sz3_chunk_sizes<<<grid_for(nchunks, SZ_THREADS / 8), SZ_THREADS, 0, st>>>(in, avail, g, nchunks, w.sizes, w.err);
    if ((e = sz3_scan(g, w, nchunks, st)) != cudaSuccess) return e;
    const uint64_t nsm = (uint64_t)sm_count();
    const Sz3Tasks tk = sz3_tasks<BS>(g);
    auto *unpack = tk.nseg > 1 ? k_sz3_unpack_sum<BS, true> : k_sz3_unpack_sum<BS, false>;
    const void *fn = (const void *)unpack;
    if ((e = set_max_smem(fn, U::SMEM)) != cudaSuccess) return e;
    uint32_t *carry = reinterpret_cast<uint32_t *>(w.q);
    unpack<<<persistent_grid(fn, SZ_UN_THREADS, U::SMEM, tk.ntasks), SZ_UN_THREADS, U::SMEM, st>>>(
        in, avail, g, tk, w.offs, w.sizes, vol, carry, w.err);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const uint64_t columns = g.d1 * g.d3, rows = g.d1 * g.d2;
    if (tk.nparts > 2) k_sz3_carry<<<(unsigned)((columns + 255) / 256), 256, 0, st>>>(carry, columns, tk.nparts - 1);
    Sz3Run f = {};
    if (tk.nseg > 1) {
        uint32_t *pre = carry + (tk.nparts - 1) * columns;
        f.pre = pre;
        f.seg = tk.seg * BS;
        f.nseg = tk.nseg;
        k_sz3_piece_sums<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(vol, carry, g.d1, g.d2, g.d3, U::ROWS, f.seg, f.nseg, pre);
    }
    /* small planes (see k_sz3_finish): 45 x 60, 500 planes, 38 us against 86; 300 x 300 44 against 64;
     * 384 x 384 108 against 90 */
    return g.d2 * g.d3 <= 800 * nsm ? sz3_finish<1, 8>(g, vol, carry, U::ROWS, f, twice, nsm, w.err, st)
                                    : sz3_finish<4, 2>(g, vol, carry, U::ROWS, f, twice, nsm, w.err, st);
}

} // namespace

size_t sz3_workspace_bytes(uint64_t d1, uint64_t d2, uint64_t d3, uint32_t bs, bool compress)
{
    const Sz3Dims g = sz3_dims(d1, d2, d3, bs);
    Sz3Ws w = sz3_bind(nullptr, g);
    const size_t head = (size_t)reinterpret_cast<uintptr_t>(w.q);
    return head + (sz3_rows(bs) ? sz3_carry_bytes(g) : compress ? 4 * (size_t)(d1 * d2 * d3) : 0) + 256;
}

size_t sz3_max_stream_bytes(uint64_t d1, uint64_t d2, uint64_t d3, uint32_t bs)
{
    const Sz3Dims g = sz3_dims(d1, d2, d3, bs);
    return (size_t)(g.nblocks + (size_t)sz3_payload(32, bs * bs * bs) * g.nblocks);
}

cudaError_t sz3_compress(uint8_t *out, uint64_t cap, const float *x, uint64_t d1, uint64_t d2, uint64_t d3,
                         uint32_t bs, double eb, void *ws, uint64_t *d_size, cudaStream_t st)
{
    const Sz3Dims g = sz3_dims(d1, d2, d3, bs);
    const Sz3Ws w = sz3_bind(ws, g);
    cudaError_t e = cudaMemsetAsync(w.err + 2, 0, 8, st); /* the ticket; status words stay until checked */
    if (e != cudaSuccess) return e;
    /* the rate table is part of the stream: cap must hold it */
    if (cap < g.nblocks) return cudaErrorInvalidValue;
    const Sz3Split inv = sz3_split(0.5 / eb);
    if (sz3_rows(bs)) {
        e = bs == 2 ? sz3_compress_rows<2>(out, cap, x, g, w, inv, st)
                    : bs == 4 ? sz3_compress_rows<4>(out, cap, x, g, w, inv, st) : sz3_compress_rows<8>(out, cap, x, g, w, inv, st);
        if (e != cudaSuccess) return e;
        return d_size ? cudaMemcpyAsync(d_size, w.total, 8, cudaMemcpyDeviceToDevice, st) : cudaSuccess;
    }
    const uint64_t n = d1 * d2 * d3;
    k_sz3_quant<<<grid_for(n, 1024), 256, 0, st>>>(x, w.q, n, inv, w.err);
    const bool wb = bs * bs * bs <= 512; /* a warp per block */
    if (wb)
        k_sz3_rates<32><<<grid_for(g.nblocks, SZ_THREADS / 32), SZ_THREADS, 0, st>>>(w.q, g, out, w.sizes);
    else
        k_sz3_rates<SZ_THREADS><<<grid_for(g.nblocks, 1), SZ_THREADS, 0, st>>>(w.q, g, out, w.sizes);
    if ((e = sz3_scan(g, w, g.nblocks, st)) != cudaSuccess) return e;
    if (wb) {
        k_sz3_pack<32><<<grid_for(g.nblocks, SZ_THREADS / 32), SZ_THREADS, 4ull * bs * bs * bs * (SZ_THREADS / 32), st>>>(
            w.q, g, out, cap, w.offs, w.err);
    } else {
        const size_t smem = 4ull * bs * bs * bs;
        if ((e = set_max_smem((const void *)k_sz3_pack<SZ_THREADS>, smem)) != cudaSuccess) return e;
        k_sz3_pack<SZ_THREADS><<<grid_for(g.nblocks, 1), SZ_THREADS, smem, st>>>(w.q, g, out, cap, w.offs, w.err);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return d_size ? cudaMemcpyAsync(d_size, w.total, 8, cudaMemcpyDeviceToDevice, st) : cudaSuccess;
}

cudaError_t sz3_decompress(float *y, const uint8_t *in, uint64_t avail, uint64_t d1, uint64_t d2, uint64_t d3,
                           uint32_t bs, double eb, void *ws, cudaStream_t st)
{
    const Sz3Dims g = sz3_dims(d1, d2, d3, bs);
    const Sz3Ws w = sz3_bind(ws, g);
    uint32_t *vol = reinterpret_cast<uint32_t *>(y);
    const Sz3Split twice = sz3_split(eb * 2);
    if (sz3_decode_rows(g))
        return bs == 2   ? sz3_decompress_rows<2>(in, avail, g, w, vol, twice, st)
               : bs == 4 ? sz3_decompress_rows<4>(in, avail, g, w, vol, twice, st)
                         : sz3_decompress_rows<8>(in, avail, g, w, vol, twice, st);
    k_sz3_sizes<<<grid_for(g.nblocks, 256), 256, 0, st>>>(in, avail, g, w.sizes, w.err);
    const cudaError_t e = sz3_scan(g, w, g.nblocks, st);
    if (e != cudaSuccess) return e;
    if (bs * bs * bs <= 512)
        k_sz3_unpack<32><<<grid_for(g.nblocks, SZ_THREADS / 32), SZ_THREADS, 0, st>>>(in, avail, g, w.offs, vol, w.err);
    else
        k_sz3_unpack<SZ_THREADS><<<grid_for(g.nblocks, 1), SZ_THREADS, 0, st>>>(in, avail, g, w.offs, vol, w.err);
    const uint64_t rows = d1 * d2;
    k_sz3_scan_z<<<(unsigned)((rows * 32 + 255) / 256), 256, 0, st>>>(vol, rows, d3);
    k_sz3_scan_y<<<(unsigned)((d1 * d3 + 255) / 256), 256, 0, st>>>(vol, d1, d2, d3);
    k_sz3_scan_x<<<(unsigned)((d2 * d3 + 255) / 256), 256, 0, st>>>(vol, d1, d2 * d3, twice);
    return cudaGetLastError();
}
