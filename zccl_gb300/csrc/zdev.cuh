/*
 * zdev.cuh -- device building blocks shared by the codec kernels.
 *
 *   quantize*()          bit-exact stand-ins for (int)((double)x * (double)inv)
 *   width_of()           bit-exact stand-in for (int)log2f((float)m) + 1
 *   encode_block         one block of up to 32 elements, registers -> packed bytes
 *   decode_small_f/decode_mid_f   its inverse as floats, widths below 16 / 16..23
 *   decode_add_any       any width, added to integers
 *   decode_octet         eight elements of any block
 *   encode_octet         its inverse
 *   encode_any           any block, one element at a time
 *   Packer               MSB-first bit streams in shared memory
 *   tma_load_superset()  TMA bulk copy global -> shared
 *   store_realign()      shared -> global at any byte alignment
 *   cta_excl_scan()      block-wide exclusive scan
 *   scan_publish/scan_wait/scan_tiles   the tiles' places while they are made
 */
#ifndef ZCCL_GB300_ZDEV_CUH
#define ZCCL_GB300_ZDEV_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "zccl_err.h"
#include "zgeom.h"

/* ---------------------------------------------------------------------
 * Exact arithmetic
 * ------------------------------------------------------------------- */

/* Width thresholds, filled on the host from the host's libm: thr[w] is the
 * smallest m of bit length w whose (int)log2f((float)m) equals w (so its
 * width is w + 1), or 0xFFFFFFFF when none exists.  glibc rounds log2f of
 * 5,876 integers just below a power of two up to that power. */
struct ZWidthTable {
    uint32_t thr[33];
};

/* zg_block_bytes for a full 32-element fastmode1 block of width b <= 32: the
 * header, four sign bytes and 4 b bytes of magnitudes; a zero-width block is
 * its header alone. */
__device__ __forceinline__ uint32_t block32_bytes(uint32_t b) { return b ? 4u * b + 5u : 1u; }

/* (int)log2f((float)m) + 1 for m > 0 and 0 for m == 0, as the reference
 * computes it with the host libm (ZCCL/src/ZCCL_float.c:606). */
__device__ __forceinline__ uint32_t width_of(uint32_t m, const ZWidthTable &wt)
{
    uint32_t w = 32u - __clz(m); /* bit length; 0 for m == 0 */
    return w + (m >= wt.thr[w] ? 1u : 0u);
}

/* (int)((double)x * (double)inv) without FP64.
 *
 * The product of two floats is exact in double, and the reference truncates
 * it toward zero.  mul.rz returns the float nearest the exact product on the
 * side of zero; while |P| < 2^24 every integer is a float, so truncating the
 * rz product gives trunc(P).  Above that, the TwoProduct error-free
 * transformation (Ogita, Rump, Oishi 2005) splits P = p + e exactly with p
 * an integer-valued float, and trunc(P) = p + floor(e) (P > 0) or
 * p + ceil(e) (P < 0).  Non-finite values or |P| >= 2^31 (undefined in the
 * reference) set ZERR_RANGE in *bad. */
__device__ __forceinline__ int32_t quantize(float x, float inv, uint32_t &bad)
{
    float pz = __fmul_rz(x, inv);
    if (fabsf(pz) < 16777216.0f) return __float2int_rz(pz);
    float p = __fmul_rn(x, inv);
    float e = __fmaf_rn(x, inv, -p);
    if (!(fabsf(p) < 2147483648.0f)) {
        bad |= ZERR_RANGE;
        return 0;
    }
    float c = p > 0.0f ? floorf(e) : ceilf(e);
    return (int32_t)((uint32_t)__float2int_rz(p) + (uint32_t)__float2int_rz(c));
}

__device__ __forceinline__ uint32_t bswap32(uint32_t v) { return __byte_perm(v, 0, 0x0123); }

/* ---------------------------------------------------------------------
 * Bit streams in shared memory.  A block is a sequence of bytes; bits go
 * MSB first within a byte, which is how the reference packs sign bits and
 * the low r bits of every magnitude (ZCCL/src/ZCCL_TypeManager.c:118-421,
 * :824-848).  Whole bytes put as 8k-bit values keep their order.
 * ------------------------------------------------------------------- */

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

/* OR a finished word into shared memory (the packing buffer starts zeroed,
 * so neighbouring blocks that share a boundary word need no coordination). */
__device__ __forceinline__ void sh_or(uint32_t saddr, uint32_t v)
{
    asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(saddr), "r"(v) : "memory");
}

/* Packs MSB-first bits into a zeroed shared buffer from byte offset o.  The
 * 64-bit accumulator holds nacc pending bits right-aligned; callers keep
 * nacc < 32 before a put of up to 32 bits by calling flush(). */
struct Packer {
    uint32_t wa, nacc; /* shared address of the current word; pending bits */
    uint64_t acc;

    __device__ __forceinline__ void init(uint32_t sbase, uint32_t o)
    {
        wa = sbase + (o & ~3u);
        nacc = (o & 3u) * 8u;
        acc = 0;
    }
    __device__ __forceinline__ void put(uint32_t v, uint32_t n) /* v < 2^n, n <= 32 */
    {
        acc = (acc << n) | v;
        nacc += n;
    }
    __device__ __forceinline__ void flush()
    {
        if (nacc >= 32u) {
            nacc -= 32u;
            sh_or(wa, bswap32((uint32_t)(acc >> nacc)));
            wa += 4;
        }
    }
    __device__ __forceinline__ void finish()
    {
        flush();
        if (nacc) sh_or(wa, bswap32((uint32_t)acc << (32u - nacc)));
    }
};

/* The width byte and the sign bytes (element j at bit 31 - j of smask) of a
 * block as one 40-bit little-endian value placed at byte o of the zeroed
 * packing buffer (two word ORs). */
__device__ __forceinline__ void put_head(uint32_t sbase, uint32_t o, uint32_t b, uint32_t smask)
{
    const uint32_t q = o >> 2, s8 = (o & 3u) * 8u;
    const uint64_t v = ((uint64_t)bswap32(smask) << 8 | b) << s8; /* at most 40 + 24 bits */
    sh_or(sbase + 4u * q, (uint32_t)v);
    sh_or(sbase + 4u * q + 4u, (uint32_t)(v >> 32));
}

/* The r low bits of the 32 magnitudes m, MSB-first from byte lb: every group
 * of eight elements is r whole bytes, one 64-bit value (its two halves of
 * four fields joined by one wide multiply-add) ORed into the one to three
 * words it touches.  No chain from group to group. */
__device__ __forceinline__ void put_low_bits(uint32_t sbase, uint32_t lb, uint32_t r, const uint32_t (&m)[32])
{
    const uint32_t p = 1u << r, mask = p - 1u, p4 = 1u << (4u * r), up = 64u - 8u * r;
#pragma unroll
    for (int g = 0; g < 4; g++) {
        auto f = [&](int k) { return m[8 * g + k] & mask; };
        const uint32_t h0 = ((f(0) * p + f(1)) * p + f(2)) * p + f(3), h1 = ((f(4) * p + f(5)) * p + f(6)) * p + f(7);
        const uint64_t v = ((uint64_t)h0 * p4 + h1) << up;
        const uint32_t lo = bswap32((uint32_t)(v >> 32)), hi = bswap32((uint32_t)v); /* bytes 0 .. 3, 4 .. 7 */
        const uint32_t at = lb + (uint32_t)g * r, q = sbase + (at & ~3u), sh = (at & 3u) * 8u;
        const uint32_t end = (at & 3u) + r; /* bytes from q to the group's end */
        sh_or(q, lo << sh);
        if (end > 4u) sh_or(q + 4u, __funnelshift_l(lo, hi, sh));
        if (end > 8u) sh_or(q + 8u, __funnelshift_l(hi, 0u, sh));
    }
}

/* A full block of 32 elements: magnitudes m[] (bits from the 24th on are
 * ignored for b <= 24), the sign mask (element j at bit 31 - j) and the width
 * b, packed at byte o of the zeroed shared buffer at sbase: the header and
 * the sign bytes, the B = b/8 high bytes of each element, then the r = b%8
 * low bits of each element.  Whole words where the layout allows: one-byte
 * high parts as eight words of four elements, two-byte ones as sixteen words
 * of two, realigned to their byte offset by funnel shifts.  A zero-width
 * block is a single 0x00 byte, already in the buffer. */
__device__ __forceinline__ void encode_block(uint32_t sbase, uint32_t o, uint32_t b, uint32_t smask,
                                             const uint32_t (&m)[32], uint32_t fmt = ZG_FASTMODE1)
{
    if (b == 0) return;
    uint32_t B, r;
    zg_split(fmt, b, &B, &r);
    put_head(sbase, o, b, smask);
    const uint32_t hb = o + 5u;
    if (B == 1) {
        const uint32_t q = sbase + (hb & ~3u), sh = (hb & 3u) * 8u;
        uint32_t prev = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint32_t lo2 = __byte_perm(m[4 * k] >> r, m[4 * k + 1] >> r, 0x0040u);
            const uint32_t hi2 = __byte_perm(m[4 * k + 2] >> r, m[4 * k + 3] >> r, 0x0040u);
            const uint32_t W = __byte_perm(lo2, hi2, 0x5410u); /* bytes of elements 4k .. 4k + 3 */
            sh_or(q + 4u * (uint32_t)k, __funnelshift_l(prev, W, sh));
            prev = W;
        }
        if (sh) sh_or(q + 32u, prev >> (32u - sh));
    } else if (B == 2) {
        const uint32_t q = sbase + (hb & ~3u), sh = (hb & 3u) * 8u;
        uint32_t prev = 0;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const uint32_t W = __byte_perm(m[2 * k] >> r, m[2 * k + 1] >> r, 0x5410u); /* elements 2k, 2k + 1 */
            sh_or(q + 4u * (uint32_t)k, __funnelshift_l(prev, W, sh));
            prev = W;
        }
        if (sh) sh_or(q + 64u, prev >> (32u - sh));
    } else if (__builtin_expect(B > 2, 0)) {
        const uint32_t keep = B == 3 ? 0xFFFFFFu : 0xFFFFFFFFu;
#pragma unroll
        for (int j = 0; j < 32; j++) { /* B bytes each, in two words */
            const uint32_t at = hb + B * (uint32_t)j, H = (m[j] >> r) & keep;
            if (H) {
                sh_or(sbase + (at & ~3u), H << ((at & 3u) * 8u));
                sh_or(sbase + (at & ~3u) + 4u, __funnelshift_l(H, 0u, (at & 3u) * 8u));
            }
        }
    }
    if (r) put_low_bits(sbase, hb + 32u * B, r, m);
}

/* Bytes a .. a + 7 of the shared words w as a 64-bit big-endian value
 * (hi: bytes a .. a + 3).  Reads the three words that hold them. */
__device__ __forceinline__ void be64_at(const uint32_t *w, uint32_t a, uint32_t &hi, uint32_t &lo)
{
    const uint32_t k = a >> 2, sh = (a & 3u) * 8u;
    const uint32_t w0 = bswap32(w[k]), w1 = bswap32(w[k + 1]), w2 = bswap32(w[k + 2]);
    hi = __funnelshift_l(w1, w0, sh);
    lo = __funnelshift_l(w2, w1, sh);
}

/* The deltas of a fastmode1 block of n <= 32 elements and any width b at byte
 * o added into acc (acc[j] += delta j, wrapping; garbage from element n on):
 * the homomorphic add's form for sums that floats cannot hold.  The same code for every width (a magnitude's bytes
 * are read by two words each), so that it stays small beside the float
 * forms. */
__device__ __forceinline__ void decode_add_any(const uint32_t *w, uint32_t o, uint32_t b, uint32_t n,
                                               uint32_t (&acc)[32])
{
    const uint32_t B = b >> 3, r = b & 7u;
    uint32_t sg, unused;
    be64_at(w, o + 1, sg, unused);
    const uint32_t hb = o + 1u + ((n + 7u) >> 3), lb = hb + n * B;
    const uint32_t bmask = B >= 4 ? 0xFFFFFFFFu : (1u << (8u * B)) - 1u;
#pragma unroll
    for (int g = 0; g < 4; g++) {
        uint32_t hi = 0, lo = 0;
        be64_at(w, lb + (uint32_t)g * r, hi, lo);
        const uint32_t h2 = __funnelshift_l(lo, hi, 4u * r);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint32_t a = hb + (uint32_t)(8 * g + k) * B; /* element 8g + k's little-endian bytes */
            const uint32_t H = __funnelshift_r(w[a >> 2], w[(a >> 2) + 1], (a & 3u) * 8u) & bmask;
            const uint32_t src = k < 4 ? hi : h2;
            const uint32_t m = __funnelshift_l(src << ((uint32_t)(k & 3) * r), H, r);
            const uint32_t s = (uint32_t)((int32_t)(sg << (8 * g + k)) >> 31); /* all ones when negative */
            acc[8 * g + k] += (m ^ s) - s;
        }
    }
}

/* Integer work on the float pipe.  The codec kernels are bound by the ALU
 * pipe, which takes a warp's logic, shift, permute, add or conversion every
 * second cycle, while the float pipe takes an add or multiply-add every
 * cycle; and floats hold the integers below 2^24 exactly.  So a magnitude is
 * put together under the exponent of 2^23 (0x4B000000 | m is the float
 * 2^23 + m), which costs nothing: the permute that selects its high byte
 * takes the exponent's bytes from a second operand, 0x4B000000 >> r, so that
 * the funnel shift by r completes both. */
#define ZF_TWO23 8388608.0f
#define ZF_EXP23 0x4B000000u

/* The magnitudes of a fastmode1 block of n <= 32 elements and width b <= 15
 * as floats, their signs in sg (element j at bit 31 - j): each(j, m, sg) for
 * all 32, garbage from element n on.  The same instructions for every
 * such width, so a warp whose blocks mix them does not split; a zero-width
 * block reads (and discards) what follows its header.  All 32 elements are
 * read, whatever n: see zg_lane_slack. */
template <class Each>
__device__ __forceinline__ void decode_small_f(const uint32_t *w, uint32_t o, uint32_t b, uint32_t n, Each each)
{
    const uint32_t B = b >> 3, r = b & 7u;
    uint32_t sg, unused;
    be64_at(w, o + 1, sg, unused);
    const uint32_t hb = o + 1u + ((n + 7u) >> 3), lb = hb + n * B;
    const uint32_t k0 = hb >> 2, sh = (hb & 3u) * 8u;
    const uint32_t bk = B ? 1u : 0u, s0 = B ? 0x7650u : 0x7654u; /* byte 0: high byte k, or the exponent word's zero byte */
    const uint32_t ex = ZF_EXP23 >> r;             /* its low 17 bits are zero */
    const uint32_t p1 = 1u << r, p2 = p1 * p1, p3 = p2 * p1;
    uint32_t prev = w[k0];
#pragma unroll
    for (int g = 0; g < 4; g++) {
        const uint32_t n1 = w[k0 + 2 * g + 1], n2 = w[k0 + 2 * g + 2];
        const uint32_t A0 = __funnelshift_r(prev, n1, sh), A1 = __funnelshift_r(n1, n2, sh);
        prev = n2;
        uint32_t hi, lo;
        be64_at(w, lb + (uint32_t)g * r, hi, lo);
        const uint32_t h2 = __funnelshift_l(lo, hi, 4u * r); /* fields 4 .. 7 on top */
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint32_t H = __byte_perm(k < 4 ? A0 : A1, ex, s0 + (uint32_t)(k & 3) * bk);
            const uint32_t src = k < 4 ? hi : h2;
            const uint32_t f = (k & 3) == 0 ? src : src * ((k & 3) == 1 ? p1 : (k & 3) == 2 ? p2 : p3);
            const float m = __uint_as_float(__funnelshift_l(f, H, r)) - ZF_TWO23;
            each(8 * g + k, m, sg);
        }
    }
}

/* The same for a width of 16 .. 23 (two high bytes per magnitude). */
template <class Each>
__device__ __forceinline__ void decode_mid_f(const uint32_t *w, uint32_t o, uint32_t b, uint32_t n, Each each)
{
    const uint32_t r = b & 7u;
    uint32_t sg, unused;
    be64_at(w, o + 1, sg, unused);
    const uint32_t hb = o + 1u + ((n + 7u) >> 3), lb = hb + 2u * n;
    const uint32_t k0 = hb >> 2, sh = (hb & 3u) * 8u;
    const uint32_t ex = ZF_EXP23 >> r; /* its low 16 bits are zero */
    const uint32_t p1 = 1u << r, p2 = p1 * p1, p3 = p2 * p1;
    uint32_t prev = w[k0];
#pragma unroll
    for (int g = 0; g < 4; g++) {
        uint32_t hi, lo;
        be64_at(w, lb + (uint32_t)g * r, hi, lo);
        const uint32_t h2 = __funnelshift_l(lo, hi, 4u * r); /* fields 4 .. 7 on top */
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
            const uint32_t nx = w[k0 + 4 * g + (k >> 1) + 1];
            const uint32_t A = __funnelshift_r(prev, nx, sh); /* the high bytes of elements 8g + k, 8g + k + 1 */
            prev = nx;
            const uint32_t src = k < 4 ? hi : h2;
            const uint32_t f0 = (k & 3) == 0 ? src : src * p2, f1 = src * ((k & 3) == 0 ? p1 : p3);
            each(8 * g + k, __uint_as_float(__funnelshift_l(f0, __byte_perm(A, ex, 0x7610), r)) - ZF_TWO23, sg);
            each(8 * g + k + 1, __uint_as_float(__funnelshift_l(f1, __byte_perm(A, ex, 0x7632), r)) - ZF_TWO23,
                 sg);
        }
    }
}

/* m >= 0, negated where sg has element j's sign bit: a shift, which the
 * compiler may put on the multiply pipe, and one logic operation (a select on
 * the bit takes two; the add of two 384^3 streams 135.4 -> 131.5 us). */
__device__ __forceinline__ float with_sign(float m, uint32_t sg, int j) { return copysignf(m, __uint_as_float(sg << j)); }

/* max(a, |b|, |c|), a >= 0, in one operation. */
__device__ __forceinline__ float max3_abs(float a, float b, float c)
{
    float d;
    asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

/* The same, NaN if one of them is. */
__device__ __forceinline__ float max3_abs_nan(float a, float b, float c)
{
    float d;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

/* 1.0f with the sign of bit 31 of s. */
__device__ __forceinline__ float sign_of(uint32_t s) { return __uint_as_float((s & 0x80000000u) | 0x3F800000u); }

/* N + 1 consecutive floats x become N deltas of their quantized values:
 * m[j] = 0x4B000000 | |d_j| (the float 2^23 + |d_j|), the signs in smask (d_j
 * at bit N - 1 - j), mx = max |d_j|, q0 = the first value.  One multiply-add
 * rounded toward zero, |x| inv + 2^23, has trunc(|x| inv) in its low bits:
 * the product enters it unrounded.  True when every product stayed below 2^23
 * and every delta below 2^22, which makes all of this exact; otherwise
 * (NaN and infinity included) the block is done again by quantize_exact. */
template <int N, int X>
__device__ __forceinline__ bool quantize_deltas(const float (&x)[X], float inv, uint32_t (&m)[N], uint32_t &smask,
                                                uint32_t &mx, int32_t &q0)
{
    uint32_t seen = 0;
    float mf = 0.f, qp = 0.f, dp = 0.f;
    smask = 0;
    static_assert(N % 2 == 0, "the largest of two deltas at a time");
#pragma unroll
    for (int j = 0; j <= N; j++) {
        const float t = __fmaf_rz(fabsf(x[j]), inv, ZF_TWO23);
        seen |= __float_as_uint(t);
        const float q = __fmaf_rn(sign_of(__float_as_uint(x[j])), t - ZF_TWO23, 0.f); /* never -0 */
        if (j == 0) {
            q0 = __float2int_rn(q);
        } else {
            const float d = q - qp;
            smask = __funnelshift_l(__float_as_uint(d), smask, 1);
            if (j % 2 == 0) mf = max3_abs(mf, dp, d);
            dp = d;
            m[j - 1] = __float_as_uint(fabsf(d) + ZF_TWO23);
        }
        qp = q;
    }
    mx = (uint32_t)mf;
    /* an exponent above 2^23's has a bit that 2^23's lacks; NaN too */
    return !(seen & ~(ZF_EXP23 | 0x7FFFFFu)) && mf < 4194304.f;
}

/* The same in integers, exact wherever the reference is defined; x(j) gives
 * float j.  m[j] is the magnitude alone. */
template <int N, class X>
__device__ __forceinline__ void quantize_exact(X x, float inv, uint32_t (&m)[N], uint32_t &smask, uint32_t &mx,
                                               int32_t &q0, uint32_t &bad)
{
    int32_t qp = q0 = quantize(x(0), inv, bad);
    mx = smask = 0;
#pragma unroll
    for (int j = 0; j < N; j++) {
        const int32_t q = quantize(x(j + 1), inv, bad);
        const int32_t d = (int32_t)((uint32_t)q - (uint32_t)qp);
        qp = q;
        smask = (smask << 1) | ((uint32_t)d >> 31);
        m[j] = (uint32_t)abs(d); /* |INT_MIN| wraps to 2^31, as in the reference */
        mx = max(mx, m[j]);
    }
}

/* Eight elements of a block: octet g (elements 8g .. 8g + 7) of the block of
 * n elements and width b at byte o of the shared words w: d[k] = the int32
 * delta of element 8g + k, 0 past the block's end.  G = ceil(L / 8)
 * neighbouring lanes hold a block, so a warp's shared reads are those of
 * 32 / G consecutive blocks, each read as one run.
 *   - the octet's signs are one byte;
 *   - its r low bits per element fill r whole bytes (byte g r of the low
 *     section on), read as one window whose two 4r-bit halves give four
 *     fields each;
 *   - its high bytes are 8 (B = 1) or 16 (B = 2) consecutive bytes, realigned
 *     by funnel shifts; for B = 0 the byte permute selects a zero byte, so
 *     lanes whose blocks mix B = 0 and 1 take the same instructions, and a
 *     zero-width block reads (and discards) whatever follows its header.
 * Reads up to zg_octet_slack(L) bytes past a block's end (a lane whose octet is
 * past it reads octet 0; INSIDE: there is none). */
template <bool INSIDE = false>
__device__ __forceinline__ void decode_octet(const uint32_t *w, uint32_t o, uint32_t b, uint32_t n, uint32_t g,
                                             uint32_t fmt, uint32_t (&d)[8])
{
    uint32_t B = b >> 3, r = b & 7u;
    if (fmt != ZG_FASTMODE1) {
        B = b ? min(B + 1u, 4u) : 0u;
        r = 0;
    }
    const uint32_t ns = (n + 7u) >> 3; /* a segment's last block may be shorter than L */
    const uint32_t gr = INSIDE || 8u * g < n ? g : 0u; /* the octet that is read */
    const uint32_t sg = (uint32_t)reinterpret_cast<const uint8_t *>(w)[o + 1u + gr] << 24; /* element k: bit 31 - k */
    const uint32_t hb = o + 1u + ns, la = hb + B * n + gr * r;
    uint32_t F0, F1;
    {
        const uint32_t k = la >> 2, sh = (la & 3u) * 8u;
        const uint32_t w0 = w[k], w1 = w[k + 1], w2 = w[k + 2];
        F0 = bswap32(__funnelshift_r(w0, w1, sh));
        F1 = __funnelshift_l(bswap32(__funnelshift_r(w1, w2, sh)), F0, 4u * r); /* fields 4 .. 7 on top */
    }
    const uint32_t r2 = 2u * r, r3 = 3u * r;
    auto put = [&](int k, uint32_t H) {
        const uint32_t F = k < 4 ? F0 : F1;
        const uint32_t f = (k & 3) == 0 ? F : F << ((k & 3) == 1 ? r : (k & 3) == 2 ? r2 : r3);
        const uint32_t m = __funnelshift_l(f, H, r); /* H << r | the top r bits of f */
        const uint32_t s = (uint32_t)((int32_t)(sg << k) >> 31);
        d[k] = (m ^ s) - s;
    };
    if (B <= 1) {
        const uint32_t a = hb + 8u * gr, k0 = a >> 2, sh = (a & 3u) * 8u;
        const uint32_t w0 = w[k0], w1 = w[k0 + 1], w2 = w[k0 + 2];
        const uint32_t A0 = __funnelshift_r(w0, w1, sh), A1 = __funnelshift_r(w1, w2, sh);
        const uint32_t zsel = B ? 0x4440u : 0x4444u; /* selector nibble 4: a byte of the zero operand */
#pragma unroll
        for (int k = 0; k < 8; k++) put(k, __byte_perm(k < 4 ? A0 : A1, 0, B ? 0x4440u | (uint32_t)(k & 3) : zsel));
    } else if (B == 2) {
        const uint32_t a = hb + 16u * gr, k0 = a >> 2, sh = (a & 3u) * 8u;
        uint32_t prev = w[k0];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t nx = w[k0 + i + 1];
            const uint32_t A = __funnelshift_r(prev, nx, sh);
            prev = nx;
            put(2 * i, A & 0xFFFFu);
            put(2 * i + 1, A >> 16);
        }
    } else {
        const uint32_t bmask = B >= 4 ? 0xFFFFFFFFu : 0xFFFFFFu;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint32_t a = hb + (8u * gr + (uint32_t)k) * B;
            put(k, __funnelshift_r(w[a >> 2], w[(a >> 2) + 1], (a & 3u) * 8u) & bmask);
        }
    }
    if (8u * g + 8u > n) { /* the block's end, or a lane without an octet (n = 0) */
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (8u * g + (uint32_t)k >= n) d[k] = 0;
    }
}

/* v (its low bytes first) ORed into the zeroed buffer from byte at on. */
__device__ __forceinline__ void or_bytes(uint32_t sbase, uint32_t at, uint64_t v)
{
    const uint32_t q = sbase + (at & ~3u), sh = (at & 3u) * 8u, lo = (uint32_t)v, hi = (uint32_t)(v >> 32);
    const uint32_t w0 = lo << sh, w1 = __funnelshift_l(lo, hi, sh), w2 = __funnelshift_l(hi, 0u, sh);
    if (w0) sh_or(q, w0);
    if (w1) sh_or(q + 4u, w1);
    if (w2) sh_or(q + 8u, w2);
}

/* The magnitudes m of octet g of a block of n elements whose high bytes begin
 * at byte h of the zeroed buffer at sbase: B high bytes each, then (from
 * h + n B on) r low bits each, most significant first.  Four elements' low
 * bits at a time are joined in 32 bits. */
__device__ __forceinline__ void put_octet(uint32_t sbase, uint32_t h, uint32_t n, uint32_t g, uint32_t B, uint32_t r,
                                          const uint32_t (&m)[8])
{
    if (B == 1) {
        const uint32_t lo = __byte_perm(__byte_perm(m[0] >> r, m[1] >> r, 0x0040), __byte_perm(m[2] >> r, m[3] >> r, 0x0040), 0x5410);
        const uint32_t hi = __byte_perm(__byte_perm(m[4] >> r, m[5] >> r, 0x0040), __byte_perm(m[6] >> r, m[7] >> r, 0x0040), 0x5410);
        or_bytes(sbase, h + 8u * g, (uint64_t)hi << 32 | lo);
    } else if (B > 1) {
        const uint32_t keep = B >= 4 ? 0xFFFFFFFFu : (1u << (8u * B)) - 1u;
#pragma unroll
        for (int k = 0; k < 8; k++) or_bytes(sbase, h + (8u * g + (uint32_t)k) * B, (m[k] >> r) & keep);
    }
    if (r) { /* r bytes */
        const uint32_t mask = (1u << r) - 1u;
        uint32_t a = m[0] & mask, b = m[4] & mask;
#pragma unroll
        for (int k = 1; k < 4; k++) {
            a = a << r | (m[k] & mask);
            b = b << r | (m[4 + k] & mask);
        }
        /* the 8 r bits at the top of 64, bytes first to last upward */
        const uint32_t s = 32u - 4u * r, at = a << s, bt = b << s;
        const uint32_t hi = at | (bt >> (4u * r)), lo = bt << s;
        or_bytes(sbase, h + n * B + g * r, (uint64_t)bswap32(lo) << 32 | bswap32(hi));
    }
}

/* The inverse of decode_octet: octet g of a block of n elements and width b
 * into the zeroed buffer at sbase from byte o on; s8: its signs (element k at
 * bit 7 - k); m: its magnitudes (bits from the 24th on are ignored for
 * b <= 24); both 0 past the block's end.  Octet 0 writes the header. */
__device__ __forceinline__ void encode_octet(uint32_t sbase, uint32_t o, uint32_t b, uint32_t n, uint32_t g,
                                             uint32_t s8, const uint32_t (&m)[8], uint32_t fmt)
{
    if (b == 0) return;
    uint32_t B, r;
    zg_split(fmt, b, &B, &r);
    if (g == 0)
        or_bytes(sbase, o, b | s8 << 8);
    else
        or_bytes(sbase, o + 1u + g, s8);
    put_octet(sbase, o + 1u + ((n + 7u) >> 3), n, g, B, r, m);
}

/* A block of n elements, one element at a time: separate streams for the
 * header, the sign bits, the high bytes and the low bits (a segment's short
 * last block).  elem(j, neg, mag) gives element j. */
template <class Elem>
__device__ __forceinline__ void encode_any(uint32_t sbase, uint32_t o, uint32_t b, uint32_t n,
                                           Elem elem, uint32_t fmt = ZG_FASTMODE1)
{
    if (b == 0) return;
    uint32_t B, r;
    zg_split(fmt, b, &B, &r);
    const uint32_t ns = (n + 7) >> 3;
    const uint32_t mask = r ? (1u << r) - 1u : 0u;
    Packer ph, ps, pb, pl;
    ph.init(sbase, o);
    ph.put(b, 8);
    ph.finish();
    ps.init(sbase, o + 1);
    pb.init(sbase, o + 1 + ns);
    pl.init(sbase, o + 1 + ns + B * n);
#pragma unroll 1
    for (uint32_t j = 0; j < n; j++) {
        uint32_t neg, mg;
        elem(j, neg, mg);
        ps.put(neg, 1);
        ps.flush();
        if (B) {
            pb.put(bswap32(mg >> r) >> (32u - 8u * B), 8u * B);
            pb.flush();
        }
        if (r) {
            pl.put(mg & mask, r);
            pl.flush();
        }
    }
    ps.finish();
    if (B) pb.finish();
    if (r) pl.finish();
}

/* v[j] for a runtime j, as selects so that the register array stays in
 * registers (short tail blocks only). */
__device__ __forceinline__ uint32_t pick(const uint32_t (&v)[32], uint32_t j)
{
    uint32_t r = v[0];
#pragma unroll
    for (int k = 1; k < 32; k++) r = (uint32_t)k == j ? v[k] : r;
    return r;
}

/* Barrier `id` (1..15) over the first n threads of the CTA (a multiple of
 * 32), for kernels whose warps split into groups; id 0 is __syncthreads. */
__device__ __forceinline__ void named_sync(uint32_t id, uint32_t n)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

/* ---------------------------------------------------------------------
 * TMA (cp.async.bulk) global -> shared, completion on an mbarrier
 * ------------------------------------------------------------------- */

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

/* One arrival on a barrier (release at CTA scope: the caller's earlier
 * shared-memory writes are visible to whoever sees the phase complete). */
__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

/* One try for phase `parity` of the barrier (the hardware may hold the
 * thread for up to the given time, in ns, before it answers). */
__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity, uint32_t ns)
{
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity), "r"(ns)
        : "memory");
    return done != 0;
}

/* Wait for phase `parity` of the barrier to complete.  Gives up after about
 * 2^32 SM clock cycles (two seconds or more) and reports ZERR_TIMEOUT
 * instead of hanging; a wait that spans other stages of a pipeline (which
 * may themselves wait on other CTAs) stays well inside that limit. */
static __device__ __noinline__ void mbar_wait_slow(uint32_t addr, uint32_t parity, uint32_t *err)
{
    const long long t0 = clock64();
    for (uint32_t it = 0; it < (1u << 26); it++) {
#pragma unroll 1
        for (uint32_t k = 0; k < 16; k++)
            if (mbar_try(addr, parity, 20000u)) return;
        if (clock64() - t0 > (1ll << 32)) break;
    }
    atomicOr(err, ZERR_TIMEOUT);
}
__device__ __forceinline__ void mbar_wait(uint64_t *bar, uint32_t parity, uint32_t *err)
{
    const uint32_t addr = smem_u32(bar);
    if (!mbar_try(addr, parity, 1000u)) mbar_wait_slow(addr, parity, err);
}

__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void bulk_g2s(void *sdst, const void *gsrc, uint32_t bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(sdst)),
        "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

/* Four bytes from global to shared memory, asynchronously (both addresses
 * multiples of 4); cp_async_arrive: one arrival on the barrier when all the
 * thread's copies so far have landed. */
__device__ __forceinline__ void cp_async4(uint32_t sdst, const void *gsrc)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sdst), "l"(gsrc) : "memory");
}
/* Sixteen bytes (both addresses multiples of 16), or sixteen zeros where they
 * are not wanted (gsrc may then be anything). */
__device__ __forceinline__ void cp_async16_or_zero(uint32_t sdst, const void *gsrc, bool want)
{
    asm volatile("{\n .reg .pred p;\n .reg .b32 z;\n"
                 " setp.ne.u32 p, %2, 0;\n mov.u32 z, 0;\n"
                 " @p cp.async.cg.shared.global [%0], [%1], 16;\n"
                 " @!p st.shared.v4.b32 [%0], {z, z, z, z};\n}"
                 ::"r"(sdst), "l"(gsrc), "r"((uint32_t)want)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <uint32_t N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
/* Shared accesses by address (a swizzled layout computes its own). */
__device__ __forceinline__ void st_shared_v4(uint32_t sa, float x, float y, float z, float w)
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(sa), "f"(x), "f"(y), "f"(z), "f"(w)
                 : "memory");
}
__device__ __forceinline__ void st_shared_f32(uint32_t sa, float x)
{
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(sa), "f"(x) : "memory");
}

__device__ __forceinline__ float4 ld_shared_v4(uint32_t sa)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(sa)
                 : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_shared_u32(uint32_t sa)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(sa) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_shared_u8(uint32_t sa)
{
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(sa) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ld_shared_u16(uint32_t sa)
{
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(sa) : "memory");
    return v;
}
__device__ __forceinline__ void st_shared_u16(uint32_t sa, uint32_t v)
{
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(sa), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ float ld_shared_f32(uint32_t sa)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(sa) : "memory");
    return v;
}

/* TMA tensor load of the box at (c0, c1) of a 2-D map into shared memory,
 * completing on the mbarrier (whose byte count the caller arms). */
__device__ __forceinline__ void tma_load_2d(uint32_t sa, const void *map, int32_t c0, int32_t c1, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
            "r"(sa),
        "l"((uint64_t)(uintptr_t)map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
        : "memory");
}

/* One thread: TMA bulk copy of the 16-byte-aligned superset
 * [floor16(g), ceil16(g + nbytes)) into the 16-byte-aligned buffer s, arming
 * the barrier with its byte count.  The superset only adds bytes of 16-byte
 * chunks that already contain bytes of the range, so it never touches a page
 * the range does not.  The range starts at s + (g & 15). */
__device__ __forceinline__ void tma_load_superset(uint8_t *s, const uint8_t *g, uint32_t nbytes,
                                                  uint64_t *bar)
{
    uintptr_t a0 = (uintptr_t)g & ~(uintptr_t)15u;
    uintptr_t a1 = nbytes ? ((uintptr_t)g + nbytes + 15u) & ~(uintptr_t)15u : a0; /* no bytes: g may be anywhere */
    fence_proxy_async_smem(); /* earlier generic accesses of s before the async write */
    mbar_expect_tx(bar, (uint32_t)(a1 - a0));
    if (a1 > a0) bulk_g2s(s, (const void *)a0, (uint32_t)(a1 - a0), bar);
}

/* Write shared bytes s[0, nbytes) to global [g, g + nbytes) for any
 * alignment of g.  16-byte-aligned global chunks get one vector store each,
 * assembled from two aligned shared loads and funnel shifts; the ragged
 * ends (shared with neighbouring tiles) are stored byte by byte.  s must be
 * 16-byte aligned with 32 readable bytes of slack.  Called by all threads. */
__device__ __forceinline__ void store_realign(uint8_t *g, const uint8_t *s, uint32_t nbytes, uint32_t tid,
                                              uint32_t nt)
{
    const uintptr_t g0 = (uintptr_t)g, g1 = g0 + nbytes;
    const uintptr_t a0 = (g0 + 15u) & ~(uintptr_t)15u, a1 = g1 & ~(uintptr_t)15u;
    if (a1 <= a0) {
        for (uint32_t i = tid; i < nbytes; i += nt) g[i] = s[i];
        return;
    }
    const uint32_t d = (uint32_t)(a0 - g0); /* shared offset of the first aligned chunk */
    const uint32_t tail = (uint32_t)(g1 - a1);
    for (uint32_t i = tid; i < d + tail; i += nt) { /* ragged ends, any thread count */
        const uint32_t k = i < d ? i : (uint32_t)(a1 - g0) + (i - d);
        g[k] = s[k];
    }
    const uint32_t nch = (uint32_t)((a1 - a0) >> 4), q = d >> 2, sh = (d & 3u) * 8u;
    const uint4 *s4 = reinterpret_cast<const uint4 *>(s);
    uint4 *g4 = reinterpret_cast<uint4 *>(a0);
    /* four chunks a thread in flight: one warp writes a tile alone */
#pragma unroll 1
    for (uint32_t c0 = tid; c0 < nch; c0 += 4u * nt) {
        uint4 lo[4], hi[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
            const uint32_t c = min(c0 + u * nt, nch - 1u);
            lo[u] = s4[c];
            hi[u] = s4[c + 1];
        }
        /* q is the same for every thread of the tile: uniform branches */
        if (q & 1u) {
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                lo[u].x = lo[u].y, lo[u].y = lo[u].z, lo[u].z = lo[u].w, lo[u].w = hi[u].x;
                hi[u].x = hi[u].y, hi[u].y = hi[u].z, hi[u].z = hi[u].w;
            }
        }
        if (q & 2u) {
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                lo[u].x = lo[u].z, lo[u].y = lo[u].w, lo[u].z = hi[u].x, lo[u].w = hi[u].y;
                hi[u].x = hi[u].z;
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
            uint4 v;
            v.x = __funnelshift_r(lo[u].x, lo[u].y, sh);
            v.y = __funnelshift_r(lo[u].y, lo[u].z, sh);
            v.z = __funnelshift_r(lo[u].z, lo[u].w, sh);
            v.w = __funnelshift_r(lo[u].w, hi[u].x, sh);
            if (c0 + u * nt < nch) g4[c0 + u * nt] = v;
        }
    }
}

__device__ __forceinline__ void store_realign(uint8_t *g, const uint8_t *s, uint32_t nbytes)
{
    store_realign(g, s, nbytes, threadIdx.x, blockDim.x);
}

/* ---------------------------------------------------------------------
 * Block-wide exclusive scans (blockDim.x <= 1024, multiple of 32).
 * `wsum` is shared scratch of 33 words.
 * ------------------------------------------------------------------- */
__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v)
{
    uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

/* Exclusive scan of v over the first n threads of the CTA, synchronised
 * on barrier `id` (wrapping uint32 add, so it also serves int32 sums);
 * *total receives the sum of all v. */
__device__ __forceinline__ uint32_t grp_excl_scan(uint32_t v, uint32_t *wsum, uint32_t *total, uint32_t n,
                                                  uint32_t id)
{
    uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = n >> 5;
    uint32_t inc = warp_incl_scan(v);
    if (lane == 31) wsum[warp] = inc;
    named_sync(id, n);
    if (warp == 0) {
        uint32_t t = lane < nw ? wsum[lane] : 0u;
        uint32_t ti = warp_incl_scan(t);
        if (lane < nw) wsum[lane] = ti - t;
        if (lane == 31) wsum[32] = ti;
    }
    named_sync(id, n);
    uint32_t r = wsum[warp] + inc - v;
    *total = wsum[32];
    named_sync(id, n);
    return r;
}

/* The same with one barrier: every warp reads all warp sums.  Callers
 * alternate between two scratch arrays on consecutive calls, so that a
 * warp's next write cannot overtake a slower warp's read. */
__device__ __forceinline__ uint32_t grp_excl_scan1(uint32_t v, uint32_t *ws, uint32_t *total, uint32_t n,
                                                   uint32_t id)
{
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = n >> 5;
    const uint32_t inc = warp_incl_scan(v);
    if (lane == 31) ws[warp] = inc;
    named_sync(id, n);
    const uint32_t t = lane < nw ? ws[lane] : 0u;
    *total = __reduce_add_sync(0xffffffffu, t);
    return __reduce_add_sync(0xffffffffu, lane < warp ? t : 0u) + inc - v;
}

/* grp_excl_scan over the whole CTA. */
__device__ __forceinline__ uint32_t cta_excl_scan(uint32_t v, uint32_t *wsum, uint32_t *total)
{
    return grp_excl_scan(v, wsum, total, blockDim.x, 0);
}

/* ---------------------------------------------------------------------
 * The tiles' places: an exclusive scan of their sizes while they are being
 * made.  status[t] packs a 2-bit flag (1 = the size of tile t, 2 = the
 * inclusive sum through t) over a 62-bit value.  Workers publish sizes (a
 * stream's first tile its inclusive sum at once); one warp of the grid, in
 * the CTA that started first, turns them into sums in ticket order, up to 256
 * a round; each tile's placer polls its own word only.  (With a decoupled
 * look-back in every CTA instead, every placer read its 256 predecessors and
 * more each round, and its chain of look-back and write-out set the pace of
 * the add: 384^3 floats in 111 us with all decoding left out.)  Tickets are
 * handed out in order, so the tile that the scan waits for belongs to a CTA
 * that is running and that waits for no later tile before it publishes.
 * ------------------------------------------------------------------- */
/* Polls before a wait gives up (a second or more; callers may pass a
 * smaller limit). */
#define SCAN_SPIN_LIMIT (1u << 22)
#define SCAN_ALONE (1u << 20) /* polls without any tile handed out */
#define SCAN_SIZE (1ull << 62)
#define SCAN_SUM (2ull << 62)
#define SCAN_VAL (SCAN_SIZE - 1ull)

/* A status word carries its flag and its value together, and a reader
 * uses nothing else that the writer produced, so relaxed device-scope
 * accesses suffice: no acquire (which would keep a lane's eight loads from
 * overlapping) and no release (which would hold the store until the
 * thread's earlier output stores complete). */
__device__ __forceinline__ void st_flag(uint64_t *p, uint64_t v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ uint64_t ld_flag(const uint64_t *p)
{
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

/* One thread: tile t's size (its sum, for a stream's first tile). */
__device__ __forceinline__ void scan_publish(uint64_t *status, uint64_t t, uint32_t size, bool first)
{
    st_flag(status + t, (first ? SCAN_SUM : SCAN_SIZE) | size);
}

/* All lanes of a warp: the inclusive sum through a tile of `size` bytes, waiting
 * for it; SCAN_NONE and ZERR_TIMEOUT after `limit` polls.  With no scanner (see
 * scan_tiles) the tile before gives it, which is looked at too from the
 * SCAN_HELP-th poll on (64: the add of two 512^3 streams 0.6 % slower than
 * without this look; 16, which the scanner's usual delay reaches, 2 %). */
#define SCAN_NONE (~0ull)
#define SCAN_HELP 64u
static __device__ __noinline__ uint64_t scan_wait_slow(uint64_t *word, uint32_t size, uint32_t limit, uint32_t *err)
{
    uint64_t v = ld_flag(word);
#pragma unroll 1
    for (uint32_t i = 0; (v >> 62) != 2u; i++) {
        if (i >= limit) {
            atomicOr(err, ZERR_TIMEOUT);
            break;
        }
        if ((v >> 62) == 1u) { /* not a stream's first tile */
            const uint64_t before = ld_flag(word - 1);
            if ((before >> 62) == 2u) {
                v = SCAN_SUM | ((before & SCAN_VAL) + size); /* as the scanner would have it */
                st_flag(word, v);
                break;
            }
        }
        __nanosleep(64);
        v = ld_flag(word);
    }
    return v;
}

__device__ __forceinline__ uint64_t scan_wait(uint64_t *word, uint32_t size, uint32_t limit, uint32_t *err)
{
    uint64_t v = ld_flag(word);
#pragma unroll 1
    for (uint32_t i = 0; i < SCAN_HELP && (v >> 62) != 2u; i++) { /* every lane reads the same word, but not at the same time */
        __nanosleep(64);
        v = ld_flag(word);
    }
    if ((v >> 62) != 2u) v = scan_wait_slow(word, size, limit, err);
    return __shfl_sync(0xffffffffu, (v >> 62) == 2u ? v & SCAN_VAL : SCAN_NONE, 0);
}

/* The scanning warp, over n tiles.  A tile that never publishes makes it
 * give up after `limit` polls: ZERR_TIMEOUT is set, the tile's size counts
 * as 0 and the scan goes on, so that no placer waits forever.  While the tile
 * waited for is not yet handed out (its CTA is still waiting for room on the
 * device), polls count 64-fold less.
 * If no tile at all has been handed out for a second or more, other work may hold
 * all of the device but this CTA's place: the scanner leaves it to a CTA that
 * works, and the placers take their sums from one another (scan_wait). */
static __device__ __noinline__ void scan_tiles(uint64_t *status, uint64_t n, const uint32_t *ticket, uint32_t *err,
                                               uint32_t limit)
{
    const uint32_t lane = threadIdx.x & 31u;
    uint64_t pos = 0, run = 0; /* tiles summed, their sum (within a stream) */
    uint32_t polls = 0, idle = 0;
#pragma unroll 1
    while (pos < n) {
        uint64_t v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const uint64_t i = pos + 32u * (uint32_t)k + lane;
            v[k] = i < n ? ld_flag(status + i) : 0ull;
        }
        uint32_t done = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (done == 32u * (uint32_t)k) { /* uniform: every tile before these was ready */
                const uint32_t flag = (uint32_t)(v[k] >> 62);
                const uint32_t gap = ~__ballot_sync(0xffffffffu, flag != 0u);
                const uint32_t cnt = gap ? (uint32_t)__ffs(gap) - 1u : 32u; /* ready in a row */
                const uint32_t sums = __ballot_sync(0xffffffffu, flag == 2u) & ((2u << lane) - 1u); /* up to this lane */
                const uint32_t inc = warp_incl_scan(flag == 1u && lane < cnt ? (uint32_t)v[k] : 0u);
                const uint32_t from = sums ? 31u - (uint32_t)__clz(sums) : 0u;
                const uint64_t at = __shfl_sync(0xffffffffu, v[k] & SCAN_VAL, from);
                const uint32_t at_inc = __shfl_sync(0xffffffffu, inc, from);
                const uint64_t sum = sums ? at + (inc - at_inc) : run + inc;
                if (flag == 1u && lane < cnt) st_flag(status + pos + 32u * (uint32_t)k + lane, SCAN_SUM | sum);
                if (cnt) run = __shfl_sync(0xffffffffu, sum, cnt - 1u);
                done += cnt;
            }
        }
        pos += done;
        if (done) {
            polls = 0;
            continue;
        }
        __nanosleep(32);
        if (pos == 0 && polls >= SCAN_ALONE && *(volatile const uint32_t *)ticket == 0u) return;
        if (++polls < limit) continue;
        if (limit == SCAN_SPIN_LIMIT && *(volatile const uint32_t *)ticket <= pos && ++idle < 64u) {
            polls = 0;
            continue;
        }
        if (lane == 0) { /* give up */
            atomicOr(err, ZERR_TIMEOUT);
            st_flag(status + pos, SCAN_SUM | run);
        }
        pos++;
        limit = 16;
        polls = 0;
    }
}

#endif
