/* The coefficient part of an H.261 macroblock on the device: each coded
 * block's TCOEFF codes in transmission (zig-zag) order and its EOB, as the
 * reference's host writer sends them (src/h261_macroblock.c:196-262):
 *
 *   - an intra block's DC level as its 8-bit value;
 *   - an inter block's first coefficient, when it is +-1, as the short code
 *     1s (s the sign);
 *   - every other nonzero level after `run` zeros as the table code plus a
 *     sign bit, or the 20-bit escape (000001, 6-bit run, 8-bit level) where
 *     the table has no entry;
 *   - EOB (10) after the block.
 *
 * A warp codes a macroblock from its levels in shared memory -- in a small
 * step the encode kernel's, as soon as it has them, in a larger one the codes
 * kernel's (bitstream.cu), which loads them: the levels are put into
 * transmission order, each block gets a mask of its nonzero positions, and
 * then every code of the macroblock -- the levels of all of its blocks and an
 * EOB after each -- has a lane of its own.  The codes are ORed into a zeroed
 * word buffer, MSB first. */
#pragma once

#include <cstddef>
#include <cstdint>

#include "h261b_device.h"

namespace h261b {

/* MB string words: six blocks of an 8-bit DC or a first code, 63 escapes of
 * 20 bits and an EOB */
constexpr int VLC_MB_WORDS = H261B_VLC_MB_WORDS;

/* zig-zag index of coefficient (vertical frequency v, horizontal u): the
 * diagonal d = u + v starts at d(d+1)/2 (or 64 - (15-d)(16-d)/2 past the
 * main anti-diagonal); odd diagonals run with increasing v, even ones with
 * decreasing v -- the transmission order of H.261 */
__host__ __device__ constexpr int zigzag_index(int v, int u)
{
    return (u + v < 8 ? ((u + v) * (u + v + 1)) >> 1 : 64 - (((15 - u - v) * (16 - u - v)) >> 1)) +
           (((u + v) & 1) ? v - (u + v < 8 ? 0 : u + v - 7) : (u + v < 8 ? u + v : 7) - v);
}

/* the coder's tables (the codes are the standard's, ITU-T H.261 Table 5, the
 * same values the reference's src/h261_tables.c holds), in device memory so
 * that a CTA loads them with one coalesced access a thread; lanes look them
 * up at different places, which constant memory would serve one by one */
struct alignas(16) VlcTables {
    /* TCOEFF without the sign bit, run 0..26 x level 0..15 (level 0 unused):
     * length << 8 | code; 0 = send with the 20-bit escape */
    uint16_t tc[27][16];
    /* column-major index (u * 8 + v) of the k-th coefficient sent */
    uint8_t cm[64];
};
static_assert(sizeof(VlcTables) % 16 == 0 && alignof(VlcTables) >= 16, "loaded as 16-byte words");
static_assert(offsetof(VlcTables, cm) % 4 == 0, "read as 4-byte words");

#define VLC(code, len) (uint16_t)(((len) << 8) | (code))
constexpr VlcTables make_vlc_tables()
{
    VlcTables t = { {
    { 0, VLC(3, 2), VLC(4, 4), VLC(5, 5), VLC(6, 7), VLC(38, 8), VLC(33, 8), VLC(10, 10), VLC(29, 12),
      VLC(24, 12), VLC(19, 12), VLC(16, 12), VLC(26, 13), VLC(25, 13), VLC(24, 13), VLC(23, 13) },
    { 0, VLC(3, 3), VLC(6, 6), VLC(37, 8), VLC(12, 10), VLC(27, 12), VLC(22, 13), VLC(21, 13) },
    { 0, VLC(5, 4), VLC(4, 7), VLC(11, 10), VLC(20, 12), VLC(20, 13) },
    { 0, VLC(7, 5), VLC(36, 8), VLC(28, 12), VLC(19, 13) },
    { 0, VLC(6, 5), VLC(15, 10), VLC(18, 12) },
    { 0, VLC(7, 6), VLC(9, 10), VLC(18, 13) },
    { 0, VLC(5, 6), VLC(30, 12) },
    { 0, VLC(4, 6), VLC(21, 12) },
    { 0, VLC(7, 7), VLC(17, 12) },
    { 0, VLC(5, 7), VLC(17, 13) },
    { 0, VLC(39, 8), VLC(16, 13) },
    { 0, VLC(35, 8) }, { 0, VLC(34, 8) }, { 0, VLC(32, 8) }, { 0, VLC(14, 10) }, { 0, VLC(13, 10) },
    { 0, VLC(8, 10) }, { 0, VLC(31, 12) }, { 0, VLC(26, 12) }, { 0, VLC(25, 12) }, { 0, VLC(23, 12) },
    { 0, VLC(22, 12) }, { 0, VLC(31, 13) }, { 0, VLC(30, 13) }, { 0, VLC(29, 13) }, { 0, VLC(28, 13) },
    { 0, VLC(27, 13) },
}, {} };
    for (int v = 0; v < 8; v++)
        for (int u = 0; u < 8; u++)
            t.cm[zigzag_index(v, u)] = (uint8_t)(u * 8 + v);
    return t;
}
#undef VLC
static __device__ const VlcTables g_vlc_tables = make_vlc_tables();

/* by the threads of a CTA; the caller synchronises before the first lookup */
__device__ __forceinline__ void load_vlc_tables(VlcTables &t, int tid, int nthreads)
{
    for (int i = tid; i < (int)(sizeof(VlcTables) / 16); i += nthreads)
        reinterpret_cast<uint4 *>(&t)[i] = reinterpret_cast<const uint4 *>(&g_vlc_tables)[i];
}

/* a warp's working memory */
struct alignas(16) VlcScratch {
    uint32_t stage[VLC_MB_WORDS];   /* the MB's codes; zero between MBs       */
    uint32_t cm[96];                /* the MB's levels, six blocks of 64 bytes,
                                       column-major, an intra DC as uint8     */
    uint32_t level[96];             /* the same in transmission order         */
    uint32_t mask[6][2];            /* per block: its nonzero positions       */
};

/* OR a code of len <= 32 bits into MSB-first words at bit position pos of
 * a buffer of `words` words; a position outside it is not written and
 * counts as an error */
__device__ __forceinline__ void put_bits(uint32_t *w, int words, int pos, uint32_t code, int len, int &oob)
{
    if (len <= 0)
        return;
    if (pos < 0 || pos + len > words * 32) {
        oob = 1;
        return;
    }
    const int word = pos >> 5, end = (pos & 31) + len;
    if (end <= 32) {
        atomicOr(&w[word], code << (32 - end));
    } else {
        atomicOr(&w[word], code >> (end - 32));
        atomicOr(&w[word + 1], code << (64 - end));
    }
}

/* one bit per nonzero byte of a word */
__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t w)
{
    const uint32_t f = ((((w & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w) >> 7) & 0x01010101u;
    return (f * 0x10204080u) >> 28;
}

/* the k-th set bit (from 0) of a mask that has it */
__device__ __forceinline__ int select_bit(uint32_t lo, uint32_t hi, int k)
{
    int p = 0, c = __popc(lo);
    uint32_t m = lo;
    if (k >= c) {
        k -= c;
        p = 32;
        m = hi;
    }
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
        c = __popc(m & ((1u << h) - 1u));
        if (k >= c) {
            k -= c;
            p += h;
            m >>= h;
        }
    }
    return p;
}

/* The codes of an MB's coded blocks (bit b of `blocks`) from its levels in
 * sc.cm.  They go into sc.stage from bit 0 on; returns their bits (the same
 * on every lane).  Every lane of the warp calls it; the caller's warp has
 * synchronised after writing the levels.
 *
 * Blocks hold a few nonzero levels each, so a lane a code does in one round
 * of about a hundred instructions what a kernel of its own, with eight
 * positions a lane and four blocks at a time, took two rounds of 280 for. */
__device__ __forceinline__ int code_mb(uint32_t blocks, bool intra, const VlcTables &tab, VlcScratch &sc, int lane,
                                       int &oob)
{
    constexpr unsigned FULLMASK = 0xFFFFFFFFu;
    /* transmission order: the lane's positions 4j .. 4j + 3 of block
     * lane / 16 + 2 i, for i = 0, 1, 2 */
    {
        const int j = lane & 15, half = lane >> 4;
        const uint32_t c4 = *reinterpret_cast<const uint32_t *>(&tab.cm[4 * j]);
        const uint8_t *base = reinterpret_cast<const uint8_t *>(sc.cm) + 64 * half;
        const uint8_t *a0 = base + (c4 & 0xFFu), *a1 = base + ((c4 >> 8) & 0xFFu);
        const uint8_t *a2 = base + ((c4 >> 16) & 0xFFu), *a3 = base + (c4 >> 24);
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const int b = half + 2 * i;
            const uint32_t w = __byte_perm((uint32_t)a0[128 * i] | ((uint32_t)a1[128 * i] << 8),
                                           (uint32_t)a2[128 * i] | ((uint32_t)a3[128 * i] << 8), 0x5410);
            const uint32_t nz = ((blocks >> b) & 1u) ? nonzero_bytes(w) : 0u;
            const uint32_t next = __shfl_down_sync(FULLMASK, nz, 1);
            sc.level[16 * b + j] = w;
            if (!(lane & 1))
                reinterpret_cast<uint8_t *>(sc.mask[b])[j >> 1] = (uint8_t)(nz | (next << 4));
        }
    }
    __syncwarp();
    /* codes of block `lane` (its levels and EOB) and of the blocks up to it */
    int n = 0;
    if (lane < 6 && ((blocks >> lane) & 1u))
        n = __popc(sc.mask[lane][0]) + __popc(sc.mask[lane][1]) + 1;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const int t = __shfl_up_sync(FULLMASK, incl, o);
        if (lane >= o)
            incl += t;
    }
    int upto[6];
#pragma unroll
    for (int b = 0; b < 6; b++)
        upto[b] = __shfl_sync(FULLMASK, incl, b);
    int pos = 0;
    for (int t0 = 0; t0 < upto[5]; t0 += 32) {
        const int t = t0 + lane;
        uint32_t code = 0;
        int len = 0;
        if (t < upto[5]) {
            int b = 0, first = 0;
#pragma unroll
            for (int i = 0; i < 5; i++)
                if (t >= upto[i]) {
                    b = i + 1;
                    first = upto[i];
                }
            const uint32_t lo = sc.mask[b][0], hi = sc.mask[b][1];
            const int k = t - first;
            if (k == __popc(lo) + __popc(hi)) {
                code = 2u;              /* EOB */
                len = 2;
            } else {
                const int at = select_bit(lo, hi, k);
                const int v = reinterpret_cast<const int8_t *>(sc.level)[64 * b + at], a = v < 0 ? -v : v;
                if (at == 0 && intra) {
                    code = (uint32_t)v & 0xFFu;       /* the DC level as it is */
                    len = 8;
                } else if (at == 0 && a == 1) {
                    code = v < 0 ? 3u : 2u;           /* first inter coefficient +-1 */
                    len = 2;
                } else {
                    /* zeros since the nonzero position before */
                    const uint32_t bh = at >= 32 ? hi & ((1u << (at - 32)) - 1u) : 0u;
                    const uint32_t bl = at >= 32 ? lo : lo & ((1u << at) - 1u);
                    const int prev = bh ? 63 - __clz((int)bh) : 31 - __clz((int)bl);
                    const int run = at - prev - 1;
                    const uint16_t e = (run <= 26 && a <= 15) ? tab.tc[run][a] : (uint16_t)0;
                    if (e) {
                        code = ((uint32_t)(e & 0xFF) << 1) | (v < 0 ? 1u : 0u);
                        len = (e >> 8) + 1;
                    } else {
                        /* escape 0000 01, 6-bit run, 8-bit level */
                        code = (1u << 14) | ((uint32_t)run << 8) | ((uint32_t)v & 0xFFu);
                        len = 20;
                    }
                }
            }
        }
        int end = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(FULLMASK, end, o);
            if (lane >= o)
                end += x;
        }
        put_bits(sc.stage, VLC_MB_WORDS, pos + end - len, code, len, oob);
        pos += __shfl_sync(FULLMASK, end, 31);
    }
    __syncwarp();   /* the codes are in place */
    return pos;
}

/* after code_mb: the MB's string from the staging words into dst (the
 * MB's VLC_MB_WORDS words), the staging words cleared for the next MB;
 * returns the string's bits, or -1 if a code fell outside the words (which
 * makes the layout refuse the picture).  Every lane calls it. */
__device__ __forceinline__ int store_mb_string(uint32_t *stage, uint32_t *dst, int pos, int oob, int lane)
{
    oob = __any_sync(0xFFFFFFFFu, oob);
    const int nw = min((pos + 31) >> 5, VLC_MB_WORDS);
    for (int i = lane; i < nw; i += 32) {
        dst[i] = stage[i];
        stage[i] = 0u;
    }
    __syncwarp();
    return oob ? -1 : pos;
}

} // namespace h261b
