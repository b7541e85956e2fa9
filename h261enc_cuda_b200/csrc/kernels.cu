/*
 * kernels.cu -- the sm_100a encode core: one warp per macroblock.
 *
 * A launch covers a flat list of (session, MB) work items, one frame-step
 * of any number of sessions of mixed size.  The grid is one wave of
 * resident CTAs; each warp owns a contiguous run of work items (consecutive
 * MBs of mostly one session) and, for each MB, runs the phases the launch
 * asks for while the next MB's inputs are already on their way:
 *
 *   stage   16-byte cp.async copies of the 46x48 luma search window (rows
 *           mb_y-15 .. +30, columns mb_x-16 .. +31) and of the source MB
 *           into one of two per-warp shared-memory buffers, issued one MB
 *           ahead.
 *   ME      - reference mode: SAD over the 11x11 coarse grid of
 *             megpu_kernels.cuh:27-166, then the 7x7 refinement of :307-446
 *             around its winner; full mode: every vector of [-15,15]^2;
 *           four packed pixels per step (vabsdiff4.add on funnel-shifted
 *           words), each window row aligned once for a column of vectors.
 *           The reference picks a winner with a 2-D tree of
 *           strict '<' comparisons in the order self, right, below, diagonal
 *           (:95-154); that tree returns the minimum cost and, among equal
 *           costs, the cell with the smallest Z-order index (x bits on even
 *           positions).  Each lane therefore folds (cost << 10 | zorder) into
 *           one 32-bit key and a single redux.sync min picks the same winner.
 *           Then the three 16x16 SATD costs of :617-987 (inter, inter with
 *           the 3x3 interior filter, intra), each a small matrix product.
 *   MD      the decision of h261_moded.c:53-95.
 *   ENCDEC  per 8x8 block, one lane per row then per column: prediction
 *           with the H.261 loop filter, the reference's float/double AAN
 *           FDCT (mbgpu_kernels.cuh:337-442) with every rounding step
 *           spelled out by intrinsics, denoise against the session's
 *           offsets (:506-636), quantisation (:644-724), dequantisation
 *           (:731-815), the AAN IDCT (:827-931) and reconstruction
 *           (:988-1277) into the session's output picture.
 *
 * Denoise statistics are summed per warp over its run of MBs of one session
 * and published when the session changes; the warp whose publication
 * completes a session's frame (a ticket counting MBs) turns the statistics
 * into the next frame's offsets (:478-503).  No warp waits on another, but
 * for the teams of four warps per macroblock of small launches
 * (team_kernel), which share each step's work and meet at CTA barriers.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "h261b_device.h"
#include "parts.h"
#include "vlc_coder.h"

namespace {

using namespace h261b;


constexpr int WIN_ROWS = 46;        /* rows mb_y-15 .. mb_y+30; columns mb_x-16 .. mb_x+31 */
/* A warp's two buffers (this MB, next MB) share 46 rows of 36 words.
 * Buffer k starts at word 16k of the array and holds, relative to that:
 *   words 0-11 of row r      window row r (12 words, 48 pixels)
 *   words 12-15 of row i     source luma row i (i < 16)
 *   words 12-13 of row 16+j  source chroma row j (Cb j < 8, Cr j >= 8)
 * so one base pointer addresses all of an MB's inputs.  Rows are 144 B, so
 * every row and source row is 16-byte aligned for the 16-byte copies, and
 * with a 36-word pitch the search's lanes, which read rows up to three
 * apart at up to 13 word columns, meet no bank twice. */
constexpr int WIN_PITCH_W = 36;
constexpr int SRC_COL_W = 12;
constexpr uint32_t FULL = 0xffffffffu;
/* transpose buffer: rows of 12 words, blocks of 104, so that a row moves as
 * two 16-byte accesses and neither the rows of a block (banks 12 r) nor the
 * columns of the four blocks (banks 8 slot + c) conflict */
constexpr int TB_ROW = 12, TB_BLOCK = 104;

struct __align__(16) WarpSmem {
    uint32_t buf[WIN_ROWS * WIN_PITCH_W]; /* both buffers, interleaved      */
    uint64_t bar[2];                      /* per buffer: the barrier its bulk
                                             row copies complete on (bulk
                                             staging only)                   */
    float t[4][TB_BLOCK];                 /* transpose buffer               */
    VlcScratch vlc;                       /* the MB's levels and codes      */
};

/* one MB's staged inputs: buffer k of the warp's shared memory */
struct StageBuf {
    const uint32_t *p;
    /* window row r from word c */
    __device__ __forceinline__ const uint32_t *win(int r, int c) const { return p + r * WIN_PITCH_W + c; }
    /* source luma row i from word c */
    __device__ __forceinline__ const uint32_t *cur(int i, int c) const { return p + i * WIN_PITCH_W + SRC_COL_W + c; }
    /* source chroma row j (Cb rows 0-7, Cr rows 8-15), two words */
    __device__ __forceinline__ const uint32_t *curc(int j) const { return p + (16 + j) * WIN_PITCH_W + SRC_COL_W; }
};

__device__ __forceinline__ StageBuf stage_view(const uint32_t *wbuf, int k) { return StageBuf{ wbuf + 16 * k }; }

/* shared memory of one warp: both staging buffers, plus the transpose
 * buffer for kernels that encode (the search-only kernel has none), plus the
 * coder's memory for those that also code; theirs ends with the coder's
 * tables, one per CTA */
constexpr size_t kSearchWarpBytes = sizeof(uint32_t) * WIN_ROWS * WIN_PITCH_W + 2 * sizeof(uint64_t);
constexpr size_t kEncodeWarpBytes = offsetof(WarpSmem, vlc);
static_assert(kEncodeWarpBytes % 16 == 0 && sizeof(WarpSmem) % 16 == 0, "warp shared layout");
static_assert(alignof(WarpSmem) >= alignof(VlcTables), "the tables follow the warps' shared memory");
static_assert(kSearchWarpBytes % 16 == 0 && offsetof(WarpSmem, t) == kSearchWarpBytes, "warp shared layout");

/* the coarse grid's offsets { -14, -11, -8, -5, -2, 0, 2, 5, 8, 11, 14 }
 * (megpu_kernels.cuh:27-166), by arithmetic: lanes index it at 11 places
 * at once, which a constant-memory table would serve one address at a time */
__device__ __forceinline__ int stage1_offset(int t)
{
    return 3 * t - 14 - (t == 5 ? 1 : 0) - (t > 5 ? 2 : 0);
}
/* float tables initialised from double literals like the reference's */
__constant__ float c_fwd_post[8] = { 1.0, 0.720960, 0.765367, 0.850430, 1.0, 1.272759, 1.847759, 3.624510 };
__constant__ float c_inv_pre[8] = { 1.0, 1.387040, 1.306563, 1.175876, 1.0, 0.785695, 0.541196, 0.275899 };
/* f_inv_quant = 1.0 / ( float ) ( i_quant * 2 ) (mbgpu_kernels.cuh:685), an
 * IEEE double rounded to float; by QUANT, 0 unused */
#define INV_QUANT(q) (float)(1.0 / (double)(float)((q) * 2))
#define INV_QUANT4(q) INV_QUANT(q), INV_QUANT(q + 1), INV_QUANT(q + 2), INV_QUANT(q + 3)
__constant__ float c_inv_quant[32] = { 0.0f,           INV_QUANT(1),   INV_QUANT(2),   INV_QUANT(3),  INV_QUANT4(4),
                                       INV_QUANT4(8),  INV_QUANT4(12), INV_QUANT4(16), INV_QUANT4(20),
                                       INV_QUANT4(24), INV_QUANT4(28) };

/* ------------------------------------------------ debug bounds checks
 *
 * Built with -DH261B_DEBUG_CHECKS (make check: lib/libh261b_check.so),
 * every global access whose address depends on a vector, a work item or a
 * picture size, and the shared-memory window reads of the motion
 * compensation, first test their index: a failing test is counted and its
 * site and index recorded (h261b_debug_check_status), and the access is
 * skipped or its index clamped into the buffer.  In the normal build the
 * checks compile to nothing. */
enum CheckSite {
    CHK_WORK_ITEM = 1,      /* MB index of a work item inside its picture     */
    CHK_STAGE_WINDOW = 2,   /* a staged window chunk inside the reference     */
    CHK_STAGE_SOURCE = 3,   /* a staged source row inside the picture         */
    CHK_MC_WINDOW = 4,      /* luma prediction rows inside the staged window  */
    CHK_MC_CHROMA = 5,      /* chroma prediction rows inside the reference    */
    CHK_RECON = 6,          /* reconstruction row inside the output picture   */
};

#ifdef H261B_DEBUG_CHECKS
__device__ unsigned long long g_check_count;
__device__ int g_check_first[2];

__device__ __noinline__ void check_fail(int site, int value)
{
    if (atomicAdd(&g_check_count, 1ull) == 0) {
        g_check_first[0] = site;
        g_check_first[1] = value;
    }
}
#define H261B_CHECK(cond, site, value) ((cond) ? true : (check_fail((site), (int)(value)), false))
#else
#define H261B_CHECK(cond, site, value) true
#endif

/* ------------------------------------------------------------ helpers */

__device__ __forceinline__ uint32_t spread8(uint32_t v)
{
    v &= 0xFFu;
    v = (v | (v << 4)) & 0x0F0Fu;
    v = (v | (v << 2)) & 0x3333u;
    v = (v | (v << 1)) & 0x5555u;
    return v;
}

/* spread8 of a value below 16 */
__device__ __forceinline__ constexpr uint32_t spread4(uint32_t v)
{
    v = (v | (v << 2)) & 0x33u;
    return (v | (v << 1)) & 0x55u;
}

__device__ __forceinline__ uint32_t compact8(uint32_t v)
{
    v &= 0x5555u;
    v = (v | (v >> 1)) & 0x3333u;
    v = (v | (v >> 2)) & 0x0F0Fu;
    v = (v | (v >> 4)) & 0x00FFu;
    return v;
}

__device__ __forceinline__ uint32_t zorder(uint32_t x, uint32_t y) { return spread8(x) | (spread8(y) << 1); }

/* eight window bytes of row `row` from byte column `col` (any alignment):
 * three word loads, two funnel shifts; 0 <= col <= 43 keeps the loads
 * inside the row (bytes past column 47, which are the source words or the
 * other buffer, are never used) */
__device__ __forceinline__ uint2 win8(const StageBuf s, int row, int col)
{
    const uint32_t *p = s.win(row, col >> 2);
    const uint32_t sh = (uint32_t)(col & 3) * 8u;
    const uint32_t a = p[0], b = p[1], c = p[2];
    return make_uint2(__funnelshift_r(a, b, sh), __funnelshift_r(b, c, sh));
}

/* asynchronous global -> shared copies; a 16-byte window chunk outside the
 * picture is not read (src-size 0) and its bytes are zero-filled.  Window
 * chunks are cached in L1 too: neighbouring MBs of a warp share two thirds
 * of them. */
__device__ __forceinline__ void cp_async8(void *dst, const void *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16z(void *dst, const void *src, bool valid)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

/* bulk copies (the async proxy) completed on a shared-memory barrier: the
 * alternative staging of the search window, one copy per window row.  The
 * source is always this GPU's own memory, and no copy is multicast. */
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_inval(uint64_t *bar)
{
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_addr(bar)) : "memory");
}
/* the one arrival of a phase, announcing the bytes its copies will bring */
__device__ __forceinline__ void mbar_arrive_expect(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 " selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done)
                 : "r"(smem_addr(bar)), "r"(parity)
                 : "memory");
    return done != 0;
}
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
/* this thread's earlier generic accesses of shared memory before its later
 * async-proxy writes (a buffer is refilled after the warp read it) */
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

/* bulk staging waits that gave up (bounded, so that nothing can hang);
 * reported by h261b_stage_status, always 0 in a correct run */
__device__ unsigned int g_stage_timeouts;

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

/* wait for a buffer's phase for at most 100 ms of the global timer (a row
 * copy takes about a microsecond): a copy that never completes is counted,
 * not waited for forever, and the warp stops waiting from then on */
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, int lane)
{
    if (mbar_try_wait(bar, parity))
        return true;
    const uint64_t t0 = global_ns();
    for (;;) {
        for (int i = 0; i < 64; i++)
            if (mbar_try_wait(bar, parity))
                return true;
        if (global_ns() - t0 > 100000000ull)
            break;
    }
    if (lane == 0)
        atomicAdd(&g_stage_timeouts, 1u);
    return false;
}

__device__ __forceinline__ uint32_t sad16(uint4 c, const uint32_t w[4], uint32_t acc)
{
    return sad4(c.w, w[3], sad4(c.z, w[2], sad4(c.y, w[1], sad4(c.x, w[0], acc))));
}

/* sixteen window pixels of a row from word q on, `sh` bits into it */
__device__ __forceinline__ void align16(const uint32_t *q, uint32_t sh, uint32_t w[4])
{
    const uint32_t x0 = q[0], x1 = q[1], x2 = q[2], x3 = q[3], x4 = q[4];
    w[0] = __funnelshift_r(x0, x1, sh);
    w[1] = __funnelshift_r(x1, x2, sh);
    w[2] = __funnelshift_r(x2, x3, sh);
    w[3] = __funnelshift_r(x3, x4, sh);
}

__device__ __forceinline__ uint4 cur_row(const StageBuf s, int r) { return *reinterpret_cast<const uint4 *>(s.cur(r, 0)); }

/* window rows R0 .. R0 + NR - 1 of a column of five vectors three rows
 * apart (row R of the column serves vector k with source row R - 3k), for
 * the vectors K0 .. K1 that those rows reach */
template <int R0, int NR, int K0, int K1>
__device__ __forceinline__ void grid_rows(const StageBuf s, const uint32_t *p, uint32_t sh, uint32_t sad[5])
{
#pragma unroll
    for (int i = 0; i < NR; i++) {
        uint32_t w[4];
        align16(p + (R0 + i) * WIN_PITCH_W, sh, w);
#pragma unroll
        for (int k = K0; k <= K1; k++)
            sad[k] = sad16(cur_row(s, R0 + i - 3 * k), w, sad[k]);
    }
}

/* the 11x11 coarse grid; returns the smallest (cost << 10 | Z-order) key of
 * the vectors inside the limits.
 *
 * The search's time is its ALU-pipe time: each 4-pixel difference and each
 * funnel shift that aligns a window word takes one slot.  So a lane takes a
 * column of vectors and aligns each window row once for all of them: lanes
 * 0-10 the rows -14, -11, -8, -5, -2 of column `lane`, lanes 11-21 the rows
 * 2, 5, 8, 11, 14, and lanes 22-31 row 0 of the ten columns other than x = 0
 * (the first vector of the same instruction stream; what it computes for
 * the other four is not used).  The zero vector, which needs no alignment,
 * is summed by all lanes, half a row each.  28 window rows instead of 64
 * are loaded and aligned a lane: 432 ALU slots and 690 instructions against
 * 512 and 1,150 for two vectors a lane at a time (with the refinement below,
 * 4,923 -> 3,808 instructions a macroblock and 113.9 -> 105.6 us for the
 * encode launch of 13,464 macroblocks; unrolled, the rows run 3 % faster
 * there than as loops).  Every row and word read is staged: rows 1 .. 44,
 * words 0 .. 11. */
__device__ __forceinline__ uint32_t grid_search(const StageBuf s, int lminx, int lmaxx, int lminy, int lmaxy, int lane)
{
    const int g = lane >= 22 ? 2 : lane >= 11 ? 1 : 0;
    const int c = lane - 11 * g, tx = g == 2 && c >= 5 ? c + 1 : c;
    const int x = stage1_offset(tx), b = 16 + x;
    const int y0 = g == 0 ? -14 : g == 1 ? 2 : 0;
    const uint32_t *p = s.win(15 + y0, b >> 2);
    const uint32_t sh = (uint32_t)(b & 3) * 8u;
    uint32_t sad[5] = { 0u, 0u, 0u, 0u, 0u };
    grid_rows<0, 3, 0, 0>(s, p, sh, sad);
    grid_rows<3, 3, 0, 1>(s, p, sh, sad);
    grid_rows<6, 3, 0, 2>(s, p, sh, sad);
    grid_rows<9, 3, 0, 3>(s, p, sh, sad);
    grid_rows<12, 4, 0, 4>(s, p, sh, sad);
    grid_rows<16, 3, 1, 4>(s, p, sh, sad);
    grid_rows<19, 3, 2, 4>(s, p, sh, sad);
    grid_rows<22, 3, 3, 4>(s, p, sh, sad);
    grid_rows<25, 3, 4, 4>(s, p, sh, sad);

    /* the zero vector: words 2h, 2h + 1 of row r */
    const int r = lane >> 1, h = lane & 1;
    const uint2 wz = *reinterpret_cast<const uint2 *>(s.win(15 + r, 4 + 2 * h));
    const uint2 cz = *reinterpret_cast<const uint2 *>(s.cur(r, 2 * h));
    const uint32_t zero = __reduce_add_sync(FULL, sad4(cz.y, wz.y, sad4(cz.x, wz.x, 0u)));
    uint32_t best = zero << 10 | zorder(5, 5);

    /* Z-order bits of the rows: 0..4, 6..10 (lanes 11-21), 5 (lanes 22-31) */
    const uint32_t zx = spread4((uint32_t)tx);
    const bool okx = x >= lminx && x <= lmaxx;
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const int y = y0 + 3 * k;
        const uint32_t zy = k == 0 ? (g == 0 ? spread4(0) : g == 1 ? spread4(6) : spread4(5))
                                   : (g == 0 ? spread4(k) : spread4(6 + k));
        const bool ok = okx && y >= lminy && y <= lmaxy && (k == 0 || g != 2);
        best = min(best, ok ? (sad[k] << 10) | zx | (zy << 1) : FULL);
    }
    return __reduce_min_sync(FULL, best);
}

/* the 7x7 refinement around (v1x, v1y); returns the smallest key, whose
 * Z-order counts from (v1x - 3, v1y - 3).
 *
 * Lane 4 tx + q sums rows 4q .. 4q + 3 of the block for the seven vectors of
 * column tx: ten window rows aligned for 28 rows of differences, the four
 * source rows in registers, then a reduce-scatter of the sums, two to a
 * word, over the four lanes of a column (206 + 20 instructions, 152 ALU
 * slots; two whole vectors a lane took 313 and 196).  A column that would
 * reach past +-15 starts at the nearest one inside, and each vector takes
 * its sum from there. */
__device__ __forceinline__ uint32_t refine_search(const StageBuf s, int v1x, int v1y, int lminx, int lmaxx, int lminy,
                                                  int lmaxy, int lane)
{
    const int tx = lane >> 2, q = lane & 3;
    const int x = v1x + tx - 3, ylo = v1y - 3;
    const int base = min(max(ylo, -15), 9);
    const int b = 16 + min(max(x, -15), 15);
    const uint32_t *p = s.win(15 + base + 4 * q, b >> 2);
    const uint32_t sh = (uint32_t)(b & 3) * 8u;
    uint4 c[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
        c[i] = cur_row(s, 4 * q + i);
    uint32_t sad[8] = { 0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u };
#pragma unroll
    for (int R = 0; R < 10; R++) {
        uint32_t w[4];
        align16(p + R * WIN_PITCH_W, sh, w);
#pragma unroll
        for (int k = 0; k < 7; k++)
            if (R - k >= 0 && R - k < 4)
                sad[k] = sad16(c[R - k], w, sad[k]);
    }
    /* sums of the block are at most 65,280: two fit a word */
    uint32_t pk[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
        pk[i] = sad[2 * i] + (sad[2 * i + 1] << 16);
    const bool up = (q & 2) != 0, odd = (q & 1) != 0;
    uint32_t a0 = up ? pk[2] : pk[0], a1 = up ? pk[3] : pk[1];
    a0 += __shfl_xor_sync(FULL, up ? pk[0] : pk[2], 2);
    a1 += __shfl_xor_sync(FULL, up ? pk[1] : pk[3], 2);
    const uint32_t v = (odd ? a1 : a0) + __shfl_xor_sync(FULL, odd ? a0 : a1, 1);
    /* this lane's pair of the column: vectors base + 2q and base + 2q + 1 */
    const uint32_t zx = spread4((uint32_t)tx);
    const bool okx = tx < 7 && x >= lminx && x <= lmaxx;
    uint32_t best = FULL;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int i = 2 * q + k, y = base + i, ty = y - ylo;
        const bool ok = okx && i < 7 && ty >= 0 && ty < 7 && y >= lminy && y <= lmaxy;
        const uint32_t cost = k ? v >> 16 : v & 0xFFFFu;
        best = min(best, ok ? (cost << 10) | zx | (spread4((uint32_t)ty) << 1) : FULL);
    }
    return __reduce_min_sync(FULL, best);
}

/* window rows W0 .. W1 - 1 of the exhaustive search, source rows R0 .. R1 - 1 */
template <int W0, int W1, int R0, int R1>
__device__ __forceinline__ void full_rows(const StageBuf s, const uint32_t *p, uint32_t sh, int lminy, int lmaxy,
                                          uint32_t acc[16], uint32_t &best)
{
#pragma unroll 1
    for (int W = W0; W < W1; W++) {
        uint32_t w[4];
        align16(p + W * WIN_PITCH_W, sh, w);
#pragma unroll
        for (int r = R1 - 1; r >= R0; r--)
            acc[r] = sad16(cur_row(s, r), w, r ? acc[r - 1] : 0u);
        if (R1 == 16 && W - 30 >= lminy && W - 30 <= lmaxy)
            best = min(best, (acc[15] << 10) | (spread8((uint32_t)(W - 15)) << 1));
    }
}

/* every vector of [-15, 15]^2: lane tx takes column tx - 15 (lane 31 repeats
 * column 15) and aligns each of the 46 window rows once for the sixteen
 * vectors that it can serve.  acc[r] holds the sum over source rows 0 .. r of
 * the vector whose row r is the window row at hand, so that one row of
 * differences moves each sum one place on, and acc[15] is complete: 2,068
 * differences and 184 alignments a lane, where columns of four vectors took
 * 2,048 and 608, and half the instructions (64 QCIF pictures: 111.2 -> 95.5
 * us for the encode launch; the first and last rows two at a time instead of
 * four, 71.1 -> 69.0 us later).  Returns the smallest key (Z-order from
 * (-15, -15)). */
__device__ __forceinline__ uint32_t full_search(const StageBuf s, int lminx, int lmaxx, int lminy, int lmaxy, int lane)
{
    const int tx = min(lane, 30), x = tx - 15, b = 16 + x;
    const uint32_t *p = s.win(0, b >> 2);
    const uint32_t sh = (uint32_t)(b & 3) * 8u;
    uint32_t acc[16], best = FULL;
#pragma unroll
    for (int r = 0; r < 16; r++)
        acc[r] = 0u;
    /* vectors -15 .. 15 start at window rows 0 .. 30: the first rows serve
     * only the first source rows, the last rows only the last */
    full_rows<0, 2, 0, 2>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<2, 4, 0, 4>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<4, 6, 0, 6>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<6, 8, 0, 8>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<8, 10, 0, 10>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<10, 12, 0, 12>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<12, 33, 0, 16>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<33, 35, 3, 16>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<35, 37, 5, 16>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<37, 39, 7, 16>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<39, 41, 9, 16>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<41, 43, 11, 16>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<43, 45, 13, 16>(s, p, sh, lminy, lmaxy, acc, best);
    full_rows<45, 46, 15, 16>(s, p, sh, lminy, lmaxy, acc, best);
    best = x >= lminx && x <= lmaxx && best != FULL ? best | spread8((uint32_t)tx) : FULL;
    return __reduce_min_sync(FULL, best);
}

/* ------------------------------------------------ SATD (megpu_kernels.cuh:467-500)
 *
 * The 4x4 Hadamard of a macroblock's sixteen sub-blocks is one matrix
 * product, [16 sub-blocks x 16 pixels] x [16 pixels x 16 signs], and its
 * terms are small integers: pixel differences are exact in half precision
 * (255 at most), the signs are +-1 and the sums (4,080 at most) exact in
 * float, so two mma.sync m16n8k16 give the reference's integers.  The A
 * fragment is one macroblock of pixels: lane 4g + t holds row t of sub-block
 * g (sub-blocks 0-7, the upper half) and of sub-block g + 8, pixels 0 and 2
 * of the row in one register, 1 and 3 in another (columns 2t, 2t + 1 and
 * 2t + 8, 2t + 9 of A).
 *
 * tcgen05.mma is not used here: a product this small would wait longer for
 * its operands to reach shared memory and its result to leave TMEM than the
 * two mma.sync take (8.6 cycles each on an SM quarter).  Against one 4x4
 * transform a lane in integers the costs take some 150 instructions a
 * macroblock instead of 560: 105.6 -> 98.9 us for the encode launch of
 * 13,464 macroblocks of mixed streams, 756 -> 716 us for 1024 QCIF streams. */

/* D = A x B + C, half inputs, float sums */
__device__ __forceinline__ void mma_16n8k16(float d[4], const uint32_t a[4], uint32_t b0, uint32_t b1, float c02)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%10,%11};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c02), "f"(0.0f));
}

/* the SATD of a macroblock from its A fragment; `bias` is what every pixel
 * of it has on top (it reaches only the sums with all signs +, the first
 * column of the product) */
__device__ __forceinline__ int32_t satd16x16(const uint32_t a[4], float bias, int lane)
{
    const int g = lane >> 2, t = lane & 3;
    /* sign of pixel (x, y) in the transform (u, v): the parity of u & x and
     * v & y; column g has u = g & 3 and v = g >> 2, then v + 2 */
    const uint32_t neg = 0x80008000u;
    const uint32_t b0 = (0x3C003C00u ^ ((g & 2) ? 0x80000000u : 0u)) ^ (((g >> 2) & t & 1) ? neg : 0u);
    const uint32_t b1 = b0 ^ ((g & 1) ? neg : 0u), flip = (t & 2) ? neg : 0u;
    float d[8];
    mma_16n8k16(d, a, b0, b1, t == 0 ? -16.0f * bias : 0.0f);
    mma_16n8k16(d + 4, a, b0 ^ flip, b1 ^ flip, 0.0f);
    /* 2^23 + the lane's sum (32,640 at most): the integer is the float's low bits */
    float sum = 8388608.0f;
#pragma unroll
    for (int i = 0; i < 8; i++)
        sum = __fadd_rn(sum, fabsf(d[i]));
    /* the 32 exponents add up to 32 * 0x4B000000 = 0x60000000 (mod 2^32) */
    return (int32_t)(__reduce_add_sync(FULL, __float_as_uint(sum)) - 0x60000000u);
}

/* four pixels as halves 1024 + x: pixels 0 and 2, pixels 1 and 3 */
__device__ __forceinline__ void half_pixels(uint32_t w, uint32_t &even, uint32_t &odd)
{
    even = __byte_perm(w, 0x64646464u, 0x4240);
    odd = __byte_perm(w, 0x64646464u, 0x4341);
}

__device__ __forceinline__ uint32_t half_sub(uint32_t a, uint32_t b)
{
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

/* the source MB as an A fragment of halves 1024 + x */
__device__ __forceinline__ void source_halves(const StageBuf s, int lane, uint32_t c[4])
{
    const int g = lane >> 2, row = (g >> 2) * 4 + (lane & 3);
    half_pixels(*s.cur(row, g & 3), c[0], c[2]);
    half_pixels(*s.cur(row + 8, g & 3), c[1], c[3]);
}

__device__ __forceinline__ int32_t intra_cost(const StageBuf s, int lane)
{
    uint32_t c[4];
    source_halves(s, lane, c);
    return satd16x16(c, 1024.0f, lane);
}

/* the 16x16 SATD costs at vector (vx, vy): inter, and inter with the 3x3
 * interior filter (megpu_kernels.cuh:617-987), or one of them */
template <bool PLAIN, bool FILTERED>
__device__ __forceinline__ void inter_costs(const StageBuf s, int vx, int vy, int lane, int32_t &plain,
                                            int32_t &filtered)
{
    const int g = lane >> 2, t = lane & 3, sx = g & 3, row = (g >> 2) * 4 + t;
    uint32_t c[4], p[4], f[4];
    source_halves(s, lane, c);
    /* horizontal [1 2 1] sums of the lane's two rows of four pixels, 16 bits
     * each, from the eight bytes that start one pixel to their left; the
     * rows above and below belong to neighbouring lanes (t - 1, t + 1, or
     * the sub-block four on) */
    const int col = 15 + vx + 4 * sx;
    const uint32_t *q = s.win(15 + vy + row, col >> 2);
    const uint32_t sh = (uint32_t)(col & 3) * 8u;
    const int up = t ? lane - 1 : lane - 13, down = t < 3 ? lane + 1 : lane + 13;
    /* the filter applies to the interior (1..6) of each 8x8 block */
    const int ly = (g & 4) + t;
    const uint32_t rows = ly >= 1 && ly <= 6 ? 0x00FF00FFu : 0u;
    const uint32_t even_in = rows & ((sx & 1) ? 0x00FF00FFu : 0x00FF0000u);
    const uint32_t odd_in = rows & ((sx & 1) ? 0x000000FFu : 0x00FF00FFu);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint32_t w0 = q[8 * h * WIN_PITCH_W], w1 = q[8 * h * WIN_PITCH_W + 1], w2 = q[8 * h * WIN_PITCH_W + 2];
        const uint32_t lo = __funnelshift_r(w0, w1, sh), hi = __funnelshift_r(w1, w2, sh);
        const uint32_t e = __byte_perm(lo, 0u, 0x4240), o = __byte_perm(lo, 0u, 0x4341);   /* bytes 0, 2; 1, 3 */
        const uint32_t m = __byte_perm(e, hi, 0x1412), n = __byte_perm(o, hi, 0x1512);     /* bytes 2, 4; 3, 5 */
        const uint32_t he = e + 2u * o + m, ho = o + 2u * m + n;
        const uint32_t ve = __shfl_sync(FULL, he, up) + 2u * he + __shfl_sync(FULL, he, down) + 0x00080008u;
        const uint32_t vo = __shfl_sync(FULL, ho, up) + 2u * ho + __shfl_sync(FULL, ho, down) + 0x00080008u;
        p[h] = o | 0x64006400u;
        p[h + 2] = m | 0x64006400u;
        f[h] = (p[h] & ~even_in) | ((ve >> 4) & even_in);
        f[h + 2] = (p[h + 2] & ~odd_in) | ((vo >> 4) & odd_in);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        p[i] = half_sub(c[i], p[i]);
        f[i] = half_sub(c[i], f[i]);
    }
    if (PLAIN)
        plain = satd16x16(p, 0.0f, lane);
    if (FILTERED)
        filtered = satd16x16(f, 0.0f, lane);
}

/* ---------------------------------------------- exact float/double math */

/* `float *= double`: double product rounded to float */
__device__ __forceinline__ float dmulf(float x, double k)
{
    return __double2float_rn(__dmul_rn((double)x, k));
}

/* `float *= k` for a double constant k = hi + lo, in float: the fused
 * multiply-add rounds x * hi plus a term accurate to 2^-49 of the product,
 * which is the double product rounded to float for every float x whose
 * product is a normal number (tests/rounding_check_mul.c checks every
 * mantissa): with k = 0.382683 and 1.84776 for all of them, with k =
 * 0.707107 for all but three, of more than 18 significant bits each, so
 * there for integers.  Two instructions at full rate (1.1 cycles a warp on
 * an SM quarter each) where the conversions to and from double take 8 each. */
__device__ __forceinline__ float mul_hilo(float x, double k)
{
    const float hi = (float)k, lo = (float)(k - (double)hi);
    return __fmaf_rn(x, hi, __fmul_rn(x, lo));
}

/* `float = float * double + float`: fused (one rounding) or not */
template <int FMAD>
__device__ __forceinline__ float dmadf(float a, double k, float c)
{
    if (FMAD)
        return __double2float_rn(__fma_rn((double)a, k, (double)c));
    return __double2float_rn(__dadd_rn(__dmul_rn((double)a, k), (double)c));
}

/* the AAN forward butterfly shared by both passes (mbgpu_kernels.cuh:359-388);
 * INTS: its inputs are integers (the first pass) */
template <int FMAD, bool INTS>
__device__ __forceinline__ void fdct_butterfly(float tmp0, float tmp1, float tmp2, float tmp3, float tmp4,
                                               float tmp5, float tmp6, float tmp7, float o[8])
{
    const float tmp10 = tmp0 + tmp3, tmp13 = tmp0 - tmp3, tmp11 = tmp1 + tmp2, tmp12 = tmp1 - tmp2;
    o[0] = tmp10 + tmp11;
    o[4] = tmp10 - tmp11;
    const float z1 = INTS ? mul_hilo(tmp12 + tmp13, 0.707107) : dmulf(tmp12 + tmp13, 0.707107);
    o[2] = tmp13 + z1;
    o[6] = tmp13 - z1;
    tmp4 = tmp4 + tmp5;
    tmp5 = tmp5 + tmp6;
    tmp6 = tmp6 + tmp7;
    const float z5 = mul_hilo(tmp4 - tmp6, 0.382683);
    const float z2 = dmadf<FMAD>(tmp4, 0.541196, z5);
    const float z4 = dmadf<FMAD>(tmp6, 1.306563, z5);
    const float z3 = INTS ? mul_hilo(tmp5, 0.707107) : dmulf(tmp5, 0.707107);
    const float z11 = tmp7 + z3, z13 = tmp7 - z3;
    o[5] = z13 + z2;
    o[3] = z13 - z2;
    o[1] = z11 + z4;
    o[7] = z11 - z4;
}

/* 1.5 * 2^23: a float of that magnitude has a unit of one, so a sum with it
 * rounds to an integer, the way the addition rounds, and the integer is in
 * its low bits (two's complement).  An addition runs at full rate; the
 * conversions between float and integer take 8 cycles a warp. */
constexpr float kBias = 12582912.0f;
/* kBias + floor(x), |x| < 2^22 */
__device__ __forceinline__ float floor_biased(float x) { return __fadd_rd(x, kBias); }

/* floorf( cs * post * v + 0.49999 ) as the reference writes it
 * (mbgpu_kernels.cuh:413-437): a float product, the sum with the double
 * literal rounded to double, then to float, then the floor.  For every
 * finite float p, floorf((float)((double)p + 0.49999)) equals
 * floorf(p + 0.49999f) with the float literal (the float nearest to
 * 0.49999) -- checked for all 2.5e9 floats of magnitude below 2^24 by
 * tests/rounding_check.c; above it both leave p unchanged -- so the sum is
 * taken in float and floored by a sum that rounds down: no conversion. */
__device__ __forceinline__ float fdct_round(float cs, float post, float v)
{
    const float prod = __fmul_rn(__fmul_rn(cs, post), v);
    return __fadd_rn(floor_biased(__fadd_rn(prod, 0.49999f)), -kBias);
}

/* the AAN inverse butterfly after its first level of adds (mbgpu_kernels.cuh
 * :851-887 for columns, :892-919 for rows); the caller forms the first level
 * (tmp12 = p2 - p6, tmp13 = p2 + p6, tmp10 = p0 + p4, tmp11 = p0 - p4,
 * z11 = p1 + p7, z12 = p1 - p7, z13 = p5 + p3, z10 = p5 - p3) */
template <int FMAD>
__device__ __forceinline__ void idct_rest(float tmp12, float tmp13, float tmp10, float tmp11, float z11,
                                          float z12, float z13, float z10, float o[8])
{
    tmp12 = dmulf(tmp12, 1.414214);
    tmp12 = tmp12 - tmp13;
    const float tmp0 = tmp10 + tmp13, tmp1 = tmp11 + tmp12, tmp2 = tmp11 - tmp12, tmp3 = tmp10 - tmp13;
    tmp13 = z11 + z13;
    tmp11 = dmulf(z11 - z13, 1.414214);
    const float z5 = mul_hilo(z12 + z10, 1.84776);
    tmp10 = dmadf<FMAD>(z12, 1.082392, -z5);
    tmp12 = dmadf<FMAD>(z10, -2.613126, z5);
    tmp12 = tmp12 - tmp13;
    tmp11 = tmp11 - tmp12;
    tmp10 = tmp10 + tmp11;
    o[0] = tmp0 + tmp13;
    o[1] = tmp1 + tmp12;
    o[2] = tmp2 + tmp11;
    o[3] = tmp3 - tmp10;
    o[4] = tmp3 + tmp10;
    o[5] = tmp2 - tmp11;
    o[6] = tmp1 - tmp12;
    o[7] = tmp0 - tmp13;
}

/* first level of the column pass on prescaled products t = P * cs: the
 * reference built with nvcc defaults fuses the left-hand product of each
 * add into one FFMA (its product rounds once, with the sum) */
template <int FMAD>
__device__ __forceinline__ float first_add(float Pa, float csa, float ta, float tb)
{
    return FMAD ? __fmaf_rn(Pa, csa, tb) : __fadd_rn(ta, tb);
}
template <int FMAD>
__device__ __forceinline__ float first_sub(float Pa, float csa, float ta, float tb)
{
    return FMAD ? __fmaf_rn(Pa, csa, -tb) : __fsub_rn(ta, tb);
}

/* floor( v + 0.49999 ) with v widened to double (mbgpu_kernels.cuh:924-931),
 * in float: the sum rounded down to float has the exact sum's floor, as
 * every integer of this range is a float, and the float literal next to
 * 0.49999 separates the same floats (tests/rounding_check_mul.c checks every
 * float of magnitude below 2^18).  The reference clamps the result to
 * [-256, 255] before it adds the prediction and clamps to [0, 255], which
 * gives the same pixel without the first clamp. */
__device__ __forceinline__ float idct_round(float v)
{
    return __fadd_rn(floor_biased(__fadd_rd(v, 0.49999f)), -kBias);
}

/* ---------------------------------------------------------- per MB */

/* mb / mbw for mb < 4096: half a step above the quotient's lower end, which
 * is at least 0.5 / mbw away from an integer, where the approximate
 * reciprocal is off by less than 2^-10 / mbw */
__device__ __forceinline__ int mb_row(int mb, int mbw) { return (int)__fdividef((float)mb + 0.5f, (float)mbw); }

struct MbDecision {
    int32_t type, flags, mvx, mvy, cost;
};

/* start the asynchronous copies of one MB's inputs into buffer k.  The
 * window is 46 rows of three 16-byte chunks; picture widths are multiples
 * of 16 and luma planes 16-byte aligned, so a chunk lies wholly inside or
 * wholly outside the picture, and one outside is zero-filled.  Lanes 0-29
 * take (row, chunk) = (lane / 3 + 10 i, lane % 3). */
__device__ __forceinline__ void stage_mb(uint32_t *wbuf, int k, const h261b_session_dev_t &S, int mbx, int mby,
                                         int lane, int row_lo = 0, int row_n = WIN_ROWS, uint64_t *bar = nullptr,
                                         uint32_t extra_bytes = 0)
{
    const int H = S.mbh * 16;
    const int x0 = mbx * 16, y0 = mby * 16;
    uint32_t *base = wbuf + 16 * k;
    if (bar) {
        /* bulk staging: one copy per window row inside the picture, of its
         * 16-byte chunks inside the picture (48 bytes, or 32 at a left or
         * right picture edge), into the same pitched rows; chunks outside
         * the picture are zeroed by plain stores.  Lane 0 arrives on the
         * buffer's barrier announcing the bytes of all the copies. */
        const int c_lo = mbx > 0 ? 0 : 1, c_hi = mbx < S.mbw - 1 ? 3 : 2;
        const uint32_t row_bytes = 16u * (uint32_t)(c_hi - c_lo);
        const int y_first = max(y0 - 15 + row_lo, 0), y_last = min(y0 - 15 + row_lo + row_n, H);
        const uint32_t bytes = y_last > y_first ? row_bytes * (uint32_t)(y_last - y_first) : 0u;
        fence_proxy_async();
        if (lane == 0)
            mbar_arrive_expect(bar, bytes + extra_bytes);
        for (int r = row_lo + lane; r < row_lo + row_n; r += 32) {
            const int y = y0 - 15 + r;
            uint32_t *dst = base + r * WIN_PITCH_W;
            if (y >= 0 && y < H && H261B_CHECK(x0 - 16 + 16 * c_lo >= 0 && x0 - 16 + 16 * c_hi <= S.mbw * 16,
                                               CHK_STAGE_WINDOW, x0))
                bulk_copy(dst + 4 * c_lo, S.ref_y + (size_t)y * S.pitch_y + x0 - 16 + 16 * c_lo, row_bytes, bar);
            const uint4 z = make_uint4(0u, 0u, 0u, 0u);
            for (int j = 0; j < 3; j++)
                if (y < 0 || y >= H || j < c_lo || j >= c_hi)
                    *reinterpret_cast<uint4 *>(dst + 4 * j) = z;
        }
    } else if (lane < 30) {
        const int j = lane % 3, r0 = lane / 3;
        const bool xok = j == 1 || (j == 0 ? mbx > 0 : mbx < S.mbw - 1);
        const int x = x0 - 16 + 16 * j;
        uint32_t *dst = base + 4 * j;
        for (int r = row_lo + r0; r < row_lo + row_n; r += 10) {
            const int y = y0 - 15 + r;
            bool ok = xok && y >= 0 && y < H;
            ok = ok && H261B_CHECK(x >= 0 && x + 16 <= S.mbw * 16, CHK_STAGE_WINDOW, x);
            cp_async16z(dst + r * WIN_PITCH_W, ok ? S.ref_y + (size_t)y * S.pitch_y + x : S.ref_y, ok);
        }
    }
    if (lane < 16) {
        if (H261B_CHECK(y0 + lane < H && x0 + 16 <= S.mbw * 16, CHK_STAGE_SOURCE, y0 + lane))
            cp_async16(base + lane * WIN_PITCH_W + SRC_COL_W, S.cur_y + (size_t)(y0 + lane) * S.pitch_y + x0);
    } else {
        const int q = lane - 16, pl = q >> 3, r = q & 7;
        const uint8_t *src = pl ? S.cur_cr : S.cur_cb;
        if (H261B_CHECK(mby * 8 + r < S.mbh * 8 && mbx * 8 + 8 <= S.mbw * 8, CHK_STAGE_SOURCE, mby * 8 + r))
            cp_async8(base + (16 + q) * WIN_PITCH_W + SRC_COL_W,
                      src + (size_t)(mby * 8 + r) * S.pitch_c + mbx * 8);
    }
}

/* motion search + inter SATD costs; results are warp-uniform.  FULL: the
 * exhaustive search, else the reference's grid and refinement (a launch
 * compiles only the one it runs: a smaller body misses the instruction
 * cache less) */
template <bool FULL_SEARCH>
__device__ __forceinline__ void motion_estimate(const StageBuf s, const h261b_session_dev_t &S, int mbx, int mby,
                                                int lane, me_gpu_mb_t &res)
{
    const int bx = mbx * 16, by = mby * 16;
    /* per-MB limits, gpu_device.cu:226-265 */
    const int lminx = max(-15, -bx), lmaxx = min(15, (S.mbw - 1) * 16 - bx);
    const int lminy = max(-15, -by), lmaxy = min(15, (S.mbh - 1) * 16 - by);
    int vx, vy;
    /* a vector outside the limits never wins (the reference marks it with
     * the cost 65535, above every block's): its sum, from staged or
     * zero-filled pixels, is discarded; the zero vector is always inside */
    if (FULL_SEARCH) {
        const uint32_t best = full_search(s, lminx, lmaxx, lminy, lmaxy, lane) & 1023u;
        vx = (int)compact8(best) - 15;
        vy = (int)compact8(best >> 1) - 15;
    } else {
        const uint32_t coarse = grid_search(s, lminx, lmaxx, lminy, lmaxy, lane) & 1023u; /* Z-order index only */
        const int v1x = stage1_offset((int)compact8(coarse)), v1y = stage1_offset((int)compact8(coarse >> 1));
        const uint32_t best = refine_search(s, v1x, v1y, lminx, lmaxx, lminy, lmaxy, lane) & 1023u;
        vx = v1x + (int)compact8(best) - 3;
        vy = v1y + (int)compact8(best >> 1) - 3;
    }

    inter_costs<true, true>(s, vx, vy, lane, res.i_16x16_cost, res.i_16x16_filter_cost);
    res.s_16x16_mv.i8_mx = (int8_t)vx;
    res.s_16x16_mv.i8_my = (int8_t)vy;
}

/* a MB's ME results where the gpu_device.h boundary wants them */
__device__ __forceinline__ void me_results_out(const h261b_session_dev_t &S, int mb, const me_gpu_mb_t &me)
{
    if (S.me_out)
        S.me_out[mb] = me;
    if (S.me_host)
        S.me_host[mb] = me;
    if (S.start_mv)
        S.start_mv[mb] = S.cand_mv[mb] = me.s_16x16_mv;
}

/* a coded MB's record in the reference's layout (without its levels) */
__device__ __forceinline__ void abi_record_out(h261_macroblock_t *o, const MbDecision &m, int flags, int quant,
                                               uint32_t cbp, int mbx, int mby)
{
    o->i_macroblock_address = 0;
    o->i_macroblock_type = m.type;
    o->i_macroblock_type_flags = flags;
    o->i_macroblock_quant = quant;
    o->rgi_mv[0] = m.mvx;
    o->rgi_mv[1] = m.mvy;
    o->i_coded_block_pattern = (int32_t)cbp;
    o->i_mb_x = mbx * 16;
    o->i_mb_y = mby * 16;
}

/* h261_moded.c:53-95 */
__device__ __forceinline__ MbDecision mode_decide(const me_gpu_mb_t &g, int frame_type)
{
    MbDecision m;
    if (frame_type == H261B_FRAME_TYPE_INTRA ||
        (g.i_intra_cost <= g.i_16x16_cost && g.i_intra_cost <= g.i_16x16_filter_cost)) {
        m.type = H261B_MB_TYPE_INTRA;
        m.cost = g.i_intra_cost;
        m.flags = 0;
        m.mvx = m.mvy = 0;
    } else {
        m.type = H261B_MB_TYPE_INTER;
        if (g.i_16x16_filter_cost < g.i_16x16_cost) {
            m.flags = H261B_MB_MC | H261B_MB_FILTER;
            m.cost = g.i_16x16_filter_cost;
        } else {
            m.flags = 0;
            m.cost = g.i_16x16_cost;
        }
        m.mvx = g.s_16x16_mv.i8_mx;
        m.mvy = g.s_16x16_mv.i8_my;
        if (m.mvx != 0 || m.mvy != 0)
            m.flags |= H261B_MB_MC;
    }
    return m;
}

/* byte i of a row of eight, as the float 2^23 + x */
__device__ __forceinline__ float pixel_biased(uint2 v, int i)
{
    return __uint_as_float(__byte_perm(i < 4 ? v.x : v.y, 0x4B000000u, 0x7650u + (uint32_t)(i & 3)));
}

/* the low bytes of four words */
__device__ __forceinline__ uint32_t pack4(float a, float b, float c, float d)
{
    return __byte_perm(__byte_perm(__float_as_uint(a), __float_as_uint(b), 0x0040),
                       __byte_perm(__float_as_uint(c), __float_as_uint(d), 0x0040), 0x5410);
}

/* H.261 loop filter of one row of an 8x8 block per lane (mbgpu_kernels.cuh
 * :88-166): [1 2 1] across and down, x4 at the block's edge columns and
 * rows.  Sums of four pixels at a time in 16-bit fields (4,088 at most), the
 * rows above and below from the neighbouring lanes; an edge row takes itself
 * for both, which gives (4 h + 8) >> 4 = (h + 2) >> 2. */
__device__ __forceinline__ uint2 loop_filter(uint2 v, int lane)
{
    const uint32_t e0 = __byte_perm(v.x, 0u, 0x4240), o0 = __byte_perm(v.x, 0u, 0x4341);   /* 0, 2; 1, 3 */
    const uint32_t e1 = __byte_perm(v.y, 0u, 0x4240), o1 = __byte_perm(v.y, 0u, 0x4341);   /* 4, 6; 5, 7 */
    uint32_t h[4];
    h[0] = ((2u * e0 + o0 + (o0 << 16)) & 0xFFFF0000u) | ((4u * e0) & 0xFFFFu);            /* 0, 2 */
    h[1] = 2u * o0 + e0 + __byte_perm(e0, e1, 0x5432);                                     /* 1, 3 */
    h[2] = 2u * e1 + o1 + __byte_perm(o0, o1, 0x5432);                                     /* 4, 6 */
    h[3] = ((2u * o1 + e1 + (e1 >> 16)) & 0xFFFFu) | ((4u * o1) & 0xFFFF0000u);            /* 5, 7 */
    const int r = lane & 7;
    const bool edge = r == 0 || r == 7;
    const int up = edge ? lane : lane - 1, down = edge ? lane : lane + 1;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t t = __shfl_sync(FULL, h[i], up) + 2u * h[i] + __shfl_sync(FULL, h[i], down) + 0x00080008u;
        h[i] = (t >> 4) & 0x00FF00FFu;
    }
    return make_uint2(h[0] + (h[1] << 8), h[2] + (h[3] << 8));
}

/* what a lane needs of its block for one pass: the row lane & 7 of its
 * pixels, then the column lane & 7 of its coefficients */
struct BlockRow {
    uint2 cur, pred;       /* the source row and its prediction (0 for intra)  */
    uint8_t *rec;          /* where the reconstructed row goes                 */
    bool active;
};

/* one pass over up to four blocks of the MB: lane = slot * 8 + row (then
 * column).  Adds |coefficient| before the denoise to noise[v] (a float:
 * integers below 2^24), and returns this pass's CBP bits.
 *
 * Everything between the pixels and the packed bytes is held in floats that
 * are integers or the reference's own floats: sums with 2^23 or 1.5 * 2^23
 * take the place of conversions, which run on a pipe of an eighth of the
 * rate, and the statistics stay with their lane until a run is published.
 * With the packed loop filter, 16-byte rows in the transpose buffer and no
 * inverse transform for a pass without a coded block: 98.9 -> 83.4 us for
 * the encode launch of 13,464 macroblocks of mixed streams, 716 -> 554 us for
 * 1024 QCIF streams, 43.9 -> 40.7 us for 16 intra CIF pictures. */
template <int FMAD, bool ABI, bool CODE>
__device__ __forceinline__ uint32_t encdec_pass(float (*tb)[TB_BLOCK], uint32_t *cm, const BlockRow &row,
                                                const h261b_session_dev_t &S, int mb, const MbDecision &m, int quant,
                                                uint4 offw, bool luma_pass, int lane, float fwd_c, float inv_c,
                                                float noise[8], uint32_t &ssd)
{
    const int slot = lane >> 3, c = lane & 7;
    const int b = luma_pass ? slot : 4 + (slot & 1);
    const bool intra = m.type == H261B_MB_TYPE_INTRA, active = row.active;
    float *const t = tb[slot];
    /* ---- residual and FDCT pass 1 on row c (mbgpu_kernels.cuh:59-166, :359-388) */
    {
        float res[8], o[8];
#pragma unroll
        for (int i = 0; i < 8; i++)
            res[i] = __fsub_rn(pixel_biased(row.cur, i), pixel_biased(row.pred, i));
        fdct_butterfly<FMAD, true>(res[0] + res[7], res[1] + res[6], res[2] + res[5], res[3] + res[4],
                                   res[3] - res[4], res[2] - res[5], res[1] - res[6], res[0] - res[7], o);
        *reinterpret_cast<float4 *>(t + c * TB_ROW) = make_float4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<float4 *>(t + c * TB_ROW + 4) = make_float4(o[4], o[5], o[6], o[7]);
    }
    __syncwarp();

    /* ---- FDCT pass 2 on column c: coefficients (v, c), v = 0..7 */
    float lev[8];   /* the levels, signed */
    uint32_t lo, hi;
    int32_t acc;
    {
        float q[8], o[8];
#pragma unroll
        for (int k = 0; k < 8; k++)
            q[k] = t[k * TB_ROW + c];
        fdct_butterfly<FMAD, false>(q[0] + q[7], q[1] + q[6], q[2] + q[5], q[3] + q[4], q[3] - q[4], q[2] - q[5],
                                    q[1] - q[6], q[0] - q[7], o);
        const float inv = c_inv_quant[quant];
        const uint32_t ow[4] = { offw.x, offw.y, offw.z, offw.w };
        float mag[8];
        int32_t dc = 0;
#pragma unroll
        for (int v = 0; v < 8; v++) {
            const float lv = fdct_round(fwd_c, c_fwd_post[v], o[v]);
            noise[v] += active ? fabsf(lv) : 0.0f;
            /* denoise (mbgpu_kernels.cuh:586-604) on the magnitude, quant
             * (:689-716): the product truncated, which is the same on the
             * magnitude, at most 127 */
            const float off = (float)((ow[v >> 1] >> (16 * (v & 1))) & 0xFFFFu);
            const float shrunk = fmaxf(fabsf(lv) - off, 0.0f);
            mag[v] = __fadd_rz(fminf(__fmul_rn(shrunk, inv), 127.0f), 8388608.0f);
            lev[v] = copysignf(__fadd_rn(mag[v], -8388608.0f), lv);
            if (v == 0) {
                /* intra DC: the denoised coefficient / 8 as 1 .. 254, 128 as 255 */
                dc = (int32_t)copysignf(shrunk, lv) / 8;
                dc = min(max(dc, 1), 254);
                dc = dc == 128 ? 255 : dc;
            }
        }
        /* the coded-block rule: 100 for a level beyond +-1 (and an intra DC),
         * 1 for +-1 */
        const uint32_t m0 = pack4(mag[0], mag[1], mag[2], mag[3]), m1 = pack4(mag[4], mag[5], mag[6], mag[7]);
        lo = pack4(__fadd_rn(lev[0], kBias), __fadd_rn(lev[1], kBias), __fadd_rn(lev[2], kBias),
                   __fadd_rn(lev[3], kBias));
        hi = pack4(__fadd_rn(lev[4], kBias), __fadd_rn(lev[5], kBias), __fadd_rn(lev[6], kBias),
                   __fadd_rn(lev[7], kBias));
        acc = __popc((m0 & 0x01010101u) | ((m1 & 0x01010101u) << 1));
        acc = ((m0 | m1) & 0xFEFEFEFEu) || (intra && c == 0) ? 100 : acc;
        if (intra && c == 0) {
            lo = (lo & 0xFFFFFF00u) | (uint32_t)dc;
            lev[0] = dc == 255 ? 128.0f : (float)dc;
        }
    }
    /* block sums over the 8 lanes of a block */
    acc += __shfl_xor_sync(FULL, acc, 1);
    acc += __shfl_xor_sync(FULL, acc, 2);
    acc += __shfl_xor_sync(FULL, acc, 4);
    const bool coded = active && acc > 2;
    const uint32_t cbp = __reduce_or_sync(FULL, coded ? (uint32_t)H261B_CBP_BIT(b) : 0u);

    /* ---- levels out: column-major, this lane's eight are contiguous */
    if (active) {
        if (ABI && S.abi_out) {
            int32_t *tc = S.abi_out[mb].rgi_tcoeff[b];
#pragma unroll
            for (int v = 0; v < 8; v++) {
                const uint32_t x = (v < 4 ? lo : hi) >> (8 * (v & 3));
                tc[v * 8 + c] = v == 0 && c == 0 && intra ? (int32_t)(x & 0xFFu) : (int32_t)(int8_t)x;
            }
        }
        if (S.level_out)
            *reinterpret_cast<uint2 *>(S.level_out + (size_t)mb * 384 + b * 64 + c * 8) = make_uint2(lo, hi);
        if (CODE)
            *reinterpret_cast<uint2 *>(cm + b * 16 + c * 2) = make_uint2(lo, hi);
    }

    /* ---- dequant (mbgpu_kernels.cuh:763-814) and IDCT pass 1 on column c;
     * a block that is not coded has coefficients of zero, and a pass without
     * a coded block is its prediction */
    uint2 out = row.pred;
    if (cbp) {
        const float qa = coded ? (float)((quant - 1) | 1) : 0.0f, qm = coded ? (float)(2 * quant) : 0.0f;
        float P[8], cs[8], tt[8], o[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            /* level * 2 QUANT, plus its sign times QUANT rounded down to odd */
            const float sign = fminf(fmaxf(lev[k], -1.0f), 1.0f);
            float dq = __fmaf_rn(lev[k], qm, __fmul_rn(sign, qa));
            dq = fminf(fmaxf(dq, -2048.0f), 2047.0f);
            if (k == 0 && intra && c == 0)
                dq = lev[0] * 8.0f;
            /* prescale: t = (coef * pre[col]) * (pre[row] * 0.125) */
            cs[k] = __fmul_rn(c_inv_pre[k], 0.125f); /* exact, as dmulf(.., 0.125) */
            P[k] = __fmul_rn(dq, inv_c);
            tt[k] = __fmul_rn(P[k], cs[k]);
        }
        idct_rest<FMAD>(first_sub<FMAD>(P[2], cs[2], tt[2], tt[6]), first_add<FMAD>(P[2], cs[2], tt[2], tt[6]),
                        first_add<FMAD>(P[0], cs[0], tt[0], tt[4]), first_sub<FMAD>(P[0], cs[0], tt[0], tt[4]),
                        first_add<FMAD>(P[1], cs[1], tt[1], tt[7]), first_sub<FMAD>(P[1], cs[1], tt[1], tt[7]),
                        first_add<FMAD>(P[5], cs[5], tt[5], tt[3]), first_sub<FMAD>(P[5], cs[5], tt[5], tt[3]), o);
        __syncwarp(); /* pass-2 reads of the transpose buffer are done */
#pragma unroll
        for (int k = 0; k < 8; k++)
            t[k * TB_ROW + c] = o[k];
        __syncwarp();

        /* ---- IDCT pass 2 on row c and reconstruction (mbgpu_kernels.cuh:988-1096) */
        const float4 p0 = *reinterpret_cast<const float4 *>(t + c * TB_ROW);
        const float4 p1 = *reinterpret_cast<const float4 *>(t + c * TB_ROW + 4);
        idct_rest<FMAD>(p0.z - p1.z, p0.z + p1.z, p0.x + p1.x, p0.x - p1.x, p0.y + p1.w, p0.y - p1.w, p1.y + p0.w,
                        p1.y - p0.w, o);
#pragma unroll
        for (int i = 0; i < 8; i++)
            o[i] = fminf(fmaxf(idct_round(o[i]) + pixel_biased(row.pred, i), 8388608.0f), 8388608.0f + 255.0f);
        out = make_uint2(pack4(o[0], o[1], o[2], o[3]), pack4(o[4], o[5], o[6], o[7]));
    }
    if (active) {
        *reinterpret_cast<uint2 *>(row.rec) = out;
        if (S.ssd_out) {
            /* squared error of this row against the source, for the
             * picture's PSNR (h261_main.c:38-91) */
            const uint32_t d0 = __vabsdiffu4(row.cur.x, out.x), d1 = __vabsdiffu4(row.cur.y, out.y);
            ssd = __dp4a(d0, d0, __dp4a(d1, d1, 0u));
        }
    }
    __syncwarp();
    return cbp;
}

/* the lane's row of the luma pass: block slot = lane / 8 */
__device__ __forceinline__ BlockRow luma_row(const StageBuf s, const h261b_session_dev_t &S, int mbx, int mby,
                                             const MbDecision &m, int lane)
{
    const int b = lane >> 3, r = lane & 7, bx8 = (b & 1) * 8, by8 = (b >> 1) * 8;
    BlockRow o;
    o.cur = *reinterpret_cast<const uint2 *>(s.cur(by8 + r, bx8 >> 2));
    o.pred = make_uint2(0u, 0u);
    if (m.type != H261B_MB_TYPE_INTRA) {
        int wr = 15 + m.mvy + by8, wc = 16 + m.mvx + bx8;
        /* rows wr..wr+7 of the 46-row window, byte columns wc..wc+7 with
         * win8's three words inside the 12-word row */
        if (!H261B_CHECK(wr >= 0 && wr + 7 < WIN_ROWS && wc >= 0 && wc <= 40, CHK_MC_WINDOW, wr * 64 + wc)) {
            wr = min(max(wr, 0), WIN_ROWS - 8);
            wc = min(max(wc, 0), 40);
        }
        o.pred = win8(s, wr + r, wc);
        if (m.flags & H261B_MB_FILTER)
            o.pred = loop_filter(o.pred, lane);
    }
    o.rec = S.rec_y + (size_t)(mby * 16 + by8 + r) * S.pitch_y + mbx * 16 + bx8;
    o.active = H261B_CHECK(mby * 16 + by8 + r < S.mbh * 16 && mbx * 16 + bx8 + 8 <= S.mbw * 16, CHK_RECON,
                           mby * 4096 + mbx);
    return o;
}

/* the words of the lane's chroma prediction row: loaded before the luma
 * pass, so that their latency passes behind it */
struct ChromaRef {
    uint32_t a, b, c, sh;
};

__device__ __forceinline__ ChromaRef chroma_ref(const h261b_session_dev_t &S, int mbx, int mby, const MbDecision &m,
                                                int lane)
{
    ChromaRef o = { 0u, 0u, 0u, 0u };
    if (m.type == H261B_MB_TYPE_INTRA)
        return o;
    const int pl = (lane >> 3) & 1, r = lane & 7;
    int cmx = m.mvx / 2, cmy = m.mvy / 2; /* truncation toward zero */
#ifdef H261B_DEBUG_CHECKS
    /* rows inside the chroma plane; the words (12 bytes from the word
     * boundary when unaligned) inside the row */
    {
        const int cx = mbx * 8 + cmx, cy = mby * 8 + cmy, wc8 = S.mbw * 8;
        if (!H261B_CHECK(cy >= 0 && cy + 8 <= S.mbh * 8 && cx >= 0 && (cx & ~3) + ((cx & 3) ? 12 : 8) <= wc8,
                         CHK_MC_CHROMA, cy * 4096 + cx))
            cmx = cmy = 0;
    }
#endif
    const uint8_t *g = (pl ? S.ref_cr : S.ref_cb) + (size_t)(mby * 8 + cmy + r) * S.pitch_c + (mbx * 8 + cmx);
    /* only the words that hold one of the row's bytes */
    const uint32_t *p = reinterpret_cast<const uint32_t *>((uintptr_t)g & ~(uintptr_t)3);
    o.sh = (uint32_t)((uintptr_t)g & 3) * 8u;
    if (lane < 16) {
        o.a = p[0];
        o.b = p[1];
        o.c = o.sh ? p[2] : 0u;
    }
    return o;
}

/* the lane's row of the chroma pass: lanes 0-7 Cb, 8-15 Cr; lanes 16-31
 * write nothing */
__device__ __forceinline__ BlockRow chroma_row(const StageBuf s, const h261b_session_dev_t &S, int mbx, int mby,
                                               const MbDecision &m, const ChromaRef &f, int lane)
{
    const int pl = (lane >> 3) & 1, r = lane & 7;
    BlockRow o;
    o.cur = *reinterpret_cast<const uint2 *>(s.curc(8 * pl + r));
    o.pred = make_uint2(__funnelshift_r(f.a, f.b, f.sh), __funnelshift_r(f.b, f.c, f.sh));
    if (m.type != H261B_MB_TYPE_INTRA && (m.flags & H261B_MB_FILTER))
        o.pred = loop_filter(o.pred, lane);
    o.rec = (pl ? S.rec_cr : S.rec_cb) + (size_t)(mby * 8 + r) * S.pitch_c + mbx * 8;
    o.active = lane < 16 && H261B_CHECK(mby * 8 + r < S.mbh * 8 && mbx * 8 + 8 <= S.mbw * 8, CHK_RECON,
                                        mby * 4096 + mbx);
    return o;
}

/* frame-end denoise update by the session's last warp (mbgpu_kernels.cuh:478-503).
 * Every other warp has published, and this one has acquired their counts: it
 * alone holds the state until the launch ends, so plain loads from L2, all in
 * flight together, and stores do (one exchange after another was 2 us at the
 * end of every launch). */
__device__ __forceinline__ void denoise_frame_end(h261b_denoise_dev_t *dn, int lane)
{
    const int32_t cnt0 = __ldcg(&dn->count[0]), cnt1 = __ldcg(&dn->count[1]), strength = dn->denoise;
    int32_t n0[2], n1[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        n0[h] = __ldcg(&dn->noise[0][lane + 32 * h]);
        n1[h] = __ldcg(&dn->noise[1][lane + 32 * h]);
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int p = lane + 32 * h, u = p & 7, v = p >> 3;
        /* the reference keeps Int32 offsets and loads them as UInt16 */
        dn->offset[1][u][v] = (uint16_t)((cnt1 * strength + n1[h] / 2) / (n1[h] + 1));
        dn->offset[0][u][v] = (uint16_t)((cnt0 * strength + n0[h] / 2) / (n0[h] + 1));
        dn->noise[0][p] = dn->noise[1][p] = 0;
    }
    __syncwarp();   /* every lane has the counts */
    if (lane == 0) {
        dn->count[0] = dn->count[1] = 0;
        dn->ticket = 0u;
    }
}

/* publish a warp's statistics for a run of n MBs of one session and type,
 * and clear them; the publication that completes the session's frame updates
 * the offsets.  noise[v] holds the lane's own blocks' sum for coefficient
 * (v, lane & 7). */
__device__ __forceinline__ void add_noise(h261b_denoise_dev_t *dn, int t, float noise[8], int lane)
{
#pragma unroll
    for (int v = 0; v < 8; v++) {
        int32_t x = (int32_t)noise[v];
        noise[v] = 0.0f;
        x += __shfl_xor_sync(FULL, x, 8);
        x += __shfl_xor_sync(FULL, x, 16);
        if (lane < 8 && x)
            atomicAdd(&dn->noise[t][v * 8 + lane], x);
    }
}

__device__ __forceinline__ void publish_run(const h261b_session_dev_t &S, int t, int n, float noise[8], int lane)
{
    h261b_denoise_dev_t *dn = S.dn;
    add_noise(dn, t, noise, lane);
    if (lane == 0)
        atomicAdd(&dn->count[t], 6 * n);
    __threadfence();
    __syncwarp();
    uint32_t last = 0;
    if (lane == 0) {
        last = atomicAdd(&dn->ticket, (uint32_t)n) + (uint32_t)n == (uint32_t)(S.mbw * S.mbh) ? 1u : 0u;
        /* the run's levels, strings and records are written and fenced: count
         * its MBs for the kernel after this launch */
        atomicAdd(const_cast<int32_t *>(&S.mbs_done), n);
    }
    last = __shfl_sync(FULL, last, 0);
    if (last) {
        __threadfence();
        denoise_frame_end(dn, lane);
    }
}

/* resident CTAs of 256 threads the register allocation must allow per SM */
#ifndef H261B_STEP_MIN_BLOCKS
#define H261B_STEP_MIN_BLOCKS 2
#endif
/* the search-only kernel keeps neither the transforms' registers nor the
 * transpose buffer, so more of its CTAs fit an SM */
#ifndef H261B_SEARCH_MIN_BLOCKS
#define H261B_SEARCH_MIN_BLOCKS 3
#endif

/* Work items are handed out in two parts.  Warp w first takes the static
 * run [w * chunk, (w + 1) * chunk) of the first total_warps * chunk items
 * (consecutive MBs of mostly one session: neighbouring windows hit in L1
 * and the denoise statistics publish once per run).  With a scheduler
 * (sched != nullptr, two zeroed counters) the remaining items are then
 * drawn one at a time from sched[0], so that warps which met cheaper MBs
 * take more of the tail; every warp makes exactly one fetch past the end,
 * and the last warp to finish (sched[1]) zeroes both counters for the next
 * launch.  Without a scheduler the static runs cover every item. */
/* FMAD: the arithmetic of the reference's default build; KIND: what the
 * launch does per MB; FULL_SEARCH: the exhaustive search instead of the
 * reference's; ABI: the launch may write the reference-layout outputs
 * (h261_macroblock_t records, ME results and vectors) that only the
 * gpu_device.h boundary asks for; BULK: the search window comes by bulk row
 * copies; CODE: the launch makes the MBs' coefficient bit strings.  Each launch runs the instantiation for its flags
 * (h261b_launch_step), so no launch carries code it never runs: instruction
 * fetch is a seventh of the kernel's stalls, and leaving the bulk staging's
 * code out of the cp.async kernel alone took its launch of 13,464
 * macroblocks from 83.0 to 79.4 us. */
template <int FMAD, int KIND, bool FULL_SEARCH, bool ABI, bool BULK, bool CODE>
__global__ void __launch_bounds__(256, KIND == KIND_SEARCH ? H261B_SEARCH_MIN_BLOCKS : H261B_STEP_MIN_BLOCKS)
    step_kernel(const h261b_session_dev_t *__restrict__ sessions, const uint32_t *__restrict__ work, int32_t n_work,
                int32_t chunk, int32_t phases_arg, int32_t *sched)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    /* the kernel after this one (the encode launch after a search launch,
     * or the bitstream kernel) may launch now; it waits for the whole grid
     * before it reads anything (griddepcontrol.wait) */
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    /* an encode launch reads the mode decisions of the search launch before
     * it, a launch with the programmatic dependency what the kernel before it
     * writes: wait for that grid and its writes (a no-op when launched without
     * the dependency) */
    if (KIND == KIND_ENCODE || (phases_arg & H261B_LAUNCH_PDL))
        asm volatile("griddepcontrol.wait;" ::: "memory");
    const int phases = KIND == KIND_SEARCH   ? (H261B_PHASE_ME | H261B_PHASE_MD)
                       : KIND == KIND_ENCODE ? H261B_PHASE_ENCDEC
                       : KIND == KIND_FULL   ? (H261B_PHASE_ME | H261B_PHASE_MD | H261B_PHASE_ENCDEC)
                                             : phases_arg;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t warp_bytes = KIND == KIND_SEARCH ? kSearchWarpBytes : CODE ? sizeof(WarpSmem) : kEncodeWarpBytes;
    unsigned char *mine = smem_raw + warp * warp_bytes;
    uint32_t *wbuf = reinterpret_cast<uint32_t *>(mine);
    float(*tb)[TB_BLOCK] = reinterpret_cast<WarpSmem *>(mine)->t;   /* not used by KIND_SEARCH */
    VlcScratch &vlc = reinterpret_cast<WarpSmem *>(mine)->vlc;      /* nor this */
    VlcTables &tables = *reinterpret_cast<VlcTables *>(smem_raw + (blockDim.x >> 5) * warp_bytes);
    /* this lane's column factors: forward post-scale (times 0.125, exact)
     * and inverse pre-scale */
    const float fwd_c = __fmul_rn(c_fwd_post[lane & 7], 0.125f), inv_c = c_inv_pre[lane & 7];
    /* bulk staging: the two buffers' barriers; per buffer, the parity of
     * its next phase, whether its current staging used the barrier, and
     * whether a wait on it gave up.  A barrier whose wait gave up is not
     * armed again (its phase may never complete): that buffer falls back to
     * cp.async staging, and at the end the warp waits once more, bounded,
     * for the copies of the phase that gave up. */
    uint64_t *bars = BULK ? reinterpret_cast<WarpSmem *>(mine)->bar : nullptr;
    uint32_t parity = 0, bulk_used = 0, stuck = 0;
#ifdef H261B_DEBUG_CHECKS
    /* checking build only: the warp's first bulk staging announces 16 bytes
     * more than its copies bring, so that its wait runs out (the test of the
     * bounded wait and of h261b_stage_status) */
    uint32_t short_first = (phases_arg & H261B_STAGE_SHORT) ? 16u : 0u;
#else
    const uint32_t short_first = 0u;
#endif
    if (bars) {
        if (lane == 0) {
            mbar_init(&bars[0]);
            mbar_init(&bars[1]);
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
        __syncwarp();
    }
    if (CODE) {
        load_vlc_tables(tables, (int)threadIdx.x, (int)blockDim.x);
        for (int i = lane; i < VLC_MB_WORDS; i += 32)
            vlc.stage[i] = 0u;
        __syncthreads();
    }
    const int warps = blockDim.x >> 5;
    const int total_warps = gridDim.x * warps;
    const int n_static = sched ? min(n_work, total_warps * chunk) : n_work;
    int static_next = (blockIdx.x * warps + warp) * chunk;
    const int static_end = min(static_next + chunk, n_static);
    /* the warp's next work item (n_work when it has none left): a static
     * index, or a draw from the scheduler while the static run lasts */
    auto next_item = [&]() -> int {
        if (static_next < static_end)
            return static_next++;
        if (!sched)
            return n_work;
        int v = 0;
        if (lane == 0)
            v = n_static + atomicAdd(&sched[0], 1);
        return min(__shfl_sync(FULL, v, 0), n_work);
    };
    const bool want_enc = (phases & H261B_PHASE_ENCDEC) != 0;
    /* start the copies of a work item's inputs into buffer k: the whole
     * search window, or for an encode launch only the 16 window rows its
     * prediction block covers (none for an intra MB) */
    auto stage_item = [&](int k, uint32_t it) {
        const h261b_session_dev_t &N = sessions[it >> 12];
        const int nmb = (int)(it & 0xFFFu), nmby = mb_row(nmb, N.mbw), nmbx = nmb - nmby * N.mbw;
        uint64_t *bar = (bars && !((stuck >> k) & 1u)) ? &bars[k] : nullptr;
        const uint32_t extra = bar ? short_first : 0u;
        if (bar) {
            bulk_used |= 1u << k;
#ifdef H261B_DEBUG_CHECKS
            short_first = 0u;
#endif
        } else {
            bulk_used &= ~(1u << k);
        }
        if (KIND == KIND_ENCODE) {
            const h261_mb_mode_decision_t &d = N.md_in[nmb];
            const bool inter = d.i_mb_type != H261B_MB_TYPE_INTRA;
            stage_mb(wbuf, k, N, nmbx, nmby, lane, 15 + d.i_mv_y, inter ? 16 : 0, bar, extra);
        } else {
            stage_mb(wbuf, k, N, nmbx, nmby, lane, 0, WIN_ROWS, bar, extra);
        }
    };

    int g = next_item();
    uint32_t item = g < n_work ? work[g] : 0u;
    if (g < n_work) {
        stage_item(0, item);
        cp_async_commit();
    }
    /* the item after g, known one MB ahead of its staging */
    int gn = g < n_work ? next_item() : n_work;
    uint32_t nitem = gn < n_work ? work[gn] : 0u;

    int run_s = -1, run_t = 0, run_n = 0;
    float noise[8];
#pragma unroll
    for (int v = 0; v < 8; v++)
        noise[v] = 0.0f;

    for (int cur = 0; g < n_work; cur ^= 1) {
        const int gnn = gn < n_work ? next_item() : n_work;
        const uint32_t nnitem = gnn < n_work ? work[gnn] : 0u;
        if (gn < n_work) {
            stage_item(cur ^ 1, nitem);
            cp_async_commit();
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        if ((bulk_used >> cur) & 1u) {
            /* a wait that gives up is counted; the buffer's barrier is not
             * used again, so no arrival meets a phase that never ended */
            if (!__all_sync(FULL, mbar_wait_bounded(&bars[cur], (parity >> cur) & 1u, lane)))
                stuck |= 1u << cur;
            else
                parity ^= 1u << cur;
        }
        __syncwarp();

        const int sidx = (int)(item >> 12);
        const h261b_session_dev_t &S = sessions[sidx];
        const int mb = (int)(item & 0xFFFu);
        if (!H261B_CHECK(mb < S.mbw * S.mbh, CHK_WORK_ITEM, (int)item)) {
            /* an item past its picture: nothing of it is read or written */
            __syncwarp();
            g = gn;
            item = nitem;
            gn = gnn;
            nitem = nnitem;
            continue;
        }
        const int mby = mb_row(mb, S.mbw), mbx = mb - mby * S.mbw;
        const StageBuf b = stage_view(wbuf, cur);
        const bool do_me = (phases & H261B_PHASE_ME) && !S.skip_search;

        me_gpu_mb_t me;
        me.i_intra_cost = me.i_zero_cost = me.i_16x16_cost = me.i_16x16_filter_cost = 0;
        me.s_16x16_mv.i8_mx = me.s_16x16_mv.i8_my = 0;
        if (do_me || (phases & H261B_PHASE_MD))
            me.i_intra_cost = intra_cost(b, lane);   /* all that an intra picture needs */
        if (do_me) {
            /* the launch's search mode is the session's (checking build) */
            (void)H261B_CHECK(S.me_mode == (FULL_SEARCH ? 1 : 0), CHK_WORK_ITEM, S.me_mode);
            motion_estimate<FULL_SEARCH>(b, S, mbx, mby, lane, me);
            if (ABI && lane == 0)
                me_results_out(S, mb, me);
        }

        MbDecision m;
        if (phases & H261B_PHASE_MD) {
            m = mode_decide(me, S.frame_type);
            if (lane == 0 && S.rc)
                atomicAdd(&S.rc->cost_sum, m.cost);   /* the rate control's picture cost */
            if (lane == 0 && S.md_out) {
                h261_mb_mode_decision_t o;
                o.i_cost = m.cost;
                o.i_quantiser_adjust = 0;
                o.i_mb_type = m.type;
                o.i_mb_flags = m.flags;
                o.i_mv_x = m.mvx;
                o.i_mv_y = m.mvy;
                S.md_out[mb] = o;
            }
        } else if (S.md_in) {
            const h261_mb_mode_decision_t &d = S.md_in[mb];
            m.type = d.i_mb_type;
            m.flags = d.i_mb_flags;
            m.mvx = d.i_mv_x;
            m.mvy = d.i_mv_y;
            m.cost = d.i_cost;
        } else {
            m.type = H261B_MB_TYPE_INTRA;
            m.flags = m.mvx = m.mvy = m.cost = 0;
        }

        /* a rate-controlled session is encoded by a second launch, once its
         * picture QUANT is known */
        if (want_enc && !(S.rc && (phases & H261B_PHASE_MD))) {
            const int t = m.type == H261B_MB_TYPE_INTRA ? 0 : 1;
            /* (the noise sums are exact below 2^24: 4,000 MBs of 2,041) */
            if (run_n > 0 && (sidx != run_s || t != run_t || run_n >= 2048)) {
                publish_run(sessions[run_s], run_t, run_n, noise, lane);
                run_n = 0;
            }
            run_s = sidx;
            run_t = t;
            int quant = S.rc ? S.rc->picture_quant : S.quant;
            if (S.md_in && !(phases & H261B_PHASE_MD))
                quant += S.md_in[mb].i_quantiser_adjust;
            quant = min(31, max(1, quant)); /* gpu_device.cu:625-627 */
            /* the luma pass, then the chroma pass, each its own copy of the
             * pass's code: straight code fetches ahead, and with the pass at
             * half its former size two copies run faster than a loop (79.5
             * -> 78.2 us for 13,464 macroblocks of mixed streams, 519 -> 504
             * us for 1024 QCIF streams) */
            uint32_t ssd_l = 0, ssd_c = 0, cbp = 0;
            /* this column's eight denoise offsets, UInt16, one 16-byte load */
            const uint4 offw = *reinterpret_cast<const uint4 *>(&S.dn->offset[t][lane & 7][0]);
            const ChromaRef ref = chroma_ref(S, mbx, mby, m, lane);
            cbp = encdec_pass<FMAD, ABI, CODE>(tb, vlc.cm, luma_row(b, S, mbx, mby, m, lane), S, mb, m, quant, offw, true, lane,
                                         fwd_c, inv_c, noise, ssd_l);
            cbp |= encdec_pass<FMAD, ABI, CODE>(tb, vlc.cm, chroma_row(b, S, mbx, mby, m, ref, lane), S, mb, m, quant, offw, false,
                                          lane, fwd_c, inv_c, noise, ssd_c);
            if (S.ssd_out) {
                const uint32_t ey = __reduce_add_sync(FULL, ssd_l);
                const uint32_t ecb = __reduce_add_sync(FULL, lane < 8 ? ssd_c : 0u);
                const uint32_t ecr = __reduce_add_sync(FULL, lane >= 8 && lane < 16 ? ssd_c : 0u);
                if (lane == 0) {
                    atomicAdd(&S.ssd_out[0], (unsigned long long)ey);
                    atomicAdd(&S.ssd_out[1], (unsigned long long)ecb);
                    atomicAdd(&S.ssd_out[2], (unsigned long long)ecr);
                }
            }
            run_n++;

            const int flags = m.flags | (cbp ? H261B_MB_COEFF : 0);
            /* the MB's coefficient bit string: all blocks of an intra MB, the
             * coded ones of an inter MB (bit b = block b) */
            int coef_bits = 0;
            if (CODE && S.bits_out) {
                const bool intra = m.type == H261B_MB_TYPE_INTRA;
                const uint32_t blocks = intra ? 63u : __brev(cbp) >> 26;
                if (blocks) {
                    int oob = 0;
                    const int pos = code_mb(blocks, intra, tables, vlc, lane, oob);
                    coef_bits = store_mb_string(vlc.stage, S.vlc_scratch + (size_t)mb * VLC_MB_WORDS, pos, oob, lane);
                }
            }
            if (lane == 0) {
                if (ABI && S.abi_out)
                    abi_record_out(&S.abi_out[mb], m, flags, quant, cbp, mbx, mby);
                if (S.info_out) {
                    h261b_mb_info_t inf;
                    inf.type = (int16_t)m.type;
                    inf.flags = (int16_t)flags;
                    inf.quant = (int8_t)quant;
                    inf.cbp = (int8_t)cbp;
                    inf.mvx = (int8_t)m.mvx;
                    inf.mvy = (int8_t)m.mvy;
                    inf.cost = m.cost;
                    inf.coef_bits = coef_bits;
                    S.info_out[mb] = inf;
                }
            }
        }
        __syncwarp(); /* this buffer may be refilled from the next iteration on */
        g = gn;
        item = nitem;
        gn = gnn;
        nitem = nnitem;
    }
    if (want_enc && run_n > 0)
        publish_run(sessions[run_s], run_t, run_n, noise, lane);
    if (bars) {
        for (int k = 0; k < 2; k++) {
            /* the copies of a phase whose wait gave up may still be landing:
             * wait for them once more, bounded, before the CTA's shared
             * memory goes; a barrier left in a phase is not invalidated */
            bool done = true;
            if ((stuck >> k) & 1u)
                done = __all_sync(FULL, mbar_wait_bounded(&bars[k], (parity >> k) & 1u, lane));
            if (done && lane == 0)
                mbar_inval(&bars[k]);
        }
    }
    if (sched && lane == 0) {
        __threadfence();
        if (atomicAdd(&sched[1], 1) == total_warps - 1) {
            atomicExch(&sched[0], 0);
            atomicExch(&sched[1], 0);
        }
    }
}

/* ---------------------------------------------- a team of warps per MB
 *
 * A small launch (at most four MBs a multiprocessor) leaves most of the
 * chip's warp slots empty, and its time is the one chain a macroblock goes
 * through.  Here a CTA of four warps takes each macroblock and the chain's
 * long links are shared out: every thread one vector of the coarse grid, two
 * threads each of the refinement's other 48 (the centre's cost is known) or
 * eight vectors each of the exhaustive search, the three costs on three
 * warps, luma and chroma passes side by side, and the coding of the bits on a
 * third warp.  The arithmetic is the one-warp kernel's throughout. */
struct TeamSmem {
    alignas(16) uint32_t buf[WIN_ROWS * WIN_PITCH_W];   /* buffer 0 of the one-warp layout */
    alignas(16) float t[2][4][TB_BLOCK];                /* luma, chroma                    */
    VlcScratch vlc;
    VlcTables tables;
    uint32_t best[2][TEAM_WARPS];                       /* each warp's key, two stages     */
    int32_t cost[3];                                    /* inter, filtered, intra          */
    uint32_t cbp[2];
};

/* SAD over source rows r0 .. r0 + N - 1 at one vector inside the window */
template <int N>
__device__ __forceinline__ uint32_t sad_rows(const StageBuf s, int vx, int vy, int r0)
{
    const int b = 16 + vx;
    const uint32_t *p = s.win(15 + vy + r0, b >> 2);
    const uint32_t sh = (uint32_t)(b & 3) * 8u;
    uint32_t a[2] = { 0u, 0u };
#pragma unroll
    for (int r = 0; r < N; r++) {
        uint32_t w[4];
        align16(p + r * WIN_PITCH_W, sh, w);
        a[r & 1] = sad16(cur_row(s, r0 + r), w, a[r & 1]);
    }
    return a[0] + a[1];
}

/* SADs of eight vectors one below the other from (vx, vy0) on: each window
 * row is aligned once for all of them */
[[maybe_unused]] __device__ __forceinline__ void sad_column8(const StageBuf s, int vx, int vy0, uint32_t sad[8])
{
    const int b = 16 + vx;
    const uint32_t *p = s.win(15 + vy0, b >> 2);
    const uint32_t sh = (uint32_t)(b & 3) * 8u;
#pragma unroll
    for (int k = 0; k < 8; k++)
        sad[k] = 0u;
#pragma unroll
    for (int R = 0; R < 23; R++) {
        uint32_t w[4];
        align16(p + R * WIN_PITCH_W, sh, w);
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (R - k >= 0 && R - k < 16)
                sad[k] = sad16(cur_row(s, R - k), w, sad[k]);
    }
}

/* the least of the team's keys */
[[maybe_unused]] __device__ __forceinline__ uint32_t team_min(TeamSmem &sm, int stage, uint32_t key, int tid)
{
    key = __reduce_min_sync(FULL, key);
    if ((tid & 31) == 0)
        sm.best[stage][tid >> 5] = key;
    __syncthreads();
    uint32_t m = sm.best[stage][0];
#pragma unroll
    for (int w = 1; w < TEAM_WARPS; w++)
        m = min(m, sm.best[stage][w]);
    return m;
}

/* the final vector of the search; the intra cost on the way (warp 3) */
template <bool FULL_SEARCH>
__device__ __forceinline__ void team_search(TeamSmem &sm, const StageBuf s, const h261b_session_dev_t &S, int mbx,
                                            int mby, int tid, int &vx, int &vy)
{
    const int lane = tid & 31, warp = tid >> 5;
    const int bx = mbx * 16, by = mby * 16;
    const int lminx = max(-15, -bx), lmaxx = min(15, (S.mbw - 1) * 16 - bx);
    const int lminy = max(-15, -by), lmaxy = min(15, (S.mbh - 1) * 16 - by);
    auto inside = [&](int x, int y) { return x >= lminx && x <= lmaxx && y >= lminy && y <= lmaxy; };
    if (FULL_SEARCH) {
        /* 31 columns by four groups of eight rows; the last starts at row 8,
         * which the group before holds too (a repeated key changes no minimum) */
        const int q = min(tid / 31, 3), tx = min(tid - 31 * q, 30), x = tx - 15, y0 = min(-15 + 8 * q, 8);
        uint32_t sad[8], best = FULL;
        sad_column8(s, x, y0, sad);
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (inside(x, y0 + k))
                best = min(best, (sad[k] << 10) | zorder((uint32_t)tx, (uint32_t)(y0 + k + 15)));
        if (warp == 3) {
            const int32_t c = intra_cost(s, lane);
            if (lane == 0)
                sm.cost[2] = c;
        }
        const uint32_t z = team_min(sm, 0, best, tid) & 1023u;
        vx = (int)compact8(z) - 15;
        vy = (int)compact8(z >> 1) - 15;
        return;
    }
    const int t = min(tid, 120), ty = t / 11, tx = t - 11 * ty;
    const int x = stage1_offset(tx), y = stage1_offset(ty);
    const uint32_t grid = sad_rows<16>(s, x, y, 0);
    const uint32_t coarse = team_min(sm, 0, inside(x, y) ? (grid << 10) | zorder((uint32_t)tx, (uint32_t)ty) : FULL,
                                     tid);
    const int v1x = stage1_offset((int)compact8(coarse & 1023u));
    const int v1y = stage1_offset((int)compact8((coarse & 1023u) >> 1));
    uint32_t best = (coarse & ~1023u) | zorder(3, 3);
    if (warp < 3) {
        const int c = tid >> 1, k = c + (c >= 24 ? 1 : 0), ry = k / 7, rx = k - 7 * ry;
        const int x1 = v1x + rx - 3, y1 = v1y + ry - 3;
        uint32_t sad = sad_rows<8>(s, min(max(x1, -15), 15), min(max(y1, -15), 15), 8 * (tid & 1));
        sad += __shfl_xor_sync(FULL, sad, 1);
        if (inside(x1, y1))
            best = min(best, (sad << 10) | zorder((uint32_t)rx, (uint32_t)ry));
    } else {
        const int32_t c = intra_cost(s, lane);
        if (lane == 0)
            sm.cost[2] = c;
    }
    const uint32_t z = team_min(sm, 1, best, tid) & 1023u;
    vx = v1x + (int)compact8(z) - 3;
    vy = v1y + (int)compact8(z >> 1) - 3;
}

/* one MB of picture S.  phases as in step_kernel, every warp of the CTA
 * together; mbs_done may be NULL. */
template <int FMAD, bool FULL_SEARCH, bool ABI, bool CODE>
__device__ __forceinline__ void team_mb(TeamSmem &sm, const h261b_session_dev_t &S, int mb, int phases,
                                        int32_t *mbs_done)
{
    const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (!H261B_CHECK(mb < S.mbw * S.mbh, CHK_WORK_ITEM, mb))
        return;
    const int mby = mb_row(mb, S.mbw), mbx = mb - mby * S.mbw;
    const int H = S.mbh * 16, x0 = mbx * 16, y0 = mby * 16;
    /* the window's 46 x 3 chunks, the 16 luma and the 16 chroma rows */
    for (int i = tid; i < 3 * WIN_ROWS + 32; i += TEAM_THREADS) {
        if (i < 3 * WIN_ROWS) {
            const int r = i / 3, j = i - 3 * r, x = x0 - 16 + 16 * j, y = y0 - 15 + r;
            bool ok = x >= 0 && x < S.mbw * 16 && y >= 0 && y < H;
            ok = ok && H261B_CHECK(x >= 0 && x + 16 <= S.mbw * 16, CHK_STAGE_WINDOW, x);
            cp_async16z(sm.buf + r * WIN_PITCH_W + 4 * j, ok ? S.ref_y + (size_t)y * S.pitch_y + x : S.ref_y, ok);
        } else if (i < 3 * WIN_ROWS + 16) {
            const int r = i - 3 * WIN_ROWS;
            if (H261B_CHECK(y0 + r < H && x0 + 16 <= S.mbw * 16, CHK_STAGE_SOURCE, y0 + r))
                cp_async16(sm.buf + r * WIN_PITCH_W + SRC_COL_W, S.cur_y + (size_t)(y0 + r) * S.pitch_y + x0);
        } else {
            const int q = i - 3 * WIN_ROWS - 16, r = q & 7;
            const uint8_t *src = q >> 3 ? S.cur_cr : S.cur_cb;
            if (H261B_CHECK(mby * 8 + r < S.mbh * 8 && mbx * 8 + 8 <= S.mbw * 8, CHK_STAGE_SOURCE, mby * 8 + r))
                cp_async8(sm.buf + (16 + q) * WIN_PITCH_W + SRC_COL_W,
                          src + (size_t)(mby * 8 + r) * S.pitch_c + mbx * 8);
        }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();

    const StageBuf b = stage_view(sm.buf, 0);
    const bool do_me = (phases & H261B_PHASE_ME) && !S.skip_search;
    const bool enc = (phases & H261B_PHASE_ENCDEC) && !(S.rc && (phases & H261B_PHASE_MD));
    me_gpu_mb_t me;
    me.i_intra_cost = me.i_zero_cost = me.i_16x16_cost = me.i_16x16_filter_cost = 0;
    me.s_16x16_mv.i8_mx = me.s_16x16_mv.i8_my = 0;
    ChromaRef ref = { 0u, 0u, 0u, 0u };
    if (do_me) {
        int vx, vy;
        team_search<FULL_SEARCH>(sm, b, S, mbx, mby, tid, vx, vy);
        me.s_16x16_mv.i8_mx = (int8_t)vx;
        me.s_16x16_mv.i8_my = (int8_t)vy;
        int32_t c = 0, unused = 0;
        if (warp == 0) {
            inter_costs<true, false>(b, vx, vy, lane, c, unused);
        } else if (warp == 1) {
            /* the chroma prediction's loads before the cost hides them */
            const MbDecision inter = { H261B_MB_TYPE_INTER, 0, vx, vy, 0 };
            if (enc)
                ref = chroma_ref(S, mbx, mby, inter, lane);
            inter_costs<false, true>(b, vx, vy, lane, unused, c);
        }
        if (warp < 2 && lane == 0)
            sm.cost[warp] = c;
        __syncthreads();
        me.i_16x16_cost = sm.cost[0];
        me.i_16x16_filter_cost = sm.cost[1];
        me.i_intra_cost = sm.cost[2];
        if (ABI && tid == 0)
            me_results_out(S, mb, me);
    } else if (phases & H261B_PHASE_MD) {
        me.i_intra_cost = intra_cost(b, lane);   /* every warp: no exchange */
    }

    MbDecision m;
    if (phases & H261B_PHASE_MD) {
        m = mode_decide(me, S.frame_type);
        if (tid == 0 && S.rc)
            atomicAdd(&S.rc->cost_sum, m.cost);
        if (tid == 0 && S.md_out) {
            h261_mb_mode_decision_t o;
            o.i_cost = m.cost;
            o.i_quantiser_adjust = 0;
            o.i_mb_type = m.type;
            o.i_mb_flags = m.flags;
            o.i_mv_x = m.mvx;
            o.i_mv_y = m.mvy;
            S.md_out[mb] = o;
        }
    } else {
        if (ABI && !enc)
            return;   /* the boundary's motion estimation alone */
        const h261_mb_mode_decision_t &d = S.md_in[mb];
        m.type = d.i_mb_type;
        m.flags = d.i_mb_flags;
        m.mvx = d.i_mv_x;
        m.mvy = d.i_mv_y;
        m.cost = d.i_cost;
        if (enc && warp == 1)
            ref = chroma_ref(S, mbx, mby, m, lane);
    }
    if (!enc)
        return;

    const int t = m.type == H261B_MB_TYPE_INTRA ? 0 : 1;
    if (t == 0)
        ref = ChromaRef{ 0u, 0u, 0u, 0u };   /* an intra MB's prediction is zero */
    int quant = S.rc ? S.rc->picture_quant : S.quant;
    if (!(phases & H261B_PHASE_MD))
        quant += S.md_in[mb].i_quantiser_adjust;
    quant = min(31, max(1, quant));
    if (warp < 2) {
        const float fwd_c = __fmul_rn(c_fwd_post[lane & 7], 0.125f), inv_c = c_inv_pre[lane & 7];
        const uint4 offw = *reinterpret_cast<const uint4 *>(&S.dn->offset[t][lane & 7][0]);
        float noise[8];
#pragma unroll
        for (int v = 0; v < 8; v++)
            noise[v] = 0.0f;
        uint32_t ssd = 0;
        const BlockRow row = warp == 0 ? luma_row(b, S, mbx, mby, m, lane) : chroma_row(b, S, mbx, mby, m, ref, lane);
        const uint32_t cbp = encdec_pass<FMAD, ABI, CODE>(sm.t[warp], sm.vlc.cm, row, S, mb, m, quant, offw,
                                                            warp == 0, lane, fwd_c, inv_c, noise, ssd);
        if (lane == 0)
            sm.cbp[warp] = cbp;
        add_noise(S.dn, t, noise, lane);
        if (S.ssd_out) {
            /* Y on warp 0; Cb on lanes 0-7, Cr on lanes 8-15 of warp 1 */
            const uint32_t e0 = __reduce_add_sync(FULL, warp == 0 || lane < 8 ? ssd : 0u);
            const uint32_t e1 = __reduce_add_sync(FULL, lane >= 8 && lane < 16 ? ssd : 0u);
            if (lane == 0) {
                atomicAdd(&S.ssd_out[warp], (unsigned long long)e0);
                if (warp == 1)
                    atomicAdd(&S.ssd_out[2], (unsigned long long)e1);
            }
        }
        __threadfence();   /* before the last warp counts the MB done */
    }
    __syncthreads();
    if (warp == 2) {
        const uint32_t cbp = sm.cbp[0] | sm.cbp[1];
        const int flags = m.flags | (cbp ? H261B_MB_COEFF : 0);
        int coef_bits = 0;
        if (CODE && S.bits_out) {
            const uint32_t blocks = t == 0 ? 63u : __brev(cbp) >> 26;
            if (blocks) {
                int oob = 0;
                const int pos = code_mb(blocks, t == 0, sm.tables, sm.vlc, lane, oob);
                coef_bits = store_mb_string(sm.vlc.stage, S.vlc_scratch + (size_t)mb * VLC_MB_WORDS, pos, oob, lane);
            }
        }
        if (lane == 0) {
            if (ABI && S.abi_out)
                abi_record_out(&S.abi_out[mb], m, flags, quant, cbp, mbx, mby);
            if (S.info_out) {
                h261b_mb_info_t inf;
                inf.type = (int16_t)m.type;
                inf.flags = (int16_t)flags;
                inf.quant = (int8_t)quant;
                inf.cbp = (int8_t)cbp;
                inf.mvx = (int8_t)m.mvx;
                inf.mvy = (int8_t)m.mvy;
                inf.cost = m.cost;
                inf.coef_bits = coef_bits;
                S.info_out[mb] = inf;
            }
            atomicAdd(&S.dn->count[t], 6);
        }
        __threadfence();
        __syncwarp();
        uint32_t last = 0;
        if (lane == 0) {
            last = atomicAdd(&S.dn->ticket, 1u) + 1u == (uint32_t)(S.mbw * S.mbh) ? 1u : 0u;
            if (mbs_done)
                atomicAdd(mbs_done, 1);
        }
        if (__shfl_sync(FULL, last, 0)) {
            __threadfence();
            denoise_frame_end(S.dn, lane);
        }
    }
}

template <bool CODE>
__device__ __forceinline__ void team_begin(TeamSmem &sm)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (CODE) {
        load_vlc_tables(sm.tables, (int)threadIdx.x, TEAM_THREADS);
        for (int i = (int)threadIdx.x; i < VLC_MB_WORDS; i += TEAM_THREADS)
            sm.vlc.stage[i] = 0u;
    }
}

/* a work item per CTA */
template <int FMAD, bool FULL_SEARCH, bool CODE>
__global__ void __launch_bounds__(TEAM_THREADS, 4)
    team_kernel(const h261b_session_dev_t *__restrict__ sessions, const uint32_t *__restrict__ work, int32_t phases)
{
    __shared__ TeamSmem sm;
    team_begin<CODE>(sm);
    const uint32_t item = work[blockIdx.x];
    const h261b_session_dev_t &S = sessions[item >> 12];
    team_mb<FMAD, FULL_SEARCH, false, CODE>(sm, S, (int)(item & 0xFFFu), phases, const_cast<int32_t *>(&S.mbs_done));
}

/* MB blockIdx.x of one picture whose descriptor comes with the launch */
template <int FMAD, bool FULL_SEARCH, bool ABI>
__global__ void __launch_bounds__(TEAM_THREADS, 4)
    team_picture_kernel(const __grid_constant__ h261b_session_dev_t S, int32_t phases)
{
    __shared__ TeamSmem sm;
    team_begin<false>(sm);
    team_mb<FMAD, FULL_SEARCH, ABI, false>(sm, S, (int)blockIdx.x, phases, nullptr);
}

} // namespace

namespace {

constexpr int PART_FMAD = (H261B_PART >> 2) & 1;
constexpr bool PART_FULL = ((H261B_PART >> 1) & 1) != 0, PART_BULK = (H261B_PART & 1) != 0;

/* the instantiation of a launch's flags: the encode kind has no search and
 * writes no reference-layout output, the search kind no encode output */
template <bool CODE>
StepFn step_of(int kind)
{
    if constexpr (!PART_FULL)
        if (kind == KIND_ENCODE)
            return step_kernel<PART_FMAD, KIND_ENCODE, false, false, PART_BULK, CODE>;
    return kind == KIND_FULL ? step_kernel<PART_FMAD, KIND_FULL, PART_FULL, false, PART_BULK, CODE>
                             : step_kernel<PART_FMAD, KIND_FUSED, PART_FULL, false, PART_BULK, CODE>;
}

StepFn part_step(int kind, int abi, int code)
{
    if (kind == KIND_SEARCH)
        return step_kernel<PART_FMAD, KIND_SEARCH, PART_FULL, false, PART_BULK, false>;
#if !(H261B_PART & 1)
    if (abi && kind != KIND_ENCODE)
        return step_kernel<PART_FMAD, KIND_FUSED, PART_FULL, true, false, false>;
#else
    (void)abi;
#endif
    return code ? step_of<true>(kind) : step_of<false>(kind);
}

#if H261B_PART & 1
/* (bulk staging: no team kernels) */
TeamFn part_team(int) { return nullptr; }
TeamPictureFn part_team_picture(int) { return nullptr; }
#else
TeamFn part_team(int code)
{
    return code ? team_kernel<PART_FMAD, PART_FULL, true> : team_kernel<PART_FMAD, PART_FULL, false>;
}

TeamPictureFn part_team_picture(int abi)
{
    return abi ? team_picture_kernel<PART_FMAD, PART_FULL, true> : team_picture_kernel<PART_FMAD, PART_FULL, false>;
}
#endif

int part_checks(unsigned long long *n, int first[2])
{
    *n = 0;
#ifdef H261B_DEBUG_CHECKS
    const unsigned long long zero = 0;
    if (cudaMemcpyFromSymbol(n, g_check_count, sizeof(*n)) != cudaSuccess ||
        cudaMemcpyFromSymbol(first, g_check_first, 2 * sizeof(int)) != cudaSuccess ||
        cudaMemcpyToSymbol(g_check_count, &zero, sizeof(zero)) != cudaSuccess)
        return H261B_ERR_CUDA;
#else
    (void)first;
#endif
    return H261B_OK;
}

int part_timeouts(unsigned int *n)
{
    const unsigned int zero = 0;
    if (cudaMemcpyFromSymbol(n, g_stage_timeouts, sizeof(*n)) != cudaSuccess ||
        cudaMemcpyToSymbol(g_stage_timeouts, &zero, sizeof(zero)) != cudaSuccess)
        return H261B_ERR_CUDA;
    return H261B_OK;
}

} // namespace

#define PART_NAME2(n) kernel_part_##n
#define PART_NAME(n) PART_NAME2(n)
namespace h261b {
const KernelPart PART_NAME(H261B_PART) = {
    part_step, part_team, part_team_picture, part_checks, part_timeouts,
    kSearchWarpBytes, kEncodeWarpBytes, sizeof(WarpSmem), sizeof(VlcTables),
};
}
