// Q4_0 MUL_MAT for a batch of activation columns on the 5th-generation tensor cores, with the block scales folded into the
// operands so that one accumulator in tensor memory runs over K.
//
// lm_ggml_compute_forward_mul_mat (cactus/ggml-cpu/ggml-cpu.c:1257-1449) computes, per output value,
// sum over blocks b of d_w[row, b] * d_a[col, b] * dot_b with dot_b an integer.  Scaling after every block (mmq.cu) costs a
// pass over the accumulator tile per 32 values of K; here the scales go into the operands instead:
//   A[row, k] = d_w[row, b] * q[row, k]      (15 significant bits: 11 of the fp16 scale and the quant)
//   B[col, k] = d_a[col, b] * a[col, k]      (19 significant bits)
// Each is an fp16 value plus the exact fp16 remainder (x_hi = rn(x), x_lo = x - x_hi; d is a multiple of 2^-24, so the
// remainder always fits), and the product is A_hi B_hi + A_hi B_lo + A_lo B_hi (the missing A_lo B_lo is below 2^-22 of a
// term), accumulated in fp32 by tcgen05.mma.kind::f16.  The tensor core truncates when it accumulates, so a sum over many
// MMAs drifts towards zero: 2.1e-6 to 2.4e-6 rms against f64 when the accumulator ran over 16 block groups, ten times the
// error of the mma.sync kernel (0.9e-7 to 3.8e-7).  Hence it is emptied after every block group (8 MMAs) and the block groups
// are added in registers, rounding to nearest: 2.0e-7 to 2.5e-7 for K 1024 - 14336 (two block groups: 3.4e-7).  The small
// terms (A_hi B_lo, A_lo B_hi), 2^-11 of the others, have columns of their own and are emptied once per tile.
// A value beyond the fp16 range (|d q| > 65504) makes the sum non-finite; such results are recomputed exactly from the
// integers (tc_exact_value).
//
// What bounds it: issuing the MMAs.  128 x 128 x 16 + 128 x 64 x 16 per 16 values of K take 96 clk (measured: N / 2 clk per
// MMA), a block group of 256 rows x 64 columns x 128 values 1542 clk; but an issuing warp needs about as long for its
// 17 MMAs, three waits and two commits beside six busy warps on its scheduler, and the accumulator has to be read in between.
// 4096 x 28672 at 512 columns: 298 us (296 to 316 by run; 265 with 16 block groups per accumulator; mma.sync 321 to 324).  A CTA needs about
// 5 us to fill and empty its pipeline.  What is around the MMAs has to stay below that:
//   * the activations arrive as B_hi / B_lo planes written once by the quantiser (act_dims: b_offset) in the core-matrix
//     order of the MMA's B descriptor.  A CTA owns 256 weight rows (two MMA row tiles) per activation copy: 50 KB per
//     block group, 33 B/clk per SM, below the 40 B/clk that bulk copies out of L2 reach with all SMs at it.  One copy brings
//     all of it (a bulk copy costs its thread 75 clk, so 2 KB pieces bounded an earlier form);
//   * the weights are turned into fp16 in registers and go straight into tensor memory (the MMA's A operand): three half2
//     operations (2 clk each on this GPU) and 1.5 logic operations per pair of values, 768 clk per block group.  T16 tiles are
//     in MMA fragment order, which is what tcgen05.st.16x128b takes: lane (g, t) stores the words of rows g and g + 8 as it
//     loaded them, so there is no transposition; the order of K within a block that follows from it is the order the
//     quantiser writes B in;
//   * every hand-over between warps is some twenty instructions at 10-16 clk each beside busy warps, so there are few: one per
//     half block group and role, with an A stage for each team of weight warps;
//   * a block group's sums are read by 8 warps with 64 registers of sums a thread (setmaxnreg moves them from the other warps): with
//     the sums in shared memory and 4 warps, emptying after every block group cost 423 us instead of 298.
//
// Roles of a CTA (one per SM, 28 warps): warps 0 and 1 issue the MMAs of one row tile each, warp 2 the copies (a ring of
// stages of one block group), two teams of 8 warps convert weights (they take the half block groups in turn; a
// warp: 32 rows), the last eight warps, four per row tile, add up the accumulators and write results.  The two row tiles share
// the copies only: each has its own A stages, accumulator and barriers.  Code that runs once per tile is kept small and in
// loops: with 172 KB of (unrolled) code the kernel spent most of its time on instruction cache misses.  (All of it is
// inlined all the same: ptxas gives a warp the registers that setmaxnreg sets only where nothing is called.)
//
// Work split (TcPlan): clusters of up to 8 CTAs share the K range of one tile (256 rows x <= 64 columns) and add their parts
// through distributed shared memory in rank order; or, when there are many tiles, one CTA per SM takes an equal and
// contiguous share of all (tile, block group) iterations, and a tile that two or three CTAs share is added by the CTA that
// arrives last, in K order (parts parked in the workspace; a counter per tile), so sums do not depend on timing.
//
// Measured against the mma.sync kernel: the table at use_tc (mul_mat.cu).
// Every wait is bounded; on time-out the CTA raises b200_kernel_status, all roles fall through, the producer waits
// (bounded) for its copies in flight, the issuing warp for its MMAs, the CTA frees its tensor memory and returns.
#include <cuda.h>
#include <cuda_fp16.h>

#include <atomic>
#include <chrono>
#include <cstdlib>
#include <mutex>
#include <unordered_map>

#include "common.cuh"

namespace b200 {

__device__ int g_tc_error = 0;                    // non-zero after a bounded wait gave up
__device__ unsigned g_tc_spin_limit = 1u << 20;   // try_wait rounds before a wait gives up (each may suspend for a while)
constexpr uint32_t TC_DRAIN_LIMIT = 1u << 22;     // what a CTA that gave up still waits for: its own copies and MMAs in flight

constexpr int TC_RT = 16;            // 16-row tiles of a CTA at most: 256 rows, two MMA row tiles
constexpr int TC_EPI_THREADS = 256;

// Geometry.  A CTA has up to NT tiles of 8 activation columns.
struct TcCfg {
    static constexpr int NT = 8;
    static constexpr int WT = 1024;                                    // one row tile, one block group
    static constexpr int OFF_S = TC_RT * WT;                           // its scales: 128 bytes per row tile
    static constexpr int OFF_B = OFF_S + TC_RT * 128;                  // B_hi: 2 KB per column tile, then B_lo
    static constexpr int STAGE = OFF_B + NT * 4096;
    static constexpr int ACC = NT * 8 * 1024;                          // partial results, f32 [column][256 rows]
    static constexpr int FIT = (232448 - 6144 - ACC) / STAGE;
    static constexpr int STAGES = FIT > 8 ? 8 : FIT;
    // tensor memory of row tile mt: an accumulator of 2 x 8 NT columns (hi | small terms) at mt * D_MT, ABUF A stages of half a block
    // group (32 columns of A_hi, 32 of A_lo) at A_COL + mt * A_MT
    static constexpr int D_MT = 16 * NT;
    static constexpr int ABUF = 2;
    static constexpr int A_MT = ABUF * 64, A_COL = 512 - 2 * A_MT;
    // warps: 4 for MMAs and copies, a team of 8 weight warps per A stage (each waits for its own stage phase after phase, which a
    // parity wait can tell apart), 4 for the write-back
    static constexpr int WARP_EPI = 4 + 8 * ABUF, THREADS = 32 * (WARP_EPI + 8);
    // barriers: FULL a stage has landed; WREAD its weights are in registers; DONE (per row tile) all MMAs on it are complete; AFULL
    // (row tile, A stage); AFREE the first A stage of a row tile may be written again (the second: DONE); ACCE the accumulator
    // has been read (that it is complete: DONE).  A commit costs its warp 45 clk, hence no barrier of its own where one tells already.
    static constexpr int B_FULL = 0, B_WREAD = STAGES, B_DONE = 2 * STAGES, B_AFULL = 4 * STAGES, B_AFREE = B_AFULL + 2 * ABUF, B_ACCE = B_AFREE + 2,
                         B_DRAIN = B_ACCE + 2, N_BARS = B_DRAIN + 2;
    static constexpr int OFF_ACC = STAGES * STAGE;
    static constexpr int BAR_OFFSET = OFF_ACC + ACC;
    static constexpr int SH_OFFSET = BAR_OFFSET + (N_BARS * 8 + 15) / 16 * 16;   // TcShared
    static constexpr int SMEM = SH_OFFSET + 5120;
    static_assert(STAGE % 1024 == 0 && SMEM <= 232448 && 2 * D_MT <= A_COL && STAGES >= 2, "shared / tensor memory of an SM");
};

// How the iterations are dealt out (see the head comment).
struct TcPlan {
    int rt_per_group;   // row tiles of a CTA: 16 or 8
    int groups, chunks; // row groups, column chunks; tile = group * chunks + chunk
    int cs;             // > 0: clusters of cs CTAs, one tile per cluster; 0: equal shares over gridDim.x CTAs
    unsigned long long launch_id;   // equal shares: marks the arrival counters (56 bits)
    uint32_t share, extra;   // equal shares: CTA j takes share iterations, one more if j < extra
    int debug;          // tests of the give-up path: 32 no producer copies anything, 64 those of odd CTAs, 128 one write-back warp gives up
};
// The weights as tensor maps: 1 KB tiles and 128-byte scale tiles of one block group, 8 row tiles (128 rows) per copy.
struct TcMaps {
    CUtensorMap q, s;
};

__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t) ((addr >> 4) & 0x3FFF) | ((uint64_t) ((lbo >> 4) & 0x3FFF) << 16) | ((uint64_t) ((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}
__device__ __forceinline__ bool tc_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// One lane of a converged warp.  What is issued under this predicate takes its operands from uniform registers: 22 clk per
// tcgen05.mma and 45 per commit, against 56 and 120 behind a lane number compare (measured; 75 against 107 beside busy warps).
__device__ __forceinline__ bool tc_elect() {
    uint32_t el;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(el));
    return el != 0;
}
// Bounded wait of a whole (converged) warp; false = gave up (or the CTA already gave up elsewhere).  The outcome is one for
// the warp, by vote: what follows a wait (elect.sync, tcgen05.ld) needs all its lanes.
__device__ __forceinline__ bool tc_wait_slow(uint32_t bar, uint32_t parity, volatile int *abort_flag, uint32_t limit) {
#pragma unroll 1
    for (uint32_t i = 0; i < limit; ++i) {
        if (__all_sync(0xffffffffu, tc_try(bar, parity))) return true;
        if ((i & 15u) == 15u && __any_sync(0xffffffffu, *abort_flag)) return false;
    }
    *abort_flag = 1;
    atomicExch(&g_tc_error, 1);
    return false;
}
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, uint32_t limit) {
    return __all_sync(0xffffffffu, tc_try(bar, parity)) || tc_wait_slow(bar, parity, abort_flag, limit);
}
__device__ __forceinline__ void tc_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_tma_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_copy(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem], M 128, K 16, fp16 x fp16 -> f32; N comes with the instruction descriptor.  B's descriptor in two
// halves: only the low one moves, and a 64-bit addition would be two instructions beside every MMA.
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint32_t a_tmem, uint32_t bdesc_lo, uint32_t bdesc_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\n.reg .b64 b;\nsetp.ne.b32 p, %5, 0;\nmov.b64 b, {%2, %3};\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n}\n"
                 ::"r"(d_tmem), "r"(a_tmem), "r"(bdesc_lo), "r"(bdesc_hi), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ uint32_t tc_h2(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
__device__ __forceinline__ __half2 tc_as_h2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }
// 16 tensor-memory lanes x 16 columns: register 2c = (row g, column 4c + t), 2c + 1 = (row g + 8, column 4c + t)
__device__ __forceinline__ void tc_st_16x128b_x4(uint32_t taddr, const uint32_t (&a)[8]) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n"
                 ::"r"(taddr), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]) : "memory");
}
__device__ __forceinline__ void tc_ld_x16(uint32_t (&r)[16], uint32_t taddr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
}
// sum[k] += column k of the thread's row, k < cols (16, 32, 48 or 64); `read` is called once all have been read
template <typename F>
__device__ __forceinline__ void tc_add_columns(float (&sum)[64], uint32_t taddr, uint32_t cols, F read) {
    uint32_t u[2][16];
#pragma unroll
    for (int c = 0; c < 4; c += 2) {
        if (c * 16 >= (int) cols) break;
        tc_ld_x16(u[0], taddr + c * 16);
        if ((c + 1) * 16 < (int) cols) tc_ld_x16(u[1], taddr + (c + 1) * 16);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        if ((c + 2) * 16 >= (int) cols) read();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if ((c + h) * 16 >= (int) cols) break;
#pragma unroll
            for (int k = 0; k < 16; k += 2)
                asm("{\n.reg .b64 x, y;\nmov.b64 x, {%0, %1};\nmov.b64 y, {%2, %3};\nadd.rn.f32x2 x, x, y;\nmov.b64 {%0, %1}, x;\n}\n"
                    : "+f"(sum[(c + h) * 16 + k]), "+f"(sum[(c + h) * 16 + k + 1]) : "r"(u[h][k]), "r"(u[h][k + 1]));
        }
    }
}

// A piece of work: block groups [bg, bg + len) of a tile (row group x column chunk).
struct TcPiece {
    uint32_t tile, group, chunk, bg, len;
    uint32_t two;            // more than 128 rows: the second MMA row tile is in use
    uint32_t slot0, parts;   // equal shares: where the tile's first part is parked (the others: slot 2j of the CTAs that follow), how many
};
constexpr int TC_MAX_PIECES = 128;

// What the write-back needs of the launch and the CTA's share of the work, in shared memory.  All of it is worked out once, by
// one thread, while the first copies are on their way: code that every role repeats costs instruction cache misses.
struct TcShared {
    TiledDims dims;
    ActDims act;
    TcPlan plan;
    const uint8_t *w, *aq;
    float *dst;
    int64_t dst_nb_row;
    unsigned long long *counters;   // per tile {launch id, arrivals}
    float4 *slots;                  // parked parts
    uint32_t slot_n;                // float4s of one
    uint32_t tmem;
    int abort_flag, flag;
    int wb_gave_up;                 // a write-back warp gave up
    uint32_t n_pieces, n_iter;
    uint32_t n_finished;            // pieces that tc_finish has been through
    TcPiece piece[TC_MAX_PIECES];
};

static_assert(sizeof(TcShared) <= 5120, "TcShared has its place in TcCfg");

// One result from the integers themselves: what the reference computes, block by block.  Only for values whose folded
// operands left the fp16 range.
__device__ __forceinline__ float tc_exact_value(const TcShared *o, int row, int col) {
    const uint8_t *wq = o->w, *ws = wq + o->dims.qs_bytes;
    const int rt = row >> 4, r = row & 15, g = r & 7, h = r >> 3;
    float sum = 0.0f;
#pragma unroll 1
    for (int b = 0; b < (int) o->dims.nb; ++b) {
        const int64_t at = (int64_t) rt * o->dims.n_bg + (b >> 2);
        const int j = b & 3;
        const uint2 *a = reinterpret_cast<const uint2 *>(o->aq + ((col >> 3) * o->act.nbp + b) * 256) + (col & 7) * 4;
        int dot = 0;
#pragma unroll 1
        for (int t = 0; t < 4; ++t) {
            const uint32_t word = reinterpret_cast<const uint32_t *>(wq + at * 1024 + (g * 4 + t) * 32)[h * 4 + j];
            dot = __dp4a((int) ((word << 4) & 0xF0F0F0F0u), (int) a[t].x, dot);
            dot = __dp4a((int) (word & 0xF0F0F0F0u), (int) a[t].y, dot);
        }
        const float dw = __half2float(reinterpret_cast<const __half *>(ws)[at * 64 + r * 4 + j]) * 0.0625f;
        const float da = reinterpret_cast<const float *>(o->aq + o->act.d_offset)[((col >> 3) * o->act.n_bg + (b >> 2)) * 64 + act_scale_index(j, col & 7)];
        sum = fmaf(dw * da, (float) dot, sum);
    }
    return sum;
}

// Equal shares: CTA j takes iterations [first_of(j), first_of(j + 1)) of [tile][block group].  A share that ends inside a tile
// starts with that last piece: the CTA that completes the tile then finds it parked long before.  CTA j parks a piece that
// starts where its share starts in slot 2j, the piece its share ends with in slot 2j + 1.
__device__ __forceinline__ uint32_t tc_first_of(const TcPlan &p, uint32_t j) { return j * p.share + min(j, p.extra); }
__device__ __forceinline__ uint32_t tc_cta_of(const TcPlan &p, uint32_t it) {   // the CTA that holds iteration `it`
    const uint32_t big = p.extra * (p.share + 1);
    return it < big ? it / (p.share + 1) : p.extra + (it - big) / p.share;
}
__device__ __forceinline__ void tc_share(TcShared *o, const TcPlan plan, uint32_t n_bg, uint32_t n_rt) {
    uint32_t it0, it1;
    if (plan.cs > 0) {   // the CTAs of a cluster cut the K range of one tile
        const uint32_t cs = (uint32_t) plan.cs, rank = blockIdx.x % cs, tile = blockIdx.x / cs * n_bg;
        it0 = tile + rank * n_bg / cs;
        it1 = tile + (rank + 1) * n_bg / cs;
    } else {
        it0 = tc_first_of(plan, blockIdx.x);
        it1 = tc_first_of(plan, blockIdx.x + 1);
    }
    uint32_t n = 0, tile = it0 / n_bg, at = it0;
    const uint32_t tile_h = it1 / n_bg, head = tile_h * n_bg > it0 ? it1 - tile_h * n_bg : 0u;
    o->n_iter = it1 - it0;
    if (head > 0) { at = tile_h * n_bg; tile = tile_h; }
#pragma unroll 1
    while (it1 > it0) {
        TcPiece &q = o->piece[n++];
        q.tile = tile;
        q.group = tile / (uint32_t) plan.chunks;
        q.chunk = tile - q.group * (uint32_t) plan.chunks;
        q.bg = at - tile * n_bg;
        q.len = min(it1 - at, n_bg - q.bg);
        q.two = n_rt - q.group * (uint32_t) plan.rt_per_group > 8 && plan.rt_per_group > 8 ? 1u : 0u;
        q.parts = 1;
        q.slot0 = 0;
        if (plan.cs == 0 && q.len < n_bg) {
            const uint32_t first = tc_cta_of(plan, tile * n_bg);
            q.parts = tc_cta_of(plan, tile * n_bg + n_bg - 1) - first + 1;
            q.slot0 = 2 * first + (tc_first_of(plan, first) < tile * n_bg ? 1u : 0u);
        }
        if (n == 1 && head > 0) { at = it0; tile = it0 / n_bg; it1 -= head; }   // on to the start of the share
        else { at += q.len; ++tile; if (at >= it1) break; }
    }
    o->n_pieces = n;
}

// Values that do not simply go to 16 aligned bytes: a ragged or unaligned edge, or not finite
__device__ __forceinline__ void tc_write_slow(const TcShared *o, int row, int row_end, int col, float4 f) {
#pragma unroll 1
    for (int i = 0; i < 4 && row + i < row_end; ++i) {
        float y = i == 0 ? f.x : i == 1 ? f.y : i == 2 ? f.z : f.w;
        if (!isfinite(y)) y = tc_exact_value(o, row + i, col);
        *reinterpret_cast<float *>(reinterpret_cast<char *>(o->dst) + col * o->dst_nb_row + (int64_t) (row + i) * 4) = y;
    }
}
// Where a thread's share of a tile goes: elements e0, e0 + step, ... of [column][256 rows / 4]; step is a multiple of 64, so the
// rows stay the same and the column moves.
struct TcOut {
    char *to;
    int64_t inc;
    int row, row_end, col, col_inc, col_end;
    bool vec;
    __device__ __forceinline__ TcOut(const TcShared *o, const TcPiece &q, uint32_t e0, uint32_t step) {
        row = (int) q.group * o->plan.rt_per_group * 16 + (int) (e0 & 63) * 4;
        row_end = min((int) o->dims.M, ((int) q.group + 1) * o->plan.rt_per_group * 16);
        col = (int) q.chunk * o->act.chunk_nt * 8 + (int) (e0 >> 6);
        col_inc = (int) (step >> 6);
        col_end = row < row_end ? (int) o->act.N : 0;
        const int64_t nb = o->dst_nb_row;
        inc = col_inc * nb;
        to = reinterpret_cast<char *>(o->dst) + col * nb + (int64_t) row * 4;
        vec = row + 3 < row_end && ((reinterpret_cast<uintptr_t>(to) | (uintptr_t) nb) & 15) == 0;
    }
        __device__ __forceinline__ void put(const TcShared *o, float4 v) {
        if (vec && isfinite((v.x + v.y) + (v.z + v.w))) *reinterpret_cast<float4 *>(to) = v;
        else tc_write_slow(o, row, row_end, col, v);
        to += inc;
        col += col_inc;
    }
};
__device__ __forceinline__ float4 tc_lds4(uint32_t at) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at));
    return v;
}

// The tile's parts lie in the shared memory of the cluster's CTAs: this CTA adds slice `rank` of the columns in rank order.
__device__ __forceinline__ void tc_write_cluster(const TcShared *o, uint32_t acc_u32, uint32_t te, uint32_t threads) {
    const uint32_t cs = (uint32_t) o->plan.cs, rank = blockIdx.x % cs, per4 = ((uint32_t) o->act.chunk_nt * 8 + cs - 1) / cs * 64;
    const uint32_t end = min((uint32_t) o->act.chunk_nt * 512, (rank + 1) * per4);
    uint32_t e = rank * per4 + te;
    TcOut out(o, o->piece[0], e, threads);
#pragma unroll 1
    for (; e < end && out.col < out.col_end; e += threads) {
        float4 x[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {   // all in flight at once
            uint32_t remote;
            x[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k < cs) {
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(acc_u32 + e * 16u), "r"(k));
                asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(x[k].x), "=f"(x[k].y), "=f"(x[k].z), "=f"(x[k].w) : "r"(remote));
            }
        }
#pragma unroll
        for (uint32_t k = 1; k < 8; ++k) { x[0].x += x[k].x; x[0].y += x[k].y; x[0].z += x[k].z; x[0].w += x[k].w; }
        out.put(o, x[0]);
    }
}

// Arrival of a part at its tile; true: it is the last one and all parts are there.  A tile's counter is {launch id, parts given up
// (4 bits), arrivals (4 bits)}; a word without this launch's id counts as zero, so the workspace needs no clearing.  Every CTA
// arrives exactly once for every piece it shares, with its part parked or given up, and the last to arrive leaves the
// counter zero: a replay of a graph comes with the same id and must find nothing of an earlier one.
__device__ __forceinline__ bool tc_arrive_tile(const TcShared *o, const TcPiece &q, bool gave_up) {
    const unsigned long long id = o->plan.launch_id << 8;
    unsigned long long *const arrived = o->counters + q.tile;
    unsigned long long old = *reinterpret_cast<volatile unsigned long long *>(arrived), seen, now;
    do {
        seen = old;
        now = ((seen ^ id) < 256 ? seen : id) + (gave_up ? 17 : 1);
        old = atomicCAS(arrived, seen, (now & 15) == q.parts ? 0ull : now);
    } while (old != seen);
    return (now & 255) == q.parts;
}
// The pieces of a CTA that gave up.  One thread, after everything else.
__device__ __forceinline__ void tc_give_up_pieces(const TcShared *o) {
#pragma unroll 1
    for (uint32_t p = o->n_finished; p < o->n_pieces; ++p)
        if (o->piece[p].parts > 1) tc_arrive_tile(o, o->piece[p], true);
}

// Piece q is complete in shared memory: write the tile if this is all of it or the last part to arrive, else park it.  Called by
// `threads` threads, te = 0 ..., which meet at barrier `bar`.  The parts (at most three) are added in K order whoever does it.
__device__ __forceinline__ void tc_finish(TcShared *o, uint32_t acc_u32, uint32_t piece, uint32_t te, uint32_t threads, uint32_t bar) {
    const TcPiece q = o->piece[piece];
    const uint32_t total4 = (uint32_t) o->act.chunk_nt * 512;
    volatile int *const flag = &o->flag;
    const uint32_t own = q.parts == 1 ? 0u : blockIdx.x - (q.slot0 >> 1);
    bool write = true;
    const float4 *at[3];
#pragma unroll
    for (uint32_t k = 0; k < 3; ++k) at[k] = k < q.parts && k != own ? o->slots + (size_t) (k == 0 ? q.slot0 : (q.slot0 & ~1u) + 2 * k) * o->slot_n : nullptr;
    if (q.parts > 1) {
        if (te == 0) {   // every other part parked already: nothing of this one has to go through memory
            unsigned long long *const arrived = o->counters + q.tile;
            unsigned long long seen;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(seen) : "l"(arrived) : "memory");
            *flag = seen == (o->plan.launch_id << 8) + q.parts - 1;
            if (*flag) *arrived = 0;   // nobody else is to come
        }
        asm volatile("bar.sync %0, %1;\n" ::"r"(bar), "r"(threads) : "memory");
        write = *flag != 0;
        if (!write) {
            float4 *to = o->slots + (size_t) (own == 0 ? q.slot0 : 2 * blockIdx.x) * o->slot_n;
#pragma unroll 1
            for (uint32_t e = te; e < total4; e += threads) {
                __stcg(to + e, tc_lds4(acc_u32 + e * 16u));
            }
            __threadfence();
            asm volatile("bar.sync %0, %1;\n" ::"r"(bar), "r"(threads) : "memory");
            if (te == 0) {
                *flag = tc_arrive_tile(o, q, false);
                __threadfence();
            }
            asm volatile("bar.sync %0, %1;\n" ::"r"(bar), "r"(threads) : "memory");
            write = *flag != 0;
        }
    }
    if (te == 0) o->n_finished = piece + 1;
    if (write) {
        TcOut out(o, q, te, threads);
#pragma unroll 1
        for (uint32_t e = te; e < total4 && out.col < out.col_end; e += threads) {
            float4 x[3];
#pragma unroll
            for (uint32_t k = 0; k < 3; ++k) {   // in flight together
                x[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (at[k]) x[k] = __ldcg(at[k] + e);
                else if (k == own) x[k] = tc_lds4(acc_u32 + e * 16u);
            }
            out.put(o, make_float4(x[0].x + x[1].x + x[2].x, x[0].y + x[1].y + x[2].y, x[0].z + x[1].z + x[2].z, x[0].w + x[1].w + x[2].w));
        }
    }
    asm volatile("bar.sync %0, %1;\n" ::"r"(bar), "r"(threads) : "memory");   // the partial results are free again
}

__global__ void __launch_bounds__(TcCfg::THREADS, 1) mmq_tc_kernel(TiledDims dims, const uint8_t *__restrict__ w, ActDims act, const uint8_t *__restrict__ aq,
                                                              float *__restrict__ dst, int64_t dst_nb_row, void *__restrict__ workspace, TcPlan plan,
                                                              const __grid_constant__ TcMaps maps) {
    using C = TcCfg;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t smem_u32 = (uint32_t) __cvta_generic_to_shared(smem);
    const uint32_t bars = smem_u32 + C::BAR_OFFSET;
    TcShared *const sh = reinterpret_cast<TcShared *>(smem + C::SH_OFFSET);
    volatile int *const abort_flag = &sh->abort_flag;
    volatile int *const wb_gave_up = &sh->wb_gave_up;
    float *const acc_s = reinterpret_cast<float *>(smem + C::OFF_ACC);
    const uint32_t acc_u32 = smem_u32 + C::OFF_ACC;
#define BAR(which, i) (bars + 8u * (uint32_t) ((which) + (i)))
    const uint32_t n_bg = (uint32_t) dims.n_bg;
    const uint32_t spin_limit = g_tc_spin_limit;

    if (tid == 96) {   // warp 3 has no role of its own
        sh->dims = dims;
        sh->act = act;
        sh->plan = plan;
        sh->w = w; sh->aq = aq; sh->dst = dst; sh->dst_nb_row = dst_nb_row;
        sh->counters = reinterpret_cast<unsigned long long *>(workspace);
        sh->slots = reinterpret_cast<float4 *>(reinterpret_cast<char *>(workspace) + ((size_t) plan.groups * plan.chunks * 8 + 255) / 256 * 256);
        sh->slot_n = (uint32_t) act.chunk_nt * 512;
    }
    if (tid == 64) {
        sh->abort_flag = 0;
        sh->wb_gave_up = 0;
        sh->n_finished = 0;
        tc_share(sh, plan, n_bg, (uint32_t) dims.n_rt);
    }
    if (tid < C::N_BARS) {
        const int i = tid;
        const int count = (i >= C::B_WREAD && i < C::B_DONE) ? 16
                        : (i >= C::B_AFULL && i < C::B_AFREE) || (i >= C::B_ACCE && i < C::B_DRAIN) ? 4 : 1;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(BAR(0, i)), "r"(count));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {   // all 512 columns (the CTA is alone on its SM)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"((uint32_t) __cvta_generic_to_shared(&sh->tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = sh->tmem;
    pdl_prologue();   // everything above touches no global memory

    // Registers: 72 a thread at launch (504 for a lane of the seven warpgroups), 40 + 4 x 56 + 2 x 120 = 504 while the roles run.
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;\n");
        if (warp < 2) {
            // ---------------- MMA issue for row tile mt = warp ----------------
            const uint32_t mt = (uint32_t) warp, nt = (uint32_t) act.chunk_nt;
            const uint32_t idesc_wide = (1u << 4) | (2 * nt << 17) | (8u << 24), idesc_hi = (1u << 4) | (nt << 17) | (8u << 24);   // f16 x f16 -> f32, K-major both, M 128
            const uint32_t d = tmem + mt * C::D_MT, d_small = d + 8 * nt, a0 = tmem + C::A_COL + mt * C::A_MT;
            const uint64_t bdesc0 = tc_smem_desc(smem_u32 + C::OFF_B, 128, 2048);
            const uint32_t b_hi = (uint32_t) (bdesc0 >> 32);
            uint32_t s = 0, acc_par = 1, a_par = 0;
            bool ok = true;
#pragma unroll 1
            for (uint32_t p = 0; p < sh->n_pieces && ok; ++p) {
                const bool active = mt == 0 || sh->piece[p].two;
                const uint32_t len = sh->piece[p].len;
#pragma unroll 1
                for (uint32_t i = 0; i < len && ok; ++i, a_par ^= 1) {
                    // (that the stage has landed follows from AFULL: the weight warps waited for it)
                    const uint32_t b = (uint32_t) bdesc0 + s * (C::STAGE >> 4);
                    if (i == 0) ok = tc_wait(BAR(C::B_ACCE, mt), acc_par, abort_flag, spin_limit);
                    ok = ok && tc_wait(BAR(C::B_AFULL, C::ABUF * mt), a_par, abort_flag, spin_limit);
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    if (i > 0) {   // the large terms start from zero, once what they were has been read; the small ones go on meanwhile
                        if (tc_elect() && ok && active) {
#pragma unroll
                            for (uint32_t k = 0; k < 4; ++k) tc_mma(d_small, a0 + 8 * k + 32, b + k * 16, b_hi, idesc_hi, 1u);
                            tc_mma(d_small, a0, b + nt * 128, b_hi, idesc_hi, 1u);
                        }
                        __syncwarp();
                        ok = ok && tc_wait(BAR(C::B_ACCE, mt), acc_par, abort_flag, spin_limit);
                        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                        if (tc_elect() && ok) {
                            if (active) {
                                tc_mma(d, a0, b, b_hi, idesc_hi, 0u);
#pragma unroll
                                for (uint32_t k = 1; k < 4; ++k) tc_mma(d, a0 + 8 * k, b + k * 16, b_hi, idesc_wide, 1u);
                            }
                            tc_commit(BAR(C::B_AFREE, mt));
                        }
                    } else if (tc_elect() && ok) {
                        if (active) {
#pragma unroll
                            for (uint32_t k = 0; k < 4; ++k) {
                                tc_mma(d, a0 + 8 * k, b + k * 16, b_hi, idesc_wide, k == 0 ? 0u : 1u);   // A_hi (B_hi | B_lo)
                                tc_mma(d_small, a0 + 8 * k + 32, b + k * 16, b_hi, idesc_hi, 1u);   // A_lo B_hi, on the small terms
                            }
                        }
                        tc_commit(BAR(C::B_AFREE, mt));
                    }
                    __syncwarp();
                    acc_par ^= 1;
                    ok = ok && tc_wait(BAR(C::B_AFULL, C::ABUF * mt + 1), a_par, abort_flag, spin_limit);
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    if (tc_elect() && ok) {
                        if (active) {
#pragma unroll
                            for (uint32_t k = 0; k < 4; ++k) {
                                tc_mma(d, a0 + 64 + 8 * k, b + 64 + k * 16, b_hi, idesc_wide, 1u);
                                tc_mma(d_small, a0 + 64 + 8 * k + 32, b + 64 + k * 16, b_hi, idesc_hi, 1u);
                            }
                        }
                        tc_commit(BAR(C::B_DONE, 2 * s + mt));
                    }
                    __syncwarp();
                    if (++s == C::STAGES) s = 0;
                }
            }
            // no MMA of this CTA may be in flight when its tensor memory is freed, whatever happened elsewhere.  (elect.sync picks the
            // same lane every time, the one whose MMAs the commit has to cover.)
            if (tc_elect()) {
                tc_commit(BAR(C::B_DRAIN, mt));
#pragma unroll 1
                for (uint32_t spin = 0; spin < TC_DRAIN_LIMIT && !tc_try(BAR(C::B_DRAIN, mt), 0); ++spin) {}
            }
            __syncwarp();
        } else if (warp == 2) {
            // ---------------- producer: two or four tensor copies of weights, one bulk copy of activations per block group ----------------
            uint32_t s = 0, par = 1, issued = 0;
            bool ok = !(plan.debug & 32) && !(plan.debug & 64 && blockIdx.x & 1);
            const uint32_t b_bytes = (uint32_t) act.chunk_nt * 4096u;
#pragma unroll 1
            for (uint32_t p = 0; p < sh->n_pieces && ok; ++p) {
                const TcPiece q = sh->piece[p];
                const int boxes = 1 + (int) q.two;   // rows past the end read as zero
                const uint32_t bytes = (uint32_t) boxes * 8u * (C::WT + 128u) + b_bytes;
                const int rt_in = (int) q.group * plan.rt_per_group;
                const uint8_t *bsrc = aq + act.b_offset + ((int64_t) q.chunk * n_bg + q.bg) * b_bytes;
#pragma unroll 1
                for (uint32_t i = 0; i < q.len; ++i) {
                    const uint32_t st = smem_u32 + s * C::STAGE, bar = BAR(C::B_FULL, s);
                    if (!tc_wait(BAR(C::B_WREAD, s), par, abort_flag, spin_limit) || !tc_wait(BAR(C::B_DONE, 2 * s), par, abort_flag, spin_limit) ||
                        !tc_wait(BAR(C::B_DONE, 2 * s + 1), par, abort_flag, spin_limit)) { ok = false; break; }
                    if (tc_elect()) {
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
                        const int bg = (int) (q.bg + i);
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            if (k < boxes) {
                                tc_tma_2d(st + (uint32_t) (k * 8 * C::WT), &maps.q, bg * 256, rt_in + 8 * k, bar);
                                tc_tma_2d(st + (uint32_t) (C::OFF_S + k * 1024), &maps.s, bg * 32, rt_in + 8 * k, bar);
                            }
                        }
                        tc_copy(st + C::OFF_B, bsrc + (int64_t) i * b_bytes, b_bytes, bar);
                    }
                    __syncwarp();
                    ++issued;
                    if (++s == C::STAGES) { s = 0; par ^= 1; }
                }
            }
            // copies in flight must land before the CTA may exit, whatever happened elsewhere
#pragma unroll 1
            for (uint32_t k = issued > C::STAGES ? issued - C::STAGES : 0; k < issued && lane == 0; ++k) {
                const uint32_t bar = BAR(C::B_FULL, k % C::STAGES), parity = (k / C::STAGES) & 1;
#pragma unroll 1
                for (uint32_t spin = 0; spin < TC_DRAIN_LIMIT && !tc_try(bar, parity); ++spin) {}
            }
            __syncwarp();
        }
    } else if (warp < C::WARP_EPI) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;\n");
        // ---------------- weights: a warp owns 32 rows (two T16 tiles: the lanes of tensor memory it can reach) of every second half block group ----------------
        const int q4 = warp & 3, mt = ((warp - 4) >> 2) & 1, team = (warp - 4) >> 3;
        const uint32_t rt0 = (uint32_t) (mt * 8 + q4 * 2);
        const uint32_t a_base = tmem + ((uint32_t) (32 * q4) << 16) + C::A_COL + (uint32_t) (mt * C::A_MT);
        const uint32_t w_at = smem_u32 + rt0 * C::WT + (uint32_t) (lane * 32);
        const uint32_t s_at = smem_u32 + C::OFF_S + rt0 * 128 + (uint32_t) ((lane >> 2) * 8);
        const bool active = mt == 0 || plan.rt_per_group > 8;
        const uint32_t halves = 2 * sh->n_iter;
        uint32_t s = 0, full_par = 0, free_par = 1;
#pragma unroll 1
        for (uint32_t hc = (uint32_t) team; hc < halves; hc += 2, free_par ^= 1) {
            const uint32_t half = hc & 1, ab = (uint32_t) team;
            if (!tc_wait(BAR(C::B_FULL, s), full_par, abort_flag, spin_limit)) break;
            uint32_t r[2][4];       // rows g, g + 8 x word t of the two blocks
            uint32_t sc[2][2];      // the two block scales of rows g, g + 8
#pragma unroll
            for (int u = 0; u < 2; ++u) {
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const uint32_t at = w_at + s * C::STAGE + half * 8 + (uint32_t) (u * C::WT + v * 16);
                    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];\n" : "=r"(r[u][2 * v]), "=r"(r[u][2 * v + 1]) : "r"(at));
                }
                const uint32_t sa = s_at + s * C::STAGE + half * 4 + (uint32_t) (u * 128);
                asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(sc[u][0]) : "r"(sa));
                asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(sc[u][1]) : "r"(sa + 64));
            }
            __syncwarp();
            if (lane == 0) tc_arrive(BAR(C::B_WREAD, s));   // the weights are in registers (the arrive orders the loads before it)
            if (team == 0) {
                if (!tc_wait(BAR(C::B_AFREE, mt), free_par, abort_flag, spin_limit)) break;
            } else if (hc > 1) {   // the block group before this one
                if (!tc_wait(BAR(C::B_DONE, 2 * (s == 0 ? C::STAGES - 1 : s - 1) + mt), s == 0 ? full_par ^ 1 : full_par, abort_flag, spin_limit)) break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t a_to = a_base + ab * 64;
            if (active) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {   // block 2 half + j of both tiles
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        uint32_t hi[8], lo[8];
#pragma unroll
                        for (int row = 0; row < 2; ++row) {
                            const __half2 d2 = j ? __high2half2(tc_as_h2(sc[u][row])) : __low2half2(tc_as_h2(sc[u][row]));
#pragma unroll
                            for (int si = 0; si < 4; ++si) {
                                __half2 q2;
                                // nibbles at bits 4 si and 16 + 4 si, two's complement; v = q + 8.  0x6400 | v is the fp16
                                // 1024 + v, 0x6400 | 16 v is 1024 + 16 v; both steps to q are exact
                                const uint32_t word = r[u][row * 2 + j], w8 = si < 2 ? word : word >> 8;
                                if ((si & 1) == 0) q2 = __hadd2(tc_as_h2((w8 & 0x000F000Fu) ^ 0x64086408u), __float2half2_rn(-1032.0f));
                                else q2 = __hfma2(tc_as_h2((w8 & 0x00F000F0u) ^ 0x64806480u), __float2half2_rn(0.0625f), __float2half2_rn(-72.0f));
                                const __half2 x = __hmul2(q2, d2);
                                hi[si * 2 + row] = tc_h2(x);
                                lo[si * 2 + row] = tc_h2(__hfma2(q2, d2, __hneg2(x)));
                            }
                        }
                        tc_st_16x128b_x4(a_to + ((uint32_t) (16 * u) << 16) + (uint32_t) (j * 16), hi);
                        tc_st_16x128b_x4(a_to + ((uint32_t) (16 * u) << 16) + (uint32_t) (j * 16) + 32, lo);
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            }
            __syncwarp();
            if (lane == 0) tc_arrive(BAR(C::B_AFULL, C::ABUF * mt + ab));
            s += 1;   // two halves on
            if (s >= C::STAGES) { s -= C::STAGES; full_par ^= 1; }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 120;\n");
        // ---------------- accumulator -> registers -> shared memory -> result; a warpgroup per MMA row tile ----------------
        const int q4 = warp & 3, mt = (warp - C::WARP_EPI) >> 2, et = tid - C::WARP_EPI * 32;
        const uint32_t cols = 8 * (uint32_t) act.chunk_nt, d_at = tmem + ((uint32_t) (32 * q4) << 16) + (uint32_t) (mt * C::D_MT);
        uint32_t s = 0, done_par = 0;
        bool ok = true;
#pragma unroll 1
        for (uint32_t p = 0; p < sh->n_pieces && ok; ++p) {
            const bool active = mt == 0 || sh->piece[p].two;
            const uint32_t len = sh->piece[p].len;
            float sum[64];   // of the thread's row
#pragma unroll
            for (int k = 0; k < 64; ++k) sum[k] = 0.0f;
#pragma unroll 1
            for (uint32_t i = 0; i < len && ok; ++i) {
                const uint32_t bar = BAR(C::B_DONE, 2 * s + mt), parity = done_par;
                if (++s == C::STAGES) { s = 0; done_par ^= 1; }
                ok = tc_wait(bar, parity, abort_flag, spin_limit);
                const auto read = [&] {
                    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0) tc_arrive(BAR(C::B_ACCE, mt));
                };
                if (!ok || !active) {
                    read();
                    continue;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                if (i + 1 == len) tc_add_columns(sum, d_at + cols, cols, [] {});   // the small terms, once
                tc_add_columns(sum, d_at, cols, read);
            }
            if (ok && active) {
                float *o = acc_s + mt * 128 + q4 * 32 + lane;
#pragma unroll
                for (int k = 0; k < 64; ++k)
                    if ((k & ~15) < (int) cols) o[k * 256] = sum[k];
            }
            if (plan.debug & 128 && warp == C::WARP_EPI + 1 && blockIdx.x == 1) {
                ok = false;
                *abort_flag = 1;
                atomicExch(&g_tc_error, 1);
            }
            if (p + 1 == sh->n_pieces) break;   // the last piece: all warps share what is left to do, below
            // one warp's wait may run out where its neighbours' did not: the team goes on, or leaves, together
            if (!ok) *wb_gave_up = 1;
            asm volatile("bar.sync 1, 256;\n" ::: "memory");
            if (*wb_gave_up) break;   // (written again at the earliest beyond the barriers of tc_finish)
            tc_finish(sh, acc_u32, p, (uint32_t) et, TC_EPI_THREADS, 1u);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    pdl_trigger();
    __syncthreads();   // (a warpgroup's registers change hands again: its warps must have met)
    if (warp < C::WARP_EPI) asm volatile("setmaxnreg.inc.sync.aligned.u32 72;\n");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 72;\n");
    if (plan.cs > 0) {
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
        if (!*abort_flag) tc_write_cluster(sh, acc_u32, (uint32_t) tid, C::THREADS);
        // nobody leaves while a neighbour may still read its part
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    } else {
        __syncthreads();
        if (*abort_flag) {
            if (tid == 0) tc_give_up_pieces(sh);
        } else if (sh->n_pieces > 0) {
            tc_finish(sh, acc_u32, sh->n_pieces - 1, (uint32_t) tid, C::THREADS, 0u);
        }
        __syncthreads();
    }
#undef BAR
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem) : "memory");
}

static int tc_sm_count() {   // every device of a process is the same model
    static const int n = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v > 0 ? v : 148;
    }();
    return n;
}

using tc_kernel_fn = void (*)(TiledDims, const uint8_t *, ActDims, const uint8_t *, float *, int64_t, void *, TcPlan, TcMaps);
struct TcVariant {
    tc_kernel_fn fn;
    int smem, threads;
    int max_clusters[9];   // resident clusters of 1..8 CTAs on the current device
};
static void tc_make(TcVariant &v) {
    v.fn = mmq_tc_kernel;
    v.smem = TcCfg::SMEM;
    v.threads = TcCfg::THREADS;
    cudaFuncSetAttribute(v.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem);
    for (int cs = 1; cs <= 8; ++cs) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned) cs);
        cfg.blockDim = dim3((unsigned) v.threads);
        cfg.dynamicSmemBytes = (size_t) v.smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned) cs;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cs == 1) n = tc_sm_count();
        else if (cudaOccupancyMaxActiveClusters(&n, v.fn, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        v.max_clusters[cs] = n;
    }
}
static const TcVariant &tc_variant() {
    static TcVariant table[64];   // per device: kernel attributes and occupancy are per-context properties
    static bool ready[64] = {false};
    static std::mutex mu;
    int dev = 0;
    cudaGetDevice(&dev);
    dev &= 63;
    std::lock_guard<std::mutex> lock(mu);
    if (!ready[dev]) {
        tc_make(table[dev]);
        ready[dev] = true;
    }
    return table[dev];
}

// ---- tensor maps ----
typedef CUresult (*tc_encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                 const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static tc_encode_fn tc_encoder() {
    static tc_encode_fn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) != cudaSuccess || qr != cudaDriverEntryPointSuccess) p = nullptr;
        return (tc_encode_fn) p;
    }();
    return fn;
}
// `rows` rows of `words` 32-bit words, a box of box_words x 8 rows
static bool tc_encode(CUtensorMap *m, const void *base, uint64_t words, uint64_t rows, uint32_t box_words) {
    tc_encode_fn enc = tc_encoder();
    if (!enc) return false;
    const cuuint32_t elem[2] = {1, 1}, box[2] = {box_words, 8};
    const cuuint64_t dims[2] = {words, rows}, strides[1] = {words * 4};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void *>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// encoded maps are pure functions of (pointer, extents): kept, a model has a few hundred weights
struct TcKey {
    const void *p;
    int64_t a, b;
    bool operator==(const TcKey &o) const { return p == o.p && a == o.a && b == o.b; }
};
struct TcKeyHash {
    size_t operator()(const TcKey &k) const { return std::hash<const void *>()(k.p) ^ (size_t) (k.a * 0x9E3779B97F4A7C15ull) ^ (size_t) (k.b * 0xC2B2AE3D27D4EB4Full); }
};
static bool tc_weight_maps(const TiledDims &d, const void *w, TcMaps &maps) {
    static std::mutex mu;
    static std::unordered_map<TcKey, TcMaps, TcKeyHash> cache;
    const TcKey key{w, d.n_rt, d.n_bg};
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it == cache.end()) {
        TcMaps p;
        if (!tc_encode(&p.q, w, (uint64_t) d.n_bg * 256, (uint64_t) d.n_rt, 256)) return false;
        if (!tc_encode(&p.s, (const uint8_t *) w + d.qs_bytes, (uint64_t) d.n_bg * 32, (uint64_t) d.n_rt, 32)) return false;
        if (cache.size() > 65536) cache.clear();
        it = cache.emplace(key, p).first;
    }
    maps = it->second;
    return true;
}

static size_t tc_counter_bytes(int64_t tiles) { return (size_t) ((tiles * 8 + 255) / 256 * 256); }
// workspace of the equal-share split: a counter per tile, two parked parts (64 columns x 256 rows) per CTA
size_t mmq_tc_workspace_bytes(int64_t M, int64_t N) {
    const int64_t tiles = ((M + 127) / 128) * ((N + 63) / 64);
    return tc_counter_bytes(tiles) + (size_t) tc_sm_count() * 2 * (64 * 256 * 4);
}

// The work split, from what was measured on B200 (clocks per block group of a CTA: the MMAs, or the copies when a CTA has only 128
// rows; a few block groups of fixed cost to start and to finish).
static TcPlan tc_plan(const TcVariant &v, const TiledDims &d, const ActDims &a, bool workspace) {
    static const int forced = [] {   // tuning aid: B200_TC_PLAN = 100 * (row tiles 8 / 16) + cluster size (0: equal shares)
        const char *e = getenv("B200_TC_PLAN");
        return e ? atoi(e) : -1;
    }();
    static const int debug = [] {
        const char *e = getenv("B200_TC_DEBUG");
        return e ? atoi(e) : 0;
    }();
    TcPlan best = {};
    double best_cost = -1;
    const int chunk_nt = a.chunk_nt, chunks = (int) ((a.n_nt + chunk_nt - 1) / chunk_nt);
    for (int rpg = 16; rpg >= 8; rpg -= 8) {
        const int64_t groups = (d.n_rt + rpg - 1) / rpg, tiles = groups * chunks;
        // clocks per block group: MMAs (96 per 16 values of K and 128 rows at 64 columns), against the copies at 40 B/clk
        const double mma = (rpg / 8) * 8 * 12.0 * chunk_nt, copy = (rpg * (d.tile_bytes + 128) + chunk_nt * 4096) / 40.0;
        // and what the hand-overs between the warps allow
        const double unit = std::max(std::max(mma * 1.15, copy), 1400.0) / 1000.0;
        for (int cs = 0; cs <= 8; ++cs) {
            double cost;
            if (cs == 0) {
                // few tiles would have many parts each, which one CTA would have to add (tc_finish knows three)
                const int64_t grid = std::min<int64_t>(tc_sm_count(), tiles * d.n_bg), share = tiles * d.n_bg / grid;
                if (!workspace || 2 * share < d.n_bg || share / d.n_bg + 4 > TC_MAX_PIECES) continue;
                cost = (double) (tiles * d.n_bg) / tc_sm_count() * unit + 2.0 * unit + 6.0;
            } else {
                if (cs > d.n_bg || v.max_clusters[cs] <= 0) continue;
                const int64_t waves = (tiles + v.max_clusters[cs] - 1) / v.max_clusters[cs];
                cost = waves * (((d.n_bg + cs - 1) / cs) * unit + 2.0 * unit + (cs > 1 ? 3.0 : 2.0));
            }
            if (forced >= 0 && forced != rpg * 100 + cs) continue;
            if (best_cost < 0 || cost < best_cost) {
                best_cost = cost;
                best.rt_per_group = rpg;
                best.groups = (int) groups;
                best.chunks = chunks;
                best.cs = cs;
            }
        }
    }
    if (best_cost < 0) {
        best.rt_per_group = 16;
        best.groups = (int) ((d.n_rt + 15) / 16);
        best.chunks = chunks;
        best.cs = 1;
    }
    best.debug = debug;
    return best;
}

int launch_mmq_tc(const TiledDims &d, const void *w, const ActDims &a, const void *aq, float *dst, int64_t dst_nb_row,
                  void *workspace, size_t workspace_bytes, cudaStream_t st) {
    const TcVariant &v = tc_variant();
    TcMaps maps;
    if (!tc_weight_maps(d, w, maps)) return set_error(B200_E_CUDA, "mmq_tc: no tensor map for the weights");
    const bool ws = workspace && workspace_bytes >= mmq_tc_workspace_bytes(d.M, a.N) && d.n_rt * d.n_bg * a.n_nt < (1ll << 31);
    TcPlan plan = tc_plan(v, d, a, ws);
    const int tiles = plan.groups * plan.chunks;
    static std::atomic<unsigned long long> next_id{(unsigned long long) std::chrono::steady_clock::now().time_since_epoch().count() * 0x9E3779B97F4A7C15ull};
    plan.launch_id = (next_id.fetch_add(1) & 0xffffffffffffffull) | 1ull << 55;   // never zero
    const int64_t total = (int64_t) tiles * d.n_bg;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) (plan.cs == 0 ? std::min<int64_t>(tc_sm_count(), total) : (int64_t) tiles * plan.cs));
    plan.share = (uint32_t) (total / cfg.gridDim.x);
    plan.extra = (uint32_t) (total % cfg.gridDim.x);
    cfg.blockDim = dim3((unsigned) v.threads);
    cfg.dynamicSmemBytes = (size_t) v.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (plan.cs > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned) plan.cs;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = (unsigned) n;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, v.fn, d, (const uint8_t *) w, a, (const uint8_t *) aq, dst, dst_nb_row, workspace, plan, maps);
    if (e != cudaSuccess) return set_error(B200_E_CUDA, "mmq_tc launch: %s", cudaGetErrorString(e));
    return check_launch("mmq_tc");
}

int tc_error_flag() {
    int v = 0;
    cudaMemcpyFromSymbol(&v, g_tc_error, sizeof(int));
    return v;
}
void tc_set_wait_limit(unsigned rounds) {
    const unsigned v = rounds ? rounds : 1u << 20;
    const int zero = 0;
    cudaMemcpyToSymbol(g_tc_spin_limit, &v, sizeof(v));
    cudaMemcpyToSymbol(g_tc_error, &zero, sizeof(zero));
}

}  // namespace b200
