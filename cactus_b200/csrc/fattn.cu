// FLASH_ATTN_EXT over the f16 unified KV cache for ragged multi-sequence batches.
//
// Replaces lm_ggml_compute_forward_flash_attn_ext_f16 (cactus/ggml-cpu/ops.cpp:6948-7165).
//
// The mask tensor is honoured exactly as the reference does (a cell takes part iff its mask value is
// not -inf, the finite value is added to the scaled score), but it is scanned only once per graph:
// b200_mask_index_build turns each token's mask row into one bit per cell, and the attention kernel
// walks the set bits, so a token of a 64-sequence batch touches only its own sequence's K/V rows.
//
// Kernel: one CTA per (token, kv-head, group of up to 8 query heads, KV split), tensor-core MMAs for both
// Q K^T and P V (see fattn_mma_kernel).  With KV splits the partial (max, sum, accumulator) triples go to
// scratch and a combine kernel finishes.  A second, slow kernel reproduces the reference's own rounding
// sequence for validation (fattn_parity_kernel).
#include <cooperative_groups.h>
#include <math_constants.h>

#include <cstdlib>

#include "common.cuh"
#include "mma_s8.cuh"

namespace b200 {


constexpr int FA_THREADS = 128;
#ifndef FA_MIN_CTAS
#define FA_MIN_CTAS 3
#endif
#ifndef FA_PREFETCH_V
#define FA_PREFETCH_V 0   // 1: the next chunk's V rows are requested as soon as the P V MMAs of the current one have read theirs (measured slower on B200: 67.9 us against 57.5 on 64 ragged sequences)
#endif
#ifndef FA_PREFETCH_K
#define FA_PREFETCH_K 1   // the next chunk's K rows are loaded during the softmax and P V MMAs of the current one (32 more registers)
#endif
constexpr int FA_SUPER_WORDS = 32;  // 2048 cells listed per round
constexpr int FA_MIN_SPLIT_WORDS = 2;   // 64-cell words a KV split walks at least (when the mask index gives a token's word count)
constexpr int FA_CLUSTER_MAX = 8;   // CTAs of a cluster
constexpr int FA_ADAPTIVE_SPLITS = 2;   // most KV splits a long sequence is cut into when the batch is small

// ---- mask scan: one CTA per token row --------------------------------------------------------------
// The row as one bit per cell, 64 cells to a word; the indices of the words that have any participating cell, in ascending
// order, and their count (a token of a 64-sequence batch owns a few dozen of the 1024 words of a 65536-cell cache, and the
// attention kernels walk only those); whether the row holds more than 0 and -inf in participating cells.
// Reads the mask once, 16 bytes (8 cells) per thread and load, four loads in flight; one kernel for what was a memset, a scan
// and a pass over the words that the scan had written.  Whole index build, us before / now on B200 (tokens x cells): 1 x 1024
// 8.3 / 3.5, 64 x 65536 23.9 / 9.4, 512 x 8192 49.7 / 13.3, 512 x 65536 109 / 27.  A cluster of 2 or 4 CTAs per row was faster at
// 64 x 65536 only (7.9) and slower from 1 x 1024 (4.6) to 512 x 65536 (32, 43).
constexpr int MI_THREADS = 512, MI_WORDS = 2048;   // words whose indices are listed per round
// SINGLE: one token, whose plan (below) this kernel makes as well
template <bool VEC, bool SINGLE>
__global__ void __launch_bounds__(MI_THREADS, 3) mask_index_kernel(const __half *__restrict__ mask, int64_t mask_nb_row, int64_t n_kv, int64_t nw,
                                                               unsigned long long *__restrict__ words, int32_t *__restrict__ wlist, int32_t *__restrict__ wcount,
                                                               uint8_t *__restrict__ soft, int32_t *__restrict__ order, int32_t *__restrict__ plan) {
    pdl_prologue();
    __shared__ unsigned bits[MI_WORDS / 32];
    __shared__ int warp_cnt[MI_WORDS / 1024], any_soft;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t j = blockIdx.x;
    const __half *row = reinterpret_cast<const __half *>(reinterpret_cast<const char *>(mask) + j * mask_nb_row);
    unsigned long long *out = words + j * nw;
    int32_t *list = wlist + j * nw;
    int base = 0;   // listed so far
    unsigned soft_bits = 0;
    if (tid == 0) any_soft = 0;
    for (int64_t w0 = 0; w0 < nw; w0 += MI_WORDS) {
        const int n = (int) min((int64_t) MI_WORDS, nw - w0);
        if (tid < MI_WORDS / 32) bits[tid] = 0u;
        __syncthreads();
#pragma unroll 4
        for (int i = tid; i < (n * 8 + 31) / 32 * 32; i += MI_THREADS) {   // 8 cells; whole warps
            const int64_t c0 = (w0 * 8 + i) * 8;
            unsigned h[4] = {0xFC00FC00u, 0xFC00FC00u, 0xFC00FC00u, 0xFC00FC00u};
            if (VEC ? c0 + 8 <= n_kv : false) {
                const uint4 v = __ldg(reinterpret_cast<const uint4 *>(row + c0));
                h[0] = v.x; h[1] = v.y; h[2] = v.z; h[3] = v.w;
            } else {
#pragma unroll
                for (int x = 0; x < 8; ++x)
                    if (c0 + x < n_kv) h[x >> 1] = (h[x >> 1] & (x & 1 ? 0xffffu : 0xffff0000u)) | ((unsigned) __half_as_ushort(row[c0 + x]) << (16 * (x & 1)));
            }
            unsigned m = 0;
#pragma unroll
            for (int x = 0; x < 4; ++x) {   // two cells at a time: all ones where the value is not -inf
                const unsigned in = ~__heq2_mask(*reinterpret_cast<const __half2 *>(&h[x]), __half2half2(__ushort_as_half((unsigned short) 0xFC00u)));
                m |= in & ((1u << (2 * x)) | (1u << (17 + 2 * x)));
                soft_bits |= h[x] & in & 0x7fff7fffu;   // not +-0: added to the score
            }
            m = (m | (m >> 16)) & 0xffu;
            if (i < n * 8) reinterpret_cast<uint8_t *>(out + w0)[i] = (uint8_t) m;   // byte by byte in the order of the words' bits
            unsigned any8 = __ballot_sync(0xffffffffu, m != 0u);
            if (any8 && lane == 0) {   // the warp's four words
                any8 |= any8 >> 4;
                any8 |= any8 >> 2;
                any8 |= any8 >> 1;
                atomicOr(bits + (i >> 8), ((any8 & 1u) | ((any8 >> 7) & 2u) | ((any8 >> 14) & 4u) | ((any8 >> 21) & 8u)) << ((i >> 3) & 31));
            }
        }
        __syncthreads();
        const unsigned mine = tid < MI_WORDS / 32 ? bits[tid] : 0u;
        const int cnt = __popc(mine);
        int pre = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += x;
        }
        if (lane == 31 && warp < MI_WORDS / 1024) warp_cnt[warp] = pre;
        __syncthreads();
        int at = base + pre - cnt;
#pragma unroll
        for (int w = 0; w < MI_WORDS / 1024; ++w) {
            at += w < warp ? warp_cnt[w] : 0;
            base += warp_cnt[w];
        }
        for (unsigned m = mine; m; m &= m - 1) list[at++] = (int32_t) (w0 + 32 * tid + __ffs((int) m) - 1);
        __syncthreads();
    }
    if (soft_bits) any_soft = 1;
    __syncthreads();
    if (tid == 0) {
        wcount[j] = base;
        soft[j] = (uint8_t) any_soft;
        if (SINGLE) {   // what fattn_plan_kernel would make
            order[0] = 0;
            plan[0] = base;
            plan[2] = any_soft;
            plan[1] = plan[4] = plan[5] = plan[6] = plan[7] = 0;
        }
    }
}

// Second pass: the tokens ordered by decreasing word count (longest sequence first, so the scheduler hands the long
// walks out first and the short ones fill the gaps), and the total number of words, from which the attention kernel
// derives how many words one CTA should walk.  A warp per token counts the tokens that come before it; the first CTA also
// makes the totals.
__global__ void __launch_bounds__(256) fattn_plan_kernel(const int32_t *__restrict__ wcount, const uint8_t *__restrict__ soft, int64_t Nq, int32_t *__restrict__ order,
                                                        int32_t *__restrict__ plan) {
    pdl_prologue();
    const int lane = threadIdx.x & 31;
    const int64_t j = (int64_t) blockIdx.x * 8 + (threadIdx.x >> 5);
    if (j < Nq) {
        const int32_t c = wcount[j];
        int rank = 0;   // tokens with more words, or as many and a lower index, come first
        for (int64_t i = lane; i < Nq; i += 32) {
            const int32_t ci = wcount[i];
            rank += (ci > c || (ci == c && i < j)) ? 1 : 0;
        }
        rank = __reduce_add_sync(0xffffffffu, rank);
        if (lane == 0) order[rank] = (int32_t) j;
    }
    if (blockIdx.x == 0) {
        __shared__ unsigned long long part_s[8];
        __shared__ int any;
        if (threadIdx.x == 0) any = 0;
        __syncthreads();
        unsigned long long part = 0;
        int s = 0;
        for (int64_t i = threadIdx.x; i < Nq; i += blockDim.x) {
            part += (unsigned long long) wcount[i];
            s |= soft[i];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        if (lane == 0) part_s[threadIdx.x >> 5] = part;
        if (s) any = 1;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long total = 0;
            for (int w = 0; w < 8; ++w) total += part_s[w];
            plan[0] = (int32_t) min(total, 0x7fffffffull);
            plan[1] = 0;   // this and the last four: fattn_tile_vote_kernel
            plan[2] = any;
            plan[4] = plan[5] = plan[6] = plan[7] = 0;
        }
    }
}

// Third pass: how much the tokens of a ubatch share their cells.  plan[1] = the sum, over groups of 16 consecutive
// tokens, of the number of mask words any token of the group attends to.  Against plan[0] (the same sum token by token)
// it tells whether walking the cells once per group (fattn_tile_kernel) beats walking them once per token: a prompt's
// tokens share nearly all their words, the tokens of a decode batch share none.  And the same for every tile the
// query-tiled kernel may use (4, 8, 16 or 32 tokens): tiles whose tokens share little (decode tokens beside a prompt) are
// flagged and listed, their tokens are walked one by one (plan[4 + k] = listed tiles of 4 << k tokens).  The line lies at one and a
// half tokens per word: a token's own chunk costs a CTA about two thirds of a shared one (64 sequences with 3 tokens each, 2.7
// tokens per word: 415 us token by token, 220 shared; with 2 tokens each 147 and 86).
constexpr int VOTE_WORDS = 4096;
__global__ void __launch_bounds__(256) fattn_tile_vote_kernel(const int32_t *__restrict__ wlist, const int32_t *__restrict__ wcount, int64_t Nq, int64_t nw,
                                                             int32_t *__restrict__ plan, int32_t *__restrict__ flags, int32_t *__restrict__ lists, int64_t stride) {
    pdl_prologue();
    const int64_t t0 = (int64_t) blockIdx.x * 32;
    const int n = (int) min((int64_t) 32, Nq - t0);
    int cnt[15];   // words of: 8 groups of 4 tokens, 4 of 8, 2 of 16, 1 of 32
#pragma unroll
    for (int i = 0; i < 15; ++i) cnt[i] = 0;
    __shared__ unsigned who[VOTE_WORDS];   // per word: the tokens that attend to it
    for (int64_t w0 = 0; w0 < nw; w0 += VOTE_WORDS) {
        const int m = (int) min((int64_t) VOTE_WORDS, nw - w0);
        for (int i = threadIdx.x; i < m; i += blockDim.x) who[i] = 0u;
        __syncthreads();
        for (int j = threadIdx.x >> 5; j < n; j += 8) {
            const int32_t *wl = wlist + (t0 + j) * nw;
            const int c = wcount[t0 + j];
            for (int e = threadIdx.x & 31; e < c; e += 32) {
                const int64_t wi = wl[e] - w0;
                if (wi >= 0 && wi < m) atomicOr(who + wi, 1u << j);
            }
        }
        __syncthreads();
        for (int wi = threadIdx.x; wi < m; wi += blockDim.x) {
            const unsigned nz = who[wi];
#pragma unroll
            for (int i = 0; i < 8; ++i) cnt[i] += ((nz >> (4 * i)) & 0xfu) != 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) cnt[8 + i] += ((nz >> (8 * i)) & 0xffu) != 0;
#pragma unroll
            for (int i = 0; i < 2; ++i) cnt[12 + i] += ((nz >> (16 * i)) & 0xffffu) != 0;
            cnt[14] += nz != 0;
        }
        __syncthreads();
    }
    __shared__ int sum[15];
    if (threadIdx.x < 15) sum[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 15; ++i) {
        int c = cnt[i];
        for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if ((threadIdx.x & 31) == 0 && c) atomicAdd(sum + i, c);
    }
    __syncthreads();
    if (threadIdx.x < 15) {
        const int i = threadIdx.x, k = i < 8 ? 0 : (i < 12 ? 1 : (i < 14 ? 2 : 3)), first = k == 0 ? i : (k == 1 ? i - 8 : (k == 2 ? i - 12 : 0)), size = 4 << k;
        if (first * size < n) {
            if (k == 2) atomicAdd(plan + 1, sum[i]);
            int64_t own = 0;
            for (int j = first * size; j < min(n, (first + 1) * size); ++j) own += wcount[t0 + j];
            const int32_t tile = (int32_t) (t0 / size + first), few = 2 * own < 3ll * sum[i] ? 1 : 0;
            flags[k * stride + tile] = few;
            if (few) lists[k * stride + atomicAdd(plan + 4 + k, 1)] = tile;
        }
    }
}
// the choice both attention kernels derive from the plan: true = the query-tiled kernel does the work
__device__ __forceinline__ bool fattn_tiled_chosen(const int32_t *plan) { return 2ll * plan[1] <= (long long) plan[0]; }

struct FattnParams {
    int64_t H, Hkv, Nq, n_kv, nw;
    const float *q; int64_t q_nb_tok, q_nb_head;
    const char *k; int64_t k_nb_cell, k_nb_head;
    const char *v; int64_t v_nb_cell, v_nb_head;
    const char *mask; int64_t mask_nb_row;
    const unsigned long long *words;  // NULL: every cell takes part
    const int32_t *wlist, *wcount;    // per token: indices of the non-empty words and their number (with words)
    float scale, max_bias, softcap, m0, m1;
    uint32_t n_head_log2;
    float *dst;      // may be null when qout is given
    uint8_t *qout;   // optional: the output rows quantised to Q8_0 in the B8 activation layout of the mul_mat that follows
    size_t q_d_offset;
    int64_t q_nb, q_nbp;
    int q_variant;
    float *partial;  // [Nq][H][nsplit][D + 2]
    int nsplit, hgroups;
    int w0;          // > 0: a token gets ceil(words / w0) KV splits (at most nsplit), so long sequences are cut, short ones are not;
                     // < 0: w0 is derived on the device from the mask's total word count (fattn_target_words)
    const int32_t *tflags, *tlist, *tcount;   // query-tiled kernel: tiles whose tokens share few cells (flag per tile, list, length of the list)
    int spread_rows;               // query-tiled kernel: grid rows whose CTAs take those tiles' tokens one by one
    const int32_t *order, *plan;   // tokens by decreasing word count; plan[0] = total words (NULL without a mask index)
    int slots;       // CTAs of this kernel the device holds at once
    int vote;        // both attention kernels were launched and the plan decides which one works (the other returns at once):
                     // 1 = these are the per-token kernel's launches, 2 = the query-tiled kernel's
    int parts;       // every token's result goes through `partial`, also that of a single split: the combine pass quantises them all
    int early;       // one or two tokens: the combine pass lets the next kernel's CTAs in at once (pdl_early_rows)
};

}  // namespace b200
#include "fattn_tile.cuh"   // the query-tiled kernel for ubatches with many tokens
namespace b200 {

// Tensor-core kernel.  One CTA per (token, kv-head, head group of up to 8 query heads, KV split); its 4 warps take
// 16-cell chunks of the token's cell list in turn.  Per chunk and warp:
//   S = Q K^T   heads on the MMA rows (m16n8k16, f16 inputs, f32 accumulate), 8 cells per n-tile.  Lane (g, t)
//               loads 16-byte pieces d = 32u + 8t .. +7 of the K row of cell g -- the k index of the MMA is a fixed
//               permutation of d that makes those pieces B fragments as they are; Q is held in the same permutation
//               (rounded to fp16 as the reference rounds it).
//   online softmax on the accumulator rows (a head's four lanes share max and sum through two shuffles)
//   O^T += V^T P^T   d on the MMA rows, heads on the columns, so no accumulator row is wasted: lane (g, t) loads
//               d = 8g .. 8g+7 (and 64 + 8g ..) of the V rows of cells 2t, 2t+1, 2t+8, 2t+9 and pairs the halves of
//               two cells with byte permutes; P goes in as fp16 hi + lo parts (two MMAs), which keeps the
//               probabilities at fp32 accuracy.
// Every warp keeps its own (max, sum, accumulator) state; the states are merged through shared memory at the end.
// words one CTA should walk: 1.15 x the mean load of a CTA slot if the whole mask were spread evenly (at least 4 words)
__device__ __forceinline__ int fattn_target_words(const FattnParams &p, int ctas_per_token) {
    if (p.w0 >= 0) return p.w0;
    const long long total = p.plan ? p.plan[0] : p.Nq * p.nw;
    const long long w = (115ll * total * ctas_per_token + 100ll * p.slots - 1) / (100ll * p.slots);
    return (int) max(4ll, min(w, 0x7fffffffll));
}

// Called by the 32 lanes of a warp with 32 consecutive elements of one output row: quantises them as one Q8_0 block of
// column n.  A real call (not inlined): the attention kernel sits at its register limit and its main loop must not pay
// for this code.
__device__ __noinline__ void fattn_quant_block(uint8_t *qout, size_t d_offset, int64_t nb, int64_t nbp, int variant, int64_t n, int64_t b,
                                               float val, bool real) {
    q8_quantize_store_warp<1>(val, qout, d_offset, nb, nbp, n, b, real, variant);
}

// Block b of the padding columns n .. (the rest of their 8-column tile) as the quantiser leaves it: zeros
__device__ __noinline__ void fattn_quant_pad(uint8_t *qout, size_t d_offset, int64_t nbp, int64_t n, int64_t b) {
    const int lane = threadIdx.x & 31, g = (int) (n & 7);
    if (lane >= 4 * g) *reinterpret_cast<uint2 *>(qout + ((n >> 3) * nbp + b) * 256 + lane * 8) = make_uint2(0u, 0u);
    if (lane >= g && lane < 8) {
        float *dp = reinterpret_cast<float *>(qout + d_offset) + ((n >> 3) * (nbp >> 2) + (b >> 2)) * 64 + act_scale_index((int) (b & 3), lane);
        dp[0] = 0.0f;
        dp[2] = -0.0f;
    }
}

// One output element; a warp calls this for 32 consecutive d of one (token, head).  With QUANT the row is also (or only)
// stored as Q8_0 blocks -- quantize_row_q8_0 applied to the f32 value, bit for bit what the separate quantiser makes of
// dst -- and the last token's warps zero the padding columns of its 8-column tile.
template <int D, bool QUANT>
__device__ __forceinline__ void fattn_store_out(const FattnParams &p, int64_t j, int64_t head, int d, float val) {
    if (!QUANT) {
        p.dst[(j * p.H + head) * D + d] = val;
        return;
    }
    if (p.dst) p.dst[(j * p.H + head) * D + d] = val;
    const int64_t b = (head * D + d) >> 5;
    fattn_quant_block(p.qout, p.q_d_offset, p.q_nb, p.q_nbp, p.q_variant, j, b, val, true);
    if (j == p.Nq - 1 && (p.Nq & 7)) fattn_quant_pad(p.qout, p.q_d_offset, p.q_nbp, p.Nq, b);
}

// QUANT: the instantiation behind b200_flash_attn_ext_quant; kept apart because this kernel sits at its register limit
// and the plain one must not change with it
// CLUSTER: the KV splits of a token and head group are a cluster of CTAs, which add their parts through each other's shared memory; see
// launch_mma_cluster
// VOTED: launched beside the query-tiled kernel, mostly to return.  It has one walk, which reads the mask, where the others have a second one for
// masks of 0 and -inf: with both the returning grid costs up to 0.6 us more, 0.3 in the mean of 12 processes that differed in what ran before (16 ragged
// sequences, 512 tokens, 121.2 us; what ran before moves that by as much again).  A test in a single walk instead is no way
// out: 64 decode tokens 75.3 us, 73.2 with two walks.
template <int D, bool QUANT, bool CLUSTER = false, bool VOTED = false>
__global__ void __launch_bounds__(FA_THREADS, FA_MIN_CTAS) fattn_mma_kernel(FattnParams p) {
    pdl_prologue();
    if ((VOTED || (CLUSTER && p.vote == 1)) && fattn_tiled_chosen(p.plan)) return;   // the query-tiled kernel takes this ubatch
    constexpr bool PREFETCH_V = FA_PREFETCH_V || (CLUSTER && D == 64);   // (where there are registers for it)
    constexpr int KS = D / 16;   // k-steps of the S MMA
    constexpr int NU = D / 32;   // 16-byte K pieces per lane and cell
    constexpr int NR = D / 64;   // 64-wide d ranges of V
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    // blocks are handed out heads first, then tokens in the order of the plan: the longest sequences start first
    const int64_t j = !CLUSTER && p.order ? p.order[blockIdx.y] : blockIdx.y;   // (a cluster grid is resident as a whole)
    const int hk = blockIdx.x / p.hgroups, hg = blockIdx.x % p.hgroups;
    const int split = blockIdx.z;
    const int gqa = (int) (p.H / p.Hkv);
    const int G = min(8, gqa - hg * 8);        // query heads of this CTA
    const int h0 = hk * gqa + hg * 8;

    __shared__ int cell_list[FA_SUPER_WORDS * 64];
    __shared__ int list_count;
    __shared__ float merge_m[4][8], merge_l[4][8];
    __shared__ float merge_acc[4][8][D];
    __shared__ float part_m[8], part_l[8];   // with CLUSTER: of this split; its part is in merge_acc[0]

    // Q fragments: row g = head h0 + g (zero rows beyond G)
    uint32_t qa0[KS], qa2[KS];
    {
        const bool valid = g < G;
        const float *qp = reinterpret_cast<const float *>(reinterpret_cast<const char *>(p.q) + j * p.q_nb_tok + (int64_t) (h0 + (valid ? g : 0)) * p.q_nb_head);
#pragma unroll
        for (int u = 0; u < NU; ++u)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int d0 = 32 * u + 8 * t + 4 * v;
                const float4 f = valid ? *reinterpret_cast<const float4 *>(qp + d0) : make_float4(0.f, 0.f, 0.f, 0.f);
                qa0[2 * u + v] = pack_half2(f.x, f.y);
                qa2[2 * u + v] = pack_half2(f.z, f.w);
            }
    }
    const uint32_t hh = (uint32_t) (h0 + g);
    const float slope = (p.max_bias > 0.0f) ? (hh < p.n_head_log2 ? powf(p.m0, (float) (hh + 1)) : powf(p.m1, (float) (2 * (hh - p.n_head_log2) + 1))) : 1.0f;

    float oacc[8][4];   // O^T: d-tile q; [0],[1]: d = 8g+q, heads 2t, 2t+1; [2],[3]: d = 64+8g+q
#pragma unroll
    for (int q = 0; q < 8; ++q) oacc[q][0] = oacc[q][1] = oacc[q][2] = oacc[q][3] = 0.0f;
    float m_run = -CUDART_INF_F, l_run = 0.0f;   // state of head g (l: this lane's share of the row sum)

    // the words this CTA walks: entries [w_begin, w_end) of the token's list of non-empty words (or of all words
    // when there is no mask), an equal share per KV split
    const unsigned long long *wrow = p.words ? p.words + j * p.nw : nullptr;
    const int32_t *wl = p.words ? p.wlist + j * p.nw : nullptr;
    const int64_t n_words = p.words ? (int64_t) p.wcount[j] : p.nw;
    int ns_j = p.nsplit;   // KV splits of this token
    if (p.w0 != 0) {
        const int w0 = fattn_target_words(p, (int) gridDim.x);
        ns_j = (int) min((int64_t) p.nsplit, max((int64_t) 1, (n_words + w0 - 1) / w0));
        if (!CLUSTER && split >= ns_j) return;   // the whole CTA: nothing has been synchronised yet
    }
    const int64_t per_split = (n_words + ns_j - 1) / ns_j;
    const int64_t w_begin = CLUSTER ? min(n_words, (int64_t) split * per_split) : (int64_t) split * per_split;
    const int64_t w_end = min(n_words, w_begin + per_split);
    // (a mask of nothing but 0 and -inf adds nothing in the cells that take part)
    const __half *mrow = VOTED || (p.mask && p.plan[2] != 0) ? reinterpret_cast<const __half *>(p.mask + j * p.mask_nb_row) : nullptr;
    const char *kbase = p.k + (int64_t) hk * p.k_nb_head;
    const char *vbase = p.v + (int64_t) hk * p.v_nb_head;

    auto walk = [&](auto soft) {
    for (int64_t w0 = w_begin; w0 < w_end; w0 += FA_SUPER_WORDS) {
        if (warp == 0) {   // list the participating cells of this round
            const int64_t e = w0 + lane;
            unsigned long long bits = 0;
            int64_t wi = 0;
            if (e < w_end) {
                if (wrow) {
                    wi = wl[e];
                    bits = wrow[wi];
                } else {
                    wi = e;
                    const int64_t left = p.n_kv - wi * 64;
                    bits = left >= 64 ? ~0ull : ((1ull << left) - 1ull);
                }
            }
            const int cnt = __popcll(bits);
            int pre = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, pre, o);
                if (lane >= o) pre += x;
            }
            int pos = pre - cnt;
            while (bits) {
                const int b = __ffsll((long long) bits) - 1;
                bits &= bits - 1;
                cell_list[pos++] = (int) (wi * 64 + b);
            }
            if (lane == 31) list_count = pre;
        }
        __syncthreads();
        const int count = list_count;
        const int n_chunks = (count + 15) >> 4;
        const int last = count - 1;
        uint4 kr[2][NU];   // K rows of the two 8-cell tiles of a chunk: 16-byte pieces t, t+4, ... of cell g
        auto load_k = [&](int chunk) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int64_t cell = cell_list[min((chunk << 4) + 8 * c + g, last)];
                const uint4 *kp = reinterpret_cast<const uint4 *>(kbase + cell * p.k_nb_cell) + t;
#pragma unroll
                for (int u = 0; u < NU; ++u) kr[c][u] = __ldg(kp + 4 * u);
            }
        };
        uint4 vr[4][NR];   // V rows of a chunk: 16-byte piece g (and g + 8) of cells 2t, 2t+1, 2t+8, 2t+9
        auto load_v = [&](int chunk) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int64_t cell = cell_list[min((chunk << 4) + 2 * t + (i & 1) + 8 * (i >> 1), last)];
                const uint4 *vp = reinterpret_cast<const uint4 *>(vbase + cell * p.v_nb_cell) + g;
#pragma unroll
                for (int r = 0; r < NR; ++r) vr[i][r] = __ldg(vp + 8 * r);
            }
        };
        if (FA_PREFETCH_K && warp < n_chunks) load_k(warp);
        if (PREFETCH_V && warp < n_chunks) load_v(warp);
        for (int ch = warp; ch < n_chunks; ch += 4) {
            const int base = ch << 4;
            if (!FA_PREFETCH_K) load_k(ch);
            // ---- S = Q K^T for the two 8-cell tiles ----
            float sacc[2][4];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                sacc[c][0] = sacc[c][1] = sacc[c][2] = sacc[c][3] = 0.0f;
#pragma unroll
                for (int u = 0; u < NU; ++u) {
                    mma_f16(sacc[c], qa0[2 * u], 0u, qa2[2 * u], 0u, kr[c][u].x, kr[c][u].y);
                    mma_f16(sacc[c], qa0[2 * u + 1], 0u, qa2[2 * u + 1], 0u, kr[c][u].z, kr[c][u].w);
                }
            }
            // V rows of cells 2t, 2t+1, 2t+8, 2t+9 (already on their way with PREFETCH_V)
            if (!PREFETCH_V) load_v(ch);
            // the next chunk's K rows travel during the softmax and the P V MMAs of this one
            if (FA_PREFETCH_K && ch + 4 < n_chunks) load_k(ch + 4);
            // ---- scores of head g for cells base + {2t, 2t+1, 8+2t, 9+2t} ----
            float sc[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int idx = base + 2 * t + (i & 1) + 8 * (i >> 1);
                float a = sacc[i >> 1][i & 1] * p.scale;
                if (p.softcap != 0.0f) a = p.softcap * tanhf(a);
                if (idx < count) {
                    if (decltype(soft)::value) a += slope * __half2float(mrow[cell_list[idx]]);
                } else {
                    a = -CUDART_INF_F;
                }
                sc[i] = a;
            }
            float mx = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float m_new = fmaxf(m_run, mx);   // finite: a chunk holds at least one participating cell
            const float alpha = __expf(m_run - m_new);
            float pr[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) pr[i] = __expf(sc[i] - m_new);
            l_run = l_run * alpha + (pr[0] + pr[1]) + (pr[2] + pr[3]);
            m_run = m_new;
            // P^T fragments, fp16 hi + lo
            const __half2 h01 = __floats2half2_rn(pr[0], pr[1]), h23 = __floats2half2_rn(pr[2], pr[3]);
            const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
            const uint32_t b0h = *reinterpret_cast<const uint32_t *>(&h01), b1h = *reinterpret_cast<const uint32_t *>(&h23);
            const uint32_t b0l = pack_half2(pr[0] - f01.x, pr[1] - f01.y), b1l = pack_half2(pr[2] - f23.x, pr[3] - f23.y);
            // rescale O^T columns (heads 2t, 2t+1) when some head's maximum moved
            if (__any_sync(0xffffffffu, alpha != 1.0f)) {
                const float a_lo = __shfl_sync(0xffffffffu, alpha, (2 * t) * 4);
                const float a_hi = __shfl_sync(0xffffffffu, alpha, (2 * t + 1) * 4);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    oacc[q][0] *= a_lo; oacc[q][1] *= a_hi; oacc[q][2] *= a_lo; oacc[q][3] *= a_hi;
                }
            }
            // ---- O^T += V^T P^T ----
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint32_t sel = (q & 1) ? 0x7632u : 0x5410u;
                const uint32_t *wA0 = reinterpret_cast<const uint32_t *>(&vr[0][0]), *wB0 = reinterpret_cast<const uint32_t *>(&vr[1][0]);
                const uint32_t *wC0 = reinterpret_cast<const uint32_t *>(&vr[2][0]), *wD0 = reinterpret_cast<const uint32_t *>(&vr[3][0]);
                const uint32_t a0 = __byte_perm(wA0[q >> 1], wB0[q >> 1], sel);
                const uint32_t a2 = __byte_perm(wC0[q >> 1], wD0[q >> 1], sel);
                uint32_t a1 = 0u, a3 = 0u;
                if (NR == 2) {
                    const uint32_t *wA1 = reinterpret_cast<const uint32_t *>(&vr[0][NR - 1]), *wB1 = reinterpret_cast<const uint32_t *>(&vr[1][NR - 1]);
                    const uint32_t *wC1 = reinterpret_cast<const uint32_t *>(&vr[2][NR - 1]), *wD1 = reinterpret_cast<const uint32_t *>(&vr[3][NR - 1]);
                    a1 = __byte_perm(wA1[q >> 1], wB1[q >> 1], sel);
                    a3 = __byte_perm(wC1[q >> 1], wD1[q >> 1], sel);
                }
                mma_f16(oacc[q], a0, a1, a2, a3, b0h, b1h);
                mma_f16(oacc[q], a0, a1, a2, a3, b0l, b1l);
            }
            if (PREFETCH_V && ch + 4 < n_chunks) load_v(ch + 4);
        }
        __syncthreads();
    }
    };
    if (VOTED || mrow) walk(std::true_type{});
    else walk(std::false_type{});

    pdl_trigger();
    // ---- merge the four warps ----
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
    if (t == 0) {
        merge_m[warp][g] = m_run;
        merge_l[warp][g] = l_run;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        merge_acc[warp][2 * t][8 * g + q] = oacc[q][0];
        merge_acc[warp][2 * t + 1][8 * g + q] = oacc[q][1];
        if (NR == 2) {
            merge_acc[warp][2 * t][64 + 8 * g + q] = oacc[q][2];
            merge_acc[warp][2 * t + 1][64 + 8 * g + q] = oacc[q][3];
        }
    }
    __syncthreads();
    for (int i = tid; i < G * D; i += FA_THREADS) {
        const int h = i / D, d = i - h * D;
        float mn = -CUDART_INF_F;
#pragma unroll
        for (int wv = 0; wv < 4; ++wv) mn = fmaxf(mn, merge_m[wv][h]);
        float a = 0.0f, ls = 0.0f;
#pragma unroll
        for (int wv = 0; wv < 4; ++wv) {
            const float scl = (merge_m[wv][h] == -CUDART_INF_F) ? 0.0f : expf(merge_m[wv][h] - mn);
            a += merge_acc[wv][h][d] * scl;
            ls += merge_l[wv][h] * scl;
        }
        const int64_t head = h0 + h;
        if (CLUSTER) {
            merge_acc[0][h][d] = a;   // (this thread was the one to read it)
            if (d == 0) {
                part_m[h] = mn;
                part_l[h] = ls;
            }
        } else if (ns_j == 1 && !p.parts) {
            fattn_store_out<D, QUANT>(p, j, head, d, a * (1.0f / ls));
        } else {
            float *pp = p.partial + ((j * p.H + head) * p.nsplit + split) * (D + 2);
            pp[d] = a;
            if (d == 0) {
                pp[D] = mn;
                pp[D + 1] = ls;
            }
        }
    }
    if (CLUSTER) {   // a warp per 32 elements of a head, dealt out over the cluster; the order of fattn_combine_kernel
        const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
        cluster.sync();
        for (int b = split * (FA_THREADS / 32) + warp; b < G * (D / 32); b += p.nsplit * (FA_THREADS / 32)) {
            const int h = b / (D / 32), d = (b % (D / 32)) * 32 + lane;
            float m[FA_CLUSTER_MAX], l[FA_CLUSTER_MAX], v[FA_CLUSTER_MAX], mn = -CUDART_INF_F;
#pragma unroll
            for (int s = 0; s < FA_CLUSTER_MAX; ++s) {
                const int from = min(s, p.nsplit - 1);
                m[s] = *cluster.map_shared_rank(&part_m[h], from);
                l[s] = *cluster.map_shared_rank(&part_l[h], from);
                v[s] = *cluster.map_shared_rank(&merge_acc[0][h][d], from);
            }
#pragma unroll
            for (int s = 0; s < FA_CLUSTER_MAX; ++s) mn = fmaxf(mn, m[s]);
            float a = 0.0f, ls = 0.0f;
#pragma unroll
            for (int s = 0; s < FA_CLUSTER_MAX; ++s) {
                const float f = s >= p.nsplit || m[s] == -CUDART_INF_F ? 0.0f : expf(m[s] - mn);
                a = fmaf(v[s], f, a);
                ls = fmaf(l[s], f, ls);
            }
            fattn_store_out<D, QUANT>(p, j, h0 + h, d, a * (1.0f / ls));
        }
        cluster.sync();   // its shared memory is read until here
    }
}

// The splits of a token as a cluster, where there are at most FA_CLUSTER_MAX of them and the whole grid is resident (a second wave of
// clusters costs more than the combine pass: 30 sequences of the 1B architecture, 480 CTAs, 1631 us a step against 1528): no partial
// results in memory, no second launch.  The CTAs meet twice, after their parts are in shared memory and before they leave.  Bound by
// latency; D = 64 has the registers to ask for the next chunk's V rows early.  us per decode step on B200, combine pass / cluster: 1B, one
// sequence (2 splits) 761 / 741; 1B, 16 sequences 1323 / 1222; 8B, seven sequences 2612 / 2520.  With two CTAs an SM and V rows asked for early at
// D = 128 as well, the seven sequences took 2642.
template <int D, bool QUANT>
static void launch_mma_cluster(dim3 grid, cudaStream_t st, FattnParams p) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(FA_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = grid.z;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&cfg, fattn_mma_kernel<D, QUANT, true>, p);
}

// ---- validation variant: the reference's own order of operations ------------------------------------
// One warp per (token, head) walks the unmasked cells in ascending order and reproduces
// lm_ggml_compute_forward_flash_attn_ext_f16 step by step (cactus/ggml-cpu/ops.cpp:7072-7152) as the x86
// AVX2 build executes it: Q rounded to fp16; the K.Q dot as 4 x 8 fp32 FMA lanes folded in the order of
// LM_GGML_F32x8_REDUCE (lane l of the warp is accumulator l/8, SIMD lane l%8); scale and mask applied with one
// FMA; the output accumulator kept in fp16 and rounded after every cell (vec_scale_f16 / vec_mad_f16).
// It exists to show that what separates the fast kernel from the reference is that fp16 accumulator.
template <int D>
__global__ void __launch_bounds__(128) fattn_parity_kernel(FattnParams p) {
    constexpr int E = D / 32;
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t) blockIdx.x * 4 + (threadIdx.x >> 5);   // token * H + head
    if (row >= p.Nq * p.H) return;
    const int64_t j = row / p.H;
    const int h = (int) (row - j * p.H);
    const int hk = h / (int) (p.H / p.Hkv);
    const float *qp = reinterpret_cast<const float *>(reinterpret_cast<const char *>(p.q) + j * p.q_nb_tok + (int64_t) h * p.q_nb_head);
    float qf[E];
    __half acc[E];
#pragma unroll
    for (int i = 0; i < E; ++i) {
        qf[i] = __half2float(__float2half_rn(qp[lane + 32 * i]));
        acc[i] = __float2half_rn(0.0f);
    }
    const uint32_t hh = (uint32_t) h;
    const float slope = (p.max_bias > 0.0f) ? (hh < p.n_head_log2 ? powf(p.m0, (float) (hh + 1)) : powf(p.m1, (float) (2 * (hh - p.n_head_log2) + 1))) : 1.0f;
    float S = 0.0f, M = -CUDART_INF_F;
    const unsigned long long *wrow = p.words ? p.words + j * p.nw : nullptr;
    const __half *mrow = p.mask ? reinterpret_cast<const __half *>(p.mask + j * p.mask_nb_row) : nullptr;
    for (int64_t wi = 0; wi < p.nw; ++wi) {
        unsigned long long bits;
        if (wrow) {
            bits = wrow[wi];
        } else {
            const int64_t left = p.n_kv - wi * 64;
            bits = left >= 64 ? ~0ull : ((1ull << left) - 1ull);
        }
        while (bits) {
            const int b = __ffsll((long long) bits) - 1;
            bits &= bits - 1;
            const int64_t cell = wi * 64 + b;
            const __half *kr = reinterpret_cast<const __half *>(p.k + cell * p.k_nb_cell + (int64_t) hk * p.k_nb_head);
            const __half *vr = reinterpret_cast<const __half *>(p.v + cell * p.v_nb_cell + (int64_t) hk * p.v_nb_head);
            float a = 0.0f;
#pragma unroll
            for (int i = 0; i < E; ++i) a = __fmaf_rn(__half2float(kr[lane + 32 * i]), qf[i], a);
            a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 16));
            a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 8));
            a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 4));
            a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 1));
            a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 2));
            const float mv = mrow ? __fmul_rn(slope, __half2float(mrow[cell])) : 0.0f;
            float s;
            if (p.softcap != 0.0f) {
                s = __fmul_rn(a, p.scale);
                s = __fmul_rn(p.softcap, tanhf(s));
                s = __fadd_rn(s, mv);
            } else {
                s = __fmaf_rn(a, p.scale, mv);
            }
            float ms = 1.0f, vs = 1.0f;
            if (s > M) {
                ms = (float) exp((double) __fsub_rn(M, s));   // correctly rounded, as the host libm's expf is in all but rare cases
                M = s;
#pragma unroll
                for (int i = 0; i < E; ++i) acc[i] = __float2half_rn(__fmul_rn(__half2float(acc[i]), ms));
            } else {
                vs = (float) exp((double) __fsub_rn(s, M));
            }
#pragma unroll
            for (int i = 0; i < E; ++i) acc[i] = __float2half_rn(__fmaf_rn(__half2float(vr[lane + 32 * i]), vs, __half2float(acc[i])));
            S = __fmaf_rn(S, ms, vs);
        }
    }
    const float S_inv = __fdiv_rn(1.0f, S);
#pragma unroll
    for (int i = 0; i < E; ++i) p.dst[row * D + lane + 32 * i] = __fmul_rn(__half2float(acc[i]), S_inv);
}

// Adds a row's KV splits.  A warp per row (ALL), 8 warps per CTA: with a CTA per row most of the time went into starting 16384
// CTAs (512 tokens x 32 heads, 3 splits of 128: 24 us, now 9.5).  Few rows are bound by the chain of one warp, which then takes
// 32 elements of a row.  Lane s has the scale of split s, so the parts themselves are loaded without waiting for it.
constexpr int FC_THREADS = 256, FC_ALL_ROWS = 2048;   // rows from which a warp takes a whole row
template <int D, bool QUANT, bool ALL>
__global__ void __launch_bounds__(FC_THREADS) fattn_combine_kernel(FattnParams p, int ctas_per_token) {
    pdl_prologue(p.early != 0);
    if (p.vote == 1 && fattn_tiled_chosen(p.plan)) return;    // the query-tiled kernel wrote the result
    if (p.vote == 2 && !fattn_tiled_chosen(p.plan)) return;   // this is the query-tiled kernel's combine pass and the per-token kernel worked
    constexpr int E = ALL ? D / 32 : 1, PER_ROW = D / 32 / E;
    const int lane = threadIdx.x & 31;
    const unsigned unit = blockIdx.x * (FC_THREADS / 32) + (threadIdx.x >> 5);
    const int64_t row = unit / PER_ROW;   // token * H + head
    const int d = (int) (unit % PER_ROW) * 32 + lane;
    if (row >= p.Nq * p.H) return;
    const float *pp = p.partial + row * p.nsplit * (D + 2);
    int nsplit = p.nsplit;
    const unsigned H = (unsigned) p.H, tok = (unsigned) row / H, head = (unsigned) row - tok * H;
    if (p.w0 != 0) {   // the splits this token really has; a token with one split was written directly
        const int w0 = fattn_target_words(p, ctas_per_token);
        const int64_t n_words = p.wcount ? (int64_t) p.wcount[tok] : p.nw;
        nsplit = (int) min((int64_t) nsplit, max((int64_t) 1, (n_words + w0 - 1) / w0));
        if (nsplit == 1 && !p.parts) return;
    }
    float ms[2], l[2];   // of splits lane and lane + 32 (at most 64)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int s = lane + 32 * i;
        ms[i] = s < nsplit ? pp[s * (D + 2) + D] : -CUDART_INF_F;
        l[i] = s < nsplit ? pp[s * (D + 2) + D + 1] : 0.0f;
    }
    float mn = fmaxf(ms[0], ms[1]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    float sc[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) sc[i] = ms[i] == -CUDART_INF_F ? 0.0f : expf(ms[i] - mn);
    float a[E], ls = 0.0f;
#pragma unroll
    for (int i = 0; i < E; ++i) a[i] = 0.0f;
#pragma unroll 4
    for (int s = 0; s < nsplit; ++s) {
        const float f = __shfl_sync(0xffffffffu, s < 32 ? sc[0] : sc[1], s & 31), ll = __shfl_sync(0xffffffffu, s < 32 ? l[0] : l[1], s & 31);
#pragma unroll
        for (int i = 0; i < E; ++i) a[i] = fmaf(pp[s * (D + 2) + d + 32 * i], f, a[i]);
        ls = fmaf(ll, f, ls);
    }
#pragma unroll
    for (int i = 0; i < E; ++i) fattn_store_out<D, QUANT>(p, tok, head, d + 32 * i, a[i] * (1.0f / ls));
}
template <int D, bool QUANT>
static void launch_combine(const FattnParams &p, int ctas_per_token, cudaStream_t st) {
    const int64_t rows = p.Nq * p.H;
    if (rows >= FC_ALL_ROWS) launch_pdl(fattn_combine_kernel<D, QUANT, true>, dim3((unsigned) ((rows + 7) / 8)), dim3(FC_THREADS), 0, st, p, ctas_per_token);
    else launch_pdl(fattn_combine_kernel<D, QUANT, false>, dim3((unsigned) ((rows * (D / 32) + 7) / 8)), dim3(FC_THREADS), 0, st, p, ctas_per_token);
}


static int fattn_hgroups(int gqa) { return (gqa + 7) / 8; }   // a CTA takes up to 8 query heads of one KV head

static int fa_sm_count() {   // every device of a process is the same model
    static const int n = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v > 0 ? v : 148;
    }();
    return n;
}

// Decode-sized batches over ragged sequences: one CTA per (token, kv head) makes the longest sequence the kernel's
// duration.  When the grid is small enough for spare CTAs to be cheap (at most two waves), a token whose mask has more
// words than fattn_target_words is cut into up to FA_ADAPTIVE_SPLITS KV splits; the rest are written directly.
static bool fattn_adaptive(int64_t Nq, int64_t Hkv, int hgroups, bool have_index) {
    static const int allow = [] {
        const char *e = getenv("B200_FA_ADAPTIVE");   // opt-in: on the 64-sequence decode batch the cuts cost more than they save
        return (e && atoi(e) == 1) ? 1 : 0;
    }();
    return allow && have_index && Nq * Hkv * hgroups <= 2 * (int64_t) FA_MIN_CTAS * fa_sm_count();
}

static int fattn_nsplit(int64_t Nq, int64_t Hkv, int hgroups, int64_t n_kv) {
    static const int forced = [] {
        const char *e = getenv("B200_FA_NSPLIT");
        return e ? atoi(e) : 0;
    }();
    if (forced > 0) return (int) std::min<int64_t>(forced, 64);
    const int64_t ctas = Nq * Hkv * hgroups;
    const int64_t want = 2 * fa_sm_count();
    if (ctas >= want) return 1;
    int64_t ns = (want + ctas - 1) / ctas;
    // At least 512 cells of the cache to a split.  Where a range is cut is part of the result's last bits, and the next product quantises the
    // result, where a last bit decides whole int8 steps: 128 cells to a split from 1024 cells on are faster (1B architecture, one
    // sequence of 640 cells in 1024, 681 us a step against 748) but moved the logits of every third step by 5e-3 of their norm.
    ns = std::min<int64_t>(ns, std::max<int64_t>(1, n_kv / 512));
    return (int) std::min<int64_t>(ns, 64);
}

int fattn_tile_min_nq();

// KV splits of the query-tiled kernel: enough CTAs for two per SM twice over, a split walks at least 256 cells
static int fattn_tile_nsplit(int64_t Nq, int64_t Hkv, int gqa, int64_t n_kv) {
    int gl = 0;
    while ((1 << gl) < gqa) ++gl;
    const int64_t tiles = (Nq + (64 >> gl) - 1) / (64 >> gl), ctas = tiles * Hkv, want = 4 * (int64_t) fa_sm_count();
    int64_t ns = ctas >= want ? 1 : (want + ctas - 1) / ctas;
    ns = std::min<int64_t>(ns, std::max<int64_t>(1, n_kv / 256));
    return (int) std::min<int64_t>(ns, 8);
}
static bool fattn_tile_possible(int64_t Nq, int gqa) {
    const int tile_min = fattn_tile_min_nq();
    return tile_min > 0 && Nq >= tile_min && (gqa & (gqa - 1)) == 0 && gqa >= 2 && gqa <= 16;   // a tile holds 64 / gqa tokens: at most 32
}

// token count from which the query-tiled kernel is considered (B200_FA_TILE_MIN_NQ; 0 turns it off)
int fattn_tile_min_nq() {
    static const int v = [] {
        const char *e = getenv("B200_FA_TILE_MIN_NQ");
        return e ? atoi(e) : 128;
    }();
    return v;
}

}  // namespace b200

using namespace b200;

extern "C" {

// index layout: words [Nq][nw] u64 | list of non-empty word indices [Nq][nw] i32 | their counts [Nq] i32 |
// tokens by decreasing count [Nq] i32 | plan: total words i32, words summed over 16-token groups i32, 1 if the mask
// holds values other than 0 and -inf in participating cells i32, unused, listed tiles of 4, 8, 16, 32 tokens 4 x i32 |
// flag per tile, 4 x [Nq / 4] i32 | lists of flagged tiles, 4 x [Nq / 4] i32 | per token: the row is more than its bits, [Nq] bytes (up to 224 tokens: from byte 32 of the plan on)
static size_t index_list_offset(int64_t Nq, int64_t nw) { return align_up((size_t) Nq * nw * 8, 256); }
static size_t index_count_offset(int64_t Nq, int64_t nw) { return index_list_offset(Nq, nw) + align_up((size_t) Nq * nw * 4, 256); }

static size_t index_order_offset(int64_t Nq, int64_t nw) { return index_count_offset(Nq, nw) + align_up((size_t) Nq * 4, 256); }
static size_t index_plan_offset(int64_t Nq, int64_t nw) { return index_order_offset(Nq, nw) + align_up((size_t) Nq * 4, 256); }

static size_t index_tiles_offset(int64_t Nq, int64_t nw) { return index_plan_offset(Nq, nw) + 256; }
static int64_t index_tiles_stride(int64_t Nq) { return (Nq + 255) / 256 * 64; }   // of one flag array or list, in elements
// only ubatches the query-tiled kernel may take need the vote and its arrays
static bool index_has_tiles(int64_t Nq) { return fattn_tile_min_nq() > 0 && Nq >= fattn_tile_min_nq(); }
constexpr int64_t SOFT_IN_PLAN = 224;   // so many tokens' flags fit behind the plan
static size_t index_end(int64_t Nq, int64_t nw) { return index_tiles_offset(Nq, nw) + (index_has_tiles(Nq) ? 8 * index_tiles_stride(Nq) * 4 : 0); }
static size_t index_soft_offset(int64_t Nq, int64_t nw) { return Nq <= SOFT_IN_PLAN ? index_plan_offset(Nq, nw) + 32 : index_end(Nq, nw); }

size_t b200_mask_index_bytes(int64_t Nq, int64_t n_kv) {
    if (Nq <= 0 || n_kv <= 0) return 0;
    const int64_t nw = (n_kv + 63) / 64;
    return index_end(Nq, nw) + (Nq <= SOFT_IN_PLAN ? 0 : align_up((size_t) Nq, 256));
}

int b200_mask_index_build(const void *mask, int64_t mask_nb_row, int64_t Nq, int64_t n_kv, void *index, size_t index_bytes,
                          b200_stream_t stream) {
    B200_REQUIRE(mask && index && Nq > 0 && n_kv > 0, "bad mask index arguments");
    B200_REQUIRE(is_aligned(mask, 2) && mask_nb_row % 2 == 0 && is_aligned(index, 8), "misaligned mask or index");
    if (index_bytes < b200_mask_index_bytes(Nq, n_kv)) return set_error(B200_E_SCRATCH, "mask index buffer too small");
    const int64_t nw = (n_kv + 63) / 64;
    B200_REQUIRE(Nq <= 0x0fffffff, "too many tokens");
    const cudaStream_t st = (cudaStream_t) stream;
    char *ix = (char *) index;
    int32_t *plan = (int32_t *) (ix + index_plan_offset(Nq, nw)), *wlist = (int32_t *) (ix + index_list_offset(Nq, nw)), *wcount = (int32_t *) (ix + index_count_offset(Nq, nw));
    uint8_t *soft = (uint8_t *) ix + index_soft_offset(Nq, nw);
    const bool vec = is_aligned(mask, 16) && mask_nb_row % 16 == 0;
    int32_t *order = (int32_t *) (ix + index_order_offset(Nq, nw));
    const auto kernel = Nq == 1 ? (vec ? mask_index_kernel<true, true> : mask_index_kernel<false, true>) : (vec ? mask_index_kernel<true, false> : mask_index_kernel<false, false>);
    launch_pdl(kernel, dim3((unsigned) Nq), dim3(MI_THREADS), 0, st, (const __half *) mask, mask_nb_row, n_kv, nw, (unsigned long long *) index, wlist, wcount, soft, order, plan);
    if (int e = check_launch("mask_index")) return e;
    if (Nq > 1) {
        launch_pdl(fattn_plan_kernel, dim3((unsigned) ((Nq + 7) / 8)), dim3(256), 0, st, (const int32_t *) wcount, (const uint8_t *) soft, Nq, order, plan);
        if (int e = check_launch("fattn_plan")) return e;
    }
    if (index_has_tiles(Nq)) {
        int32_t *flags = (int32_t *) ((char *) index + index_tiles_offset(Nq, nw));
        const int64_t stride = index_tiles_stride(Nq);
        launch_pdl(fattn_tile_vote_kernel, dim3((unsigned) ((Nq + 31) / 32)), dim3(256), 0, st, (const int32_t *) wlist, (const int32_t *) wcount, Nq, nw, plan, flags,
                   flags + 4 * stride, stride);
        return check_launch("fattn_tile_vote");
    }
    return B200_OK;
}

size_t b200_flash_attn_scratch_bytes(int64_t D, int64_t H, int64_t Hkv, int64_t Nq, int64_t n_kv) {
    if (D <= 0 || H <= 0 || Hkv <= 0 || Nq <= 0 || n_kv <= 0 || H % Hkv) return 0;
    const int hgroups = fattn_hgroups((int) (H / Hkv));
    int ns = fattn_nsplit(Nq, Hkv, hgroups, n_kv);
    if (ns == 1 && fattn_adaptive(Nq, Hkv, hgroups, true)) ns = FA_ADAPTIVE_SPLITS;
    if (fattn_tile_possible(Nq, (int) (H / Hkv))) ns = std::max(ns, fattn_tile_nsplit(Nq, Hkv, (int) (H / Hkv), n_kv));
    const size_t part = ns > 1 ? align_up((size_t) Nq * H * ns * (D + 2) * sizeof(float), 256) : 0;
    return b200_mask_index_bytes(Nq, n_kv) + part;
}

static int flash_attn_impl(bool parity, int64_t D, int64_t H, int64_t Hkv, int64_t Nq, int64_t n_kv, const float *q, int64_t q_nb_tok,
                           int64_t q_nb_head, const void *k, int64_t k_nb_cell, int64_t k_nb_head, const void *v,
                           int64_t v_nb_cell, int64_t v_nb_head, const void *mask, int64_t mask_nb_row, const void *index,
                           float scale, float max_bias, float logit_softcap, float *dst, void *scratch, size_t scratch_bytes,
                           b200_stream_t stream, void *act = nullptr, size_t act_bytes = 0, int variant = B200_Q8_AVX2) {
    B200_REQUIRE(D == 64 || D == 128, "head size %lld not supported (64 or 128)", (long long) D);
    B200_REQUIRE(H > 0 && Hkv > 0 && H % Hkv == 0 && Nq > 0 && n_kv > 0, "bad attention shape");
    B200_REQUIRE(q && k && v && (dst || act), "null pointer");
    if (act) {
        B200_REQUIRE(!parity && (H * D) % 128 == 0, "quantised output needs H * D to be a multiple of 128");
        B200_REQUIRE(variant == B200_Q8_AVX2 || variant == B200_Q8_SCALAR, "unknown quantiser variant %d", variant);
        B200_REQUIRE(is_aligned(act, 256), "activation scratch must be 256-byte aligned");
        if (act_bytes < act_dims(H * D, Nq).total_bytes) return set_error(B200_E_SCRATCH, "activation scratch too small: %zu < %zu", act_bytes, act_dims(H * D, Nq).total_bytes);
    }
    B200_REQUIRE((mask == nullptr) == (index == nullptr), "mask and mask index must be given together");
    B200_REQUIRE(is_aligned(q, 4) && q_nb_tok % 4 == 0 && q_nb_head % 4 == 0, "misaligned q");
    B200_REQUIRE(is_aligned(k, 16) && k_nb_cell % 16 == 0 && k_nb_head % 16 == 0, "k rows must be 16-byte aligned");
    B200_REQUIRE(is_aligned(v, 16) && v_nb_cell % 16 == 0 && v_nb_head % 16 == 0, "v rows must be 16-byte aligned");
    B200_REQUIRE(!mask || (is_aligned(mask, 2) && mask_nb_row % 2 == 0), "misaligned mask");
    const int gqa = (int) (H / Hkv);
    const int hgroups = fattn_hgroups(gqa);
    int ns = parity ? 1 : fattn_nsplit(Nq, Hkv, hgroups, n_kv);
    int w0 = 0;
    if (!parity && ns == 1 && fattn_adaptive(Nq, Hkv, hgroups, index != nullptr)) {
        ns = FA_ADAPTIVE_SPLITS;
        w0 = -1;
    }
    // a split of fewer than two 64-cell words is more launch and combine work than it saves: a token takes at most half as
    // many splits as it has words (measured on one sequence of 2048 cells: 16 splits 2.41 ms per 8B step, 32 splits 2.45,
    // 8 splits 2.46).  The token's word count is known on the device only, so this needs the mask index.
    if (!parity && ns > 1 && w0 == 0 && index) w0 = FA_MIN_SPLIT_WORDS;
    const size_t part = ns > 1 ? (size_t) Nq * H * ns * (D + 2) * sizeof(float) : 0;
    if (part && (!scratch || scratch_bytes < part)) return set_error(B200_E_SCRATCH, "flash_attn scratch too small: %zu < %zu", scratch_bytes, part);
    B200_REQUIRE(!part || is_aligned(scratch, 16), "scratch must be 16-byte aligned");

    FattnParams p;
    p.H = H; p.Hkv = Hkv; p.Nq = Nq; p.n_kv = n_kv; p.nw = (n_kv + 63) / 64;
    p.q = q; p.q_nb_tok = q_nb_tok; p.q_nb_head = q_nb_head;
    p.k = (const char *) k; p.k_nb_cell = k_nb_cell; p.k_nb_head = k_nb_head;
    p.v = (const char *) v; p.v_nb_cell = v_nb_cell; p.v_nb_head = v_nb_head;
    p.mask = (const char *) mask; p.mask_nb_row = mask_nb_row;
    p.words = (const unsigned long long *) index;
    p.wlist = index ? (const int32_t *) ((const char *) index + index_list_offset(Nq, p.nw)) : nullptr;
    p.wcount = index ? (const int32_t *) ((const char *) index + index_count_offset(Nq, p.nw)) : nullptr;
    p.scale = logit_softcap != 0.0f ? scale / logit_softcap : scale;
    p.max_bias = max_bias; p.softcap = logit_softcap;
    p.n_head_log2 = 1u << (uint32_t) floor(log2((double) H));
    p.m0 = powf(2.0f, -(max_bias) / p.n_head_log2);
    p.m1 = powf(2.0f, -(max_bias / 2.0f) / p.n_head_log2);
    p.dst = dst; p.partial = (float *) scratch; p.nsplit = ns; p.hgroups = hgroups; p.w0 = w0;
    const ActDims ad = act_dims(H * D, Nq);
    p.qout = (uint8_t *) act; p.q_d_offset = ad.d_offset; p.q_nb = ad.nb; p.q_nbp = ad.nbp;
    p.q_variant = variant;
    p.tflags = p.tlist = p.tcount = nullptr;
    p.spread_rows = 0;
    p.order = index ? (const int32_t *) ((const char *) index + index_order_offset(Nq, p.nw)) : nullptr;
    p.plan = index ? (const int32_t *) ((const char *) index + index_plan_offset(Nq, p.nw)) : nullptr;
    p.slots = FA_MIN_CTAS * fa_sm_count();
    B200_REQUIRE(Nq <= 65535, "at most 65535 tokens per call");

    cudaStream_t st = (cudaStream_t) stream;
    if (parity) {
        const unsigned blocks = (unsigned) ((Nq * H + 3) / 4);
        if (D == 128) fattn_parity_kernel<128><<<blocks, 128, 0, st>>>(p);
        else fattn_parity_kernel<64><<<blocks, 128, 0, st>>>(p);
        return check_launch("fattn_parity");
    }
    // Many query tokens: the query-tiled kernel shares every staged K/V chunk between the 64 / gqa tokens of a tile.  That
    // pays when the tokens share their cells (a prompt), not when every token has its own sequence (a large decode batch);
    // with a mask index both kernels are launched and the plan the index holds decides on the device which one works.
    int gqa_log2 = 0;
    while ((1 << gqa_log2) < gqa) ++gqa_log2;
    p.vote = 0;
    p.parts = 0;
    p.early = Nq <= pdl_early_rows() ? 1 : 0;
    if (!act && dst && fattn_tile_possible(Nq, gqa) && p.nw <= 2048) {
        FattnParams pt = p;
        pt.vote = index ? 2 : 0;
        pt.w0 = 0;
        pt.nsplit = fattn_tile_nsplit(Nq, Hkv, gqa, n_kv);
        const size_t tpart = pt.nsplit > 1 ? (size_t) Nq * H * pt.nsplit * (D + 2) * sizeof(float) : 0;
        if (tpart && (!scratch || scratch_bytes < tpart || !is_aligned(scratch, 16))) pt.nsplit = 1;   // an older scratch size: no splits
        const int tile_tokens = 64 >> gqa_log2;
        const int64_t tiles = (Nq + tile_tokens - 1) / tile_tokens;
        if (index) {
            const int k = 4 - gqa_log2;   // tiles of 4 << k tokens
            const int64_t stride = index_tiles_stride(Nq);
            const int32_t *flags = (const int32_t *) ((const char *) index + index_tiles_offset(Nq, p.nw));
            pt.tflags = flags + k * stride;
            pt.tlist = flags + (4 + k) * stride;
            pt.tcount = p.plan + 4 + k;
            // three rounds of CTAs, fewer when there are fewer tokens: one token per CTA for up to some 50 (mixed step of the 8B model, 48
            // tokens: 28.7 ms with one round, 27.7 with three or six; idle CTAs cost 1 us a round)
            pt.spread_rows = (int) std::min<int64_t>(Nq, (9 * (int64_t) fa_sm_count() + Hkv * pt.nsplit - 1) / (Hkv * pt.nsplit));
        }
        dim3 tgrid((unsigned) Hkv, (unsigned) (tiles + pt.spread_rows), (unsigned) pt.nsplit);
        // the opt-in to more than 48 KB of shared memory is per function and device
        static thread_local int tile_smem_dev = -1;
        int dev_now = 0;
        cudaGetDevice(&dev_now);
        if (tile_smem_dev != dev_now) {
            cudaFuncSetAttribute(fattn_tile_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, fattn_tile_smem_bytes(128));
            cudaFuncSetAttribute(fattn_tile_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, fattn_tile_smem_bytes(64));
            tile_smem_dev = dev_now;
        }
        if (D == 128) launch_pdl(fattn_tile_kernel<128>, tgrid, dim3(FT_THREADS), (size_t) fattn_tile_smem_bytes(128), st, pt, gqa_log2);
        else launch_pdl(fattn_tile_kernel<64>, tgrid, dim3(FT_THREADS), (size_t) fattn_tile_smem_bytes(64), st, pt, gqa_log2);
        if (int e = check_launch("fattn_tile")) return e;
        if (pt.nsplit > 1) {
            if (D == 128) launch_combine<128, false>(pt, 1, st);
            else launch_combine<64, false>(pt, 1, st);
            if (int e = check_launch("fattn_combine")) return e;
        }
        if (!index) return B200_OK;   // no mask: every token attends every cell, nothing to vote on
        p.vote = 1;
    }
    dim3 grid((unsigned) (Hkv * hgroups), (unsigned) Nq, (unsigned) ns);
    // With KV splits the combine pass is what quantises: it has the registers for that, the main kernel has not.
    const bool qo = act != nullptr && ns == 1, qc = act != nullptr;
    p.parts = qc && ns > 1 ? 1 : 0;
    if (ns > 1 && ns <= FA_CLUSTER_MAX && (int64_t) grid.x * grid.y * grid.z <= p.slots) {
        if (D == 128) {
            if (act) launch_mma_cluster<128, true>(grid, st, p);
            else launch_mma_cluster<128, false>(grid, st, p);
        } else {
            if (act) launch_mma_cluster<64, true>(grid, st, p);
            else launch_mma_cluster<64, false>(grid, st, p);
        }
        return check_launch("fattn_mma");
    }
    if (p.vote == 1) {
        if (D == 128) launch_pdl(fattn_mma_kernel<128, false, false, true>, grid, dim3(FA_THREADS), 0, st, p);
        else launch_pdl(fattn_mma_kernel<64, false, false, true>, grid, dim3(FA_THREADS), 0, st, p);
    } else if (D == 128) {
        if (qo) launch_pdl(fattn_mma_kernel<128, true>, grid, dim3(FA_THREADS), 0, st, p);
        else launch_pdl(fattn_mma_kernel<128, false>, grid, dim3(FA_THREADS), 0, st, p);
    } else {
        if (qo) launch_pdl(fattn_mma_kernel<64, true>, grid, dim3(FA_THREADS), 0, st, p);
        else launch_pdl(fattn_mma_kernel<64, false>, grid, dim3(FA_THREADS), 0, st, p);
    }
    if (int e = check_launch("fattn_mma")) return e;
    if (ns > 1) {
        const int cpt = (int) (Hkv * hgroups);
        if (D == 128) {
            if (qc) launch_combine<128, true>(p, cpt, st);
            else launch_combine<128, false>(p, cpt, st);
        } else {
            if (qc) launch_combine<64, true>(p, cpt, st);
            else launch_combine<64, false>(p, cpt, st);
        }
        return check_launch("fattn_combine");
    }
    return B200_OK;
}

int b200_flash_attn_ext_indexed(int64_t D, int64_t H, int64_t Hkv, int64_t Nq, int64_t n_kv, const float *q, int64_t q_nb_tok,
                                int64_t q_nb_head, const void *k, int64_t k_nb_cell, int64_t k_nb_head, const void *v,
                                int64_t v_nb_cell, int64_t v_nb_head, const void *mask, int64_t mask_nb_row, const void *index,
                                float scale, float max_bias, float logit_softcap, float *dst, void *scratch, size_t scratch_bytes,
                                b200_stream_t stream) {
    return flash_attn_impl(false, D, H, Hkv, Nq, n_kv, q, q_nb_tok, q_nb_head, k, k_nb_cell, k_nb_head, v, v_nb_cell, v_nb_head, mask, mask_nb_row,
                           index, scale, max_bias, logit_softcap, dst, scratch, scratch_bytes, stream);
}

int b200_flash_attn_ext_quant(int64_t D, int64_t H, int64_t Hkv, int64_t Nq, int64_t n_kv, const float *q, int64_t q_nb_tok,
                              int64_t q_nb_head, const void *k, int64_t k_nb_cell, int64_t k_nb_head, const void *v,
                              int64_t v_nb_cell, int64_t v_nb_head, const void *mask, int64_t mask_nb_row, const void *index,
                              float scale, float max_bias, float logit_softcap, float *dst, void *act, size_t act_bytes, int variant,
                              void *scratch, size_t scratch_bytes, b200_stream_t stream) {
    B200_REQUIRE(act, "null activation scratch");
    return flash_attn_impl(false, D, H, Hkv, Nq, n_kv, q, q_nb_tok, q_nb_head, k, k_nb_cell, k_nb_head, v, v_nb_cell, v_nb_head, mask, mask_nb_row,
                           index, scale, max_bias, logit_softcap, dst, scratch, scratch_bytes, stream, act, act_bytes, variant);
}

int b200_flash_attn_ext_parity(int64_t D, int64_t H, int64_t Hkv, int64_t Nq, int64_t n_kv, const float *q, int64_t q_nb_tok,
                               int64_t q_nb_head, const void *k, int64_t k_nb_cell, int64_t k_nb_head, const void *v,
                               int64_t v_nb_cell, int64_t v_nb_head, const void *mask, int64_t mask_nb_row, const void *index,
                               float scale, float max_bias, float logit_softcap, float *dst, b200_stream_t stream) {
    return flash_attn_impl(true, D, H, Hkv, Nq, n_kv, q, q_nb_tok, q_nb_head, k, k_nb_cell, k_nb_head, v, v_nb_cell, v_nb_head, mask, mask_nb_row,
                           index, scale, max_bias, logit_softcap, dst, nullptr, 0, stream);
}

int b200_flash_attn_ext(int64_t D, int64_t H, int64_t Hkv, int64_t Nq, int64_t n_kv, const float *q, int64_t q_nb_tok,
                        int64_t q_nb_head, const void *k, int64_t k_nb_cell, int64_t k_nb_head, const void *v, int64_t v_nb_cell,
                        int64_t v_nb_head, const void *mask, int64_t mask_nb_row, float scale, float max_bias, float logit_softcap,
                        float *dst, void *scratch, size_t scratch_bytes, b200_stream_t stream) {
    const size_t ib = mask ? b200_mask_index_bytes(Nq, n_kv) : 0;
    if (mask) {
        if (!scratch || scratch_bytes < ib) return set_error(B200_E_SCRATCH, "flash_attn scratch too small for the mask index");
        B200_REQUIRE(is_aligned(scratch, 256), "scratch must be 256-byte aligned");
        if (int e = b200_mask_index_build(mask, mask_nb_row, Nq, n_kv, scratch, ib, stream)) return e;
    }
    return b200_flash_attn_ext_indexed(D, H, Hkv, Nq, n_kv, q, q_nb_tok, q_nb_head, k, k_nb_cell, k_nb_head, v, v_nb_cell, v_nb_head,
                                       mask, mask_nb_row, mask ? scratch : nullptr, scale, max_bias, logit_softcap, dst,
                                       scratch ? (char *) scratch + ib : nullptr, scratch_bytes > ib ? scratch_bytes - ib : 0, stream);
}

}  // extern "C"
