// FLASH_ATTN_EXT for ubatches with many query tokens (prefill): query-tiled kernel.
//
// Same computation as fattn_mma_kernel (lm_ggml_compute_forward_flash_attn_ext_f16, cactus/ggml-cpu/ops.cpp:6948-7165),
// different work split.  The decode kernel gives every (token, kv-head) its own CTA, so the tokens of one prompt walk the
// same K/V rows once each.  Here a CTA owns a tile of consecutive tokens of the ubatch and one kv-head: 4 warps x 16 MMA
// rows, a row being one (token, query head of the group) pair -- 16 / gqa tokens per warp, 64 / gqa per CTA.  The CTA walks
// the union of its tokens' cells (the OR of their mask words) in chunks of 32 cells; a chunk's K and V rows are staged in
// shared memory once (cp.async, three stages) and used by all 64 rows.  A row's own mask value (-inf outside its
// sequence and beyond its position) is added to every score, so the causal triangle and ragged tiles that straddle two
// sequences need no special case.  When the mask holds nothing but 0 and -inf (the index build records that) the row's
// mask value comes from its mask-word bits (turned, once per round of 1024 cells, into 32 bits per token and chunk in
// shared memory) instead of from the f16 mask in global memory.  Long tiles are cut into KV splits (grid z): split z takes every nsplit-th
// chunk of the union list, the partial (max, sum, accumulator) triples go to scratch and fattn_combine_kernel finishes.
//   S = Q K^T   m16n8k16, Q rounded to fp16 as the reference rounds it, K fragments from the staged rows through ldmatrix
//   online softmax per row (the four lanes of a row share max and sum through two shuffles)
//   O += P V    P goes in as fp16 hi + lo parts (two MMAs), which keeps the probabilities at fp32 accuracy; V fragments
//               come from the staged rows through ldmatrix.trans
#pragma once

namespace b200 {

constexpr int FT_THREADS = 128;
constexpr int FT_CHUNK = 32;            // cells per step
constexpr int FT_RW = 16;               // mask words (of 64 cells) listed per round
constexpr int FT_LIST = FT_RW * 64;     // cells listed per round at most
constexpr int FT_STAGES = 3;            // K/V chunks in flight
constexpr int FT_MAX_TILE = 32;         // tokens of a tile at most (gqa 2)
constexpr int FT_MAX_WORDS = 2048;      // mask words of a row at most (131072 cells)

__device__ __forceinline__ void ft_cp16(uint32_t smem, const void *g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem), "l"(g) : "memory");
}
__device__ __forceinline__ void ft_ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

__device__ __forceinline__ void ft_ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// dynamic shared memory of the kernel: FT_STAGES stages of K and V rows
constexpr int fattn_tile_smem_bytes(int D) { return FT_STAGES * 2 * FT_CHUNK * (D * 2 + 16); }   // ft_spread uses them the same way

// ---- the steps of one chunk of 32 cells; rows g and g + 8 of a warp's 16 ----
// S = Q K^T for the four n-tiles of 8 cells (independent accumulator chains)
template <int D>
__device__ __forceinline__ void ft_s(float (&sacc)[4][4], const uint32_t (&qa)[D / 16][4], uint32_t Ks, int lane) {
    constexpr int ROW = D * 2 + 16;
    const uint32_t at = Ks + (uint32_t) ((8 * (lane >> 4) + (lane & 7)) * ROW + ((lane >> 3) & 1) * 16);
#pragma unroll
    for (int c = 0; c < 4; ++c) sacc[c][0] = sacc[c][1] = sacc[c][2] = sacc[c][3] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks)
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
            uint32_t b[4];   // both halves of this k-step for n-tile c, then for n-tile c + 1
            ft_ldmatrix_x4(b, at + (uint32_t) (8 * c * ROW + 32 * ks));
            mma_f16(sacc[c], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b[0], b[1]);
            mma_f16(sacc[c + 1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b[2], b[3]);
        }
}
// Online softmax: element [c][2 i + e] is (row g + 8 i, cell 8 c + 2 t + e of the chunk); rm: which cells row g + 8 i attends
// to; cells: the chunk's cell list.  P comes back as A fragments of two k-steps of 16 cells, fp16 hi + lo.
template <int D>
__device__ __forceinline__ void ft_softmax(const FattnParams &p, float (&sacc)[4][4], const unsigned (&rm)[2], bool binary_mask, const __half *const (&mrow)[2],
                                           const float (&slope)[2], const int *cells, int t, float (&m_run)[2], float (&l_run)[2], float (&o)[D / 8][4],
                                           uint32_t (&ph)[2][4], uint32_t (&pl)[2][4]) {
    float mx[2] = {-CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int x = 8 * c + 2 * t + e;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float a = sacc[c][2 * i + e] * p.scale;
                if (p.softcap != 0.0f) a = p.softcap * tanhf(a);
                if (!((rm[i] >> x) & 1u)) a = -CUDART_INF_F;
                else if (!binary_mask && mrow[i]) a += slope[i] * __half2float(mrow[i][cells[x]]);
                sacc[c][2 * i + e] = a;
                mx[i] = fmaxf(mx[i], a);
            }
        }
    float alpha[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
        const float m_new = fmaxf(m_run[i], mx[i]);
        // a row that has seen no participating cell yet keeps a zero state (exp(-inf - -inf) must not be formed)
        alpha[i] = (m_new == -CUDART_INF_F) ? 1.0f : __expf(m_run[i] - m_new);
        const float m_use = (m_new == -CUDART_INF_F) ? 0.0f : m_new;
        float sum = 0.0f;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float pr = __expf(sacc[c][2 * i + e] - m_use);
                sacc[c][2 * i + e] = pr;
                sum += pr;
            }
        l_run[i] = l_run[i] * alpha[i] + sum;
        m_run[i] = m_new;
    }
    if (__any_sync(0xffffffffu, alpha[0] != 1.0f || alpha[1] != 1.0f)) {
#pragma unroll
        for (int nt = 0; nt < D / 8; ++nt) {
            o[nt][0] *= alpha[0]; o[nt][1] *= alpha[0]; o[nt][2] *= alpha[1]; o[nt][3] *= alpha[1];
        }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float x0 = sacc[c][2 * i], x1 = sacc[c][2 * i + 1];
            const __half2 h = __floats2half2_rn(x0, x1);
            const float2 f = __half22float2(h);
            ph[c >> 1][2 * (c & 1) + i] = *reinterpret_cast<const uint32_t *>(&h);
            pl[c >> 1][2 * (c & 1) + i] = pack_half2(x0 - f.x, x1 - f.y);
        }
}
// O += P V for one k-step of 16 cells, whose V rows start at Vs: V^T fragments of two n-tiles per ldmatrix
template <int D, int NT = D / 8>   // NT n-tiles, from the one Vs points to
__device__ __forceinline__ void ft_pv(float (&o)[NT][4], const uint32_t (&ph)[4], const uint32_t (&pl)[4], uint32_t Vs, int lane) {
    constexpr int ROW = D * 2 + 16;
    const int mi = lane >> 3, mr = lane & 7;
#pragma unroll
    for (int nt = 0; nt < NT; nt += 2) {
        uint32_t vb[4];   // {cells 0-7, cells 8-15} of this k-step for n-tile nt, then for n-tile nt + 1
        ft_ldmatrix_x4_trans(vb, Vs + (uint32_t) ((8 * (mi & 1) + mr) * ROW + (8 * (nt + (mi >> 1))) * 2));
        mma_f16(o[nt], ph[0], ph[1], ph[2], ph[3], vb[0], vb[1]);
        mma_f16(o[nt], pl[0], pl[1], pl[2], pl[3], vb[0], vb[1]);
        mma_f16(o[nt + 1], ph[0], ph[1], ph[2], ph[3], vb[2], vb[3]);
        mma_f16(o[nt + 1], pl[0], pl[1], pl[2], pl[3], vb[2], vb[3]);
    }
}
// The words any of the tile's tokens attends to, ascending, from the tokens' lists (all of them without a mask).  bits: one per
// word.  The whole CTA calls it; the result may be read after it.
__device__ __forceinline__ int ft_union(const FattnParams &p, int64_t tok0, int n_tok, unsigned *bits, unsigned short *uw_index, int *warp_cnt, unsigned short *before = nullptr) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n32 = (int) ((p.nw + 31) / 32);
    if (p.words && p.nw <= FT_THREADS) {   // a thread per word: no dependent loads (list length, list, word)
        unsigned long long w = 0;
        if (tid < p.nw)
#pragma unroll 8
            for (int j = 0; j < n_tok; ++j) w |= p.words[(tok0 + j) * p.nw + tid];
        const unsigned m = __ballot_sync(0xffffffffu, w != 0ull);
        if (lane == 0) bits[warp] = m;
    } else for (int i = tid; i < n32; i += FT_THREADS) bits[i] = p.words ? 0u : (p.nw - 32 * i >= 32 ? ~0u : (1u << (p.nw - 32 * i)) - 1u);
    __syncthreads();
    if (p.words && p.nw > FT_THREADS)
        for (int j = warp; j < n_tok; j += FT_THREADS / 32) {
            const int32_t *wl = p.wlist + (tok0 + j) * p.nw;
            const int n = p.wcount[tok0 + j];
            for (int e = lane; e < n; e += 32) atomicOr(bits + (wl[e] >> 5), 1u << (wl[e] & 31));
        }
    __syncthreads();
    const unsigned mine = tid < n32 ? bits[tid] : 0u;   // FT_MAX_WORDS / 32 <= FT_THREADS
    const int cnt = __popc(mine);
    int pre = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, pre, o);
        if (lane >= o) pre += x;
    }
    if (lane == 31) warp_cnt[warp] = pre;
    __syncthreads();
    int at = pre - cnt, all = 0;
#pragma unroll
    for (int w = 0; w < FT_THREADS / 32; ++w) {
        at += w < warp ? warp_cnt[w] : 0;
        all += warp_cnt[w];
    }
    if (before && tid < n32) before[tid] = (unsigned short) at;
    for (unsigned m = mine; m; m &= m - 1) uw_index[at++] = (unsigned short) (32 * tid + __ffs((int) m) - 1);
    __syncthreads();
    return all;
}
// A finished row pair: O / l, or the split's partial triple
template <int D, int NT = D / 8>   // NT n-tiles, from nt0 on
__device__ __forceinline__ void ft_write(const FattnParams &p, int64_t tok, int head, int split, int i, const float (&o)[NT][4], float m, float l, int t, int nt0 = 0) {
    if (p.nsplit == 1) {
        const float inv = 1.0f / l;
        float *dst = p.dst + (tok * p.H + head) * D + 8 * nt0 + 2 * t;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) *reinterpret_cast<float2 *>(dst + 8 * nt) = make_float2(o[nt][2 * i] * inv, o[nt][2 * i + 1] * inv);
    } else {
        float *pp = p.partial + ((tok * p.H + head) * p.nsplit + split) * (D + 2);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) *reinterpret_cast<float2 *>(pp + 8 * (nt0 + nt) + 2 * t) = make_float2(o[nt][2 * i], o[nt][2 * i + 1]);
        if (t == 0 && nt0 == 0) {
            pp[D] = m;
            pp[D + 1] = l;
        }
    }
}

struct FtTileShared {
    int cell_list[FT_LIST];                    // the cells of this round, ascending
    unsigned short cell_kb[FT_LIST];           // where each sits among the round's words: 64 * slot + bit
    unsigned short uw_index[FT_MAX_WORDS];     // the mask words any token of the tile attends to, ascending
    unsigned long long tile_words[FT_MAX_TILE][FT_RW];   // the round's words, token by token
    unsigned long long ubits[FT_RW];           // their union
    int wbase[FT_RW];                          // cells listed before each word
    unsigned rmask[FT_MAX_TILE][FT_LIST / FT_CHUNK];   // per token and chunk: which of the chunk's 32 cells the token attends to
    unsigned bits[FT_MAX_WORDS / 32];
    int list_count, warp_cnt[FT_THREADS / 32];
};
struct FtSpreadShared {
    unsigned short uw_index[FT_MAX_WORDS];
    unsigned bits[FT_MAX_WORDS / 32];
    unsigned short before[FT_MAX_WORDS / 32];   // union words before each 32
    int warp_cnt[FT_THREADS / 32];
    alignas(16) short list[FT_THREADS / 32][FT_LIST];     // per warp: the round's union positions, 64 * slot + bit of a cell its token attends to or -1
    int cells[FT_THREADS / 32][4][FT_CHUNK];   // per warp: the cells of the chunk at work and of the next two
    float scores[2][16][FT_CHUNK + 4];           // of the chunk at work: a warp computes 8 cells, all warps read 32
};

// Tokens of tiles whose tokens share few cells (decode tokens beside a prompt, in which a shared walk of the union would have
// every token step over all the others' cells): one CTA per token and KV head, over the chunks the token attends to.  The chunks
// are those of the shared walk -- 32 neighbours in the tile's union list, every nsplit-th to each split -- and a chunk without a
// cell of the token would have changed nothing, so results are the same bits.
// What bounds it: the chain of the longest token, chunk after chunk.  So the four warps share each chunk: 8 cells of S each, the
// softmax by all of them (every warp needs P), a quarter of D of P V each; three chunks in the ring.  One token of 2048 cells
// beside a 464-token prompt (32 heads of 128, 8 KV heads; the prompt alone 51 us): 107 us with a warp per token, 69 so; 48
// tokens of 16 to 2048 cells 141 / 127.  (Many short ones were better off with a warp each: 48 of 64 cells 54 / 67.)
template <int D>
__device__ __forceinline__ void ft_spread(const FattnParams &p, int gqa_log2, FtSpreadShared &sh, uint8_t *kv_s) {
    constexpr int KS = D / 16, NT = D / 32, ROW = D * 2 + 16;   // NT: n-tiles of a warp
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int gqa = 1 << gqa_log2, tile_tok = 64 >> gqa_log2;
    const int hk = blockIdx.x, split = blockIdx.z, nsplit = p.nsplit;
    const bool binary_mask = p.plan[2] == 0;
    const char *kbase = p.k + (int64_t) hk * p.k_nb_head, *vbase = p.v + (int64_t) hk * p.v_nb_head;
    const uint32_t kv_u32 = (uint32_t) __cvta_generic_to_shared(kv_s);
    short *list = sh.list[warp];
    // a contiguous share of the tokens: neighbours have their tile's union in common
    const int n_units = *p.tcount * tile_tok, unit1 = (int) (((int64_t) blockIdx.y + 1) * n_units / p.spread_rows);
    int last_tile = -1, n_uw = 0;
    for (int unit = (int) ((int64_t) blockIdx.y * n_units / p.spread_rows); unit < unit1; ++unit) {
        const int tile = p.tlist[unit / tile_tok];
        const int64_t tok0 = (int64_t) tile * tile_tok, tok = tok0 + unit % tile_tok;
        if (tok >= p.Nq) continue;
        __syncthreads();   // the lists and scores of the unit before are no longer read
        if (tile != last_tile) n_uw = ft_union(p, tok0, (int) min((int64_t) tile_tok, p.Nq - tok0), sh.bits, sh.uw_index, sh.warp_cnt, sh.before);
        last_tile = tile;
        const int n_tok = (int) min((int64_t) tile_tok, p.Nq - tok0);
        uint32_t qa[KS][4];
        int head[2];
        bool live[2];
        float slope[2];
        const __half *mrow[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {   // row r is head r of the group
            const int r = g + 8 * i;
            live[i] = r < gqa;
            head[i] = hk * gqa + (live[i] ? r : 0);
            const float *qp = reinterpret_cast<const float *>(reinterpret_cast<const char *>(p.q) + tok * p.q_nb_tok + (int64_t) head[i] * p.q_nb_head);
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                const float2 lo = live[i] ? *reinterpret_cast<const float2 *>(qp + 16 * ks + 2 * t) : make_float2(0.f, 0.f);
                const float2 hi = live[i] ? *reinterpret_cast<const float2 *>(qp + 16 * ks + 8 + 2 * t) : make_float2(0.f, 0.f);
                qa[ks][i] = pack_half2(lo.x, lo.y);
                qa[ks][2 + i] = pack_half2(hi.x, hi.y);
            }
            const uint32_t hh = (uint32_t) head[i];
            slope[i] = (p.max_bias > 0.0f) ? (hh < p.n_head_log2 ? powf(p.m0, (float) (hh + 1)) : powf(p.m1, (float) (2 * (hh - p.n_head_log2) + 1))) : 1.0f;
            mrow[i] = live[i] && p.mask ? reinterpret_cast<const __half *>(p.mask + tok * p.mask_nb_row) : nullptr;
        }
        float o[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) o[nt][0] = o[nt][1] = o[nt][2] = o[nt][3] = 0.0f;
        float m_run[2] = {-CUDART_INF_F, -CUDART_INF_F}, l_run[2] = {0.0f, 0.0f};

        // the chunks of this split with a cell of the token, one after the other: rm and, in sh.cells[warp][b], 32 cells (where the
        // token does not attend, one that it does attend)
        int r0 = 0, chunk = 0, n_chunks = 0;   // r0: the round whose list is built
        const int32_t *wl = p.wlist + tok * p.nw;
        const int n_wl = p.wcount[tok];
        int entry = 0, wl_at = 0;              // the token's words up to `entry` are in rounds up to r0; lane i holds the word wl_at + i
        int wl_mine = lane < n_wl ? wl[lane] : 0;
        auto next_chunk = [&](int b) -> unsigned {
            while (true) {
                if (chunk >= n_chunks) {   // on to the next round in which the token attends to a word
                    if (entry >= n_wl) return 0u;
                    if (entry - wl_at >= 32) {
                        wl_at = entry;
                        wl_mine = wl_at + lane < n_wl ? wl[wl_at + lane] : 0;
                    }
                    const int first = __shfl_sync(0xffffffffu, wl_mine, entry - wl_at);
                    r0 = (sh.before[first >> 5] + __popc(sh.bits[first >> 5] & ((1u << (first & 31)) - 1u))) & ~(FT_RW - 1);
                    unsigned long long own = 0, all = 0;
                    const int k = lane & 15;
                    if (r0 + k < n_uw) {
                        const unsigned long long *w = p.words + sh.uw_index[r0 + k];
                        own = w[tok * p.nw];
#pragma unroll 8
                        for (int j = lane >> 4; j < n_tok; j += 2) all |= w[(tok0 + j) * p.nw];
                    }
                    unsigned own_set = __ballot_sync(0xffffffffu, own != 0ull) & 0xffffu;
                    entry += __popc(own_set);
                    all |= __shfl_xor_sync(0xffffffffu, all, 16);
                    const int cnt = __popcll(all);
                    int pre = cnt;
#pragma unroll
                    for (int s = 1; s < 16; s <<= 1) {
                        const int x = __shfl_up_sync(0xffffffffu, pre, s, 16);
                        if (k >= s) pre += x;
                    }
                    const int total = __shfl_sync(0xffffffffu, pre, 15);
                    n_chunks = (total + FT_CHUNK - 1) / FT_CHUNK;
                    chunk = split;
                    for (int i = lane; i < n_chunks * (FT_CHUNK / 8); i += 32) reinterpret_cast<uint4 *>(list)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
                    __syncwarp();
                    for (; own_set; own_set &= own_set - 1) {
                        const int w = __ffs((int) own_set) - 1;
                        const unsigned long long ow = __shfl_sync(0xffffffffu, own, w);
                        const unsigned long long aw = __shfl_sync(0xffffffffu, all, w);
                        const int base = __shfl_sync(0xffffffffu, pre - cnt, w);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int bit = lane + 32 * h;
                            if ((ow >> bit) & 1ull) list[base + __popcll(aw & ((1ull << bit) - 1ull))] = (short) (64 * w + bit);
                        }
                    }
                    __syncwarp();
                }
                for (; chunk < n_chunks; chunk += nsplit) {
                    const int v = list[chunk * FT_CHUNK + lane];
                    const unsigned rm = __ballot_sync(0xffffffffu, v >= 0);
                    if (!rm) continue;
                    int cell = v >= 0 ? (int) sh.uw_index[r0 + (v >> 6)] * 64 + (v & 63) : 0;
                    const int some = __shfl_sync(0xffffffffu, cell, __ffs((int) rm) - 1);
                    sh.cells[warp][b][lane] = v >= 0 ? cell : some;
                    __syncwarp();
                    chunk += nsplit;
                    return rm;
                }
            }
        };
        // a warp copies 8 rows of K and of V of a chunk
        constexpr int PIECES = D / 8, PER = 8 * PIECES / 32;
        auto fetch = [&](int stage, const int *cells) {
            const uint32_t to = kv_u32 + (uint32_t) ((2 * stage) * FT_CHUNK * ROW + 8 * warp * ROW);
#pragma unroll
            for (int n = 0; n < PER; ++n) {
                const int c = lane + 32 * n, r = c / PIECES, piece = c % PIECES;
                const int64_t cell = cells[8 * warp + r];
                ft_cp16(to + (uint32_t) (r * ROW + piece * 16), kbase + cell * p.k_nb_cell + piece * 16);
                ft_cp16(to + (uint32_t) (FT_CHUNK * ROW + r * ROW + piece * 16), vbase + cell * p.v_nb_cell + piece * 16);
            }
        };
        auto commit = [&] { asm volatile("cp.async.commit_group;\n" ::: "memory"); };
        unsigned rm0 = next_chunk(0);
        if (rm0) fetch(0, sh.cells[warp][0]);
        commit();
        unsigned rm1 = next_chunk(1);
        if (rm1) fetch(1, sh.cells[warp][1]);
        commit();
        int s = 0, s2 = 2;   // ring stage of this chunk, of the one after the next
        for (int it = 0; rm0; ++it) {   // (all warps go through the same chunks)
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncthreads();   // the chunk has landed for every warp, and nobody uses the one before any more
            const unsigned rm2 = next_chunk((it + 2) & 3);
            if (rm2) fetch(s2, sh.cells[warp][(it + 2) & 3]);
            commit();
            const uint32_t Ks = kv_u32 + (uint32_t) ((2 * s) * FT_CHUNK * ROW), Vs = Ks + (uint32_t) (FT_CHUNK * ROW);
            float sacc[4][4];
            uint32_t ph[2][4], pl[2][4];
            {   // 8 cells of S
                float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                const uint32_t at = Ks + (uint32_t) ((8 * warp + (lane & 7)) * ROW + (lane >> 3) * 16);
#pragma unroll
                for (int ks = 0; ks < KS; ks += 2) {
                    uint32_t b[4];   // both halves of k-step ks, of ks + 1
                    ft_ldmatrix_x4(b, at + (uint32_t) (32 * ks));
                    mma_f16(a, qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b[0], b[1]);
                    mma_f16(a, qa[ks + 1][0], qa[ks + 1][1], qa[ks + 1][2], qa[ks + 1][3], b[2], b[3]);
                }
                *reinterpret_cast<float2 *>(&sh.scores[it & 1][g][8 * warp + 2 * t]) = make_float2(a[0], a[1]);
                *reinterpret_cast<float2 *>(&sh.scores[it & 1][g + 8][8 * warp + 2 * t]) = make_float2(a[2], a[3]);
            }
            __syncthreads();
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float2 x = *reinterpret_cast<const float2 *>(&sh.scores[it & 1][g + 8 * i][8 * c + 2 * t]);
                    sacc[c][2 * i] = x.x;
                    sacc[c][2 * i + 1] = x.y;
                }
            const unsigned rm[2] = {live[0] ? rm0 : 0u, live[1] ? rm0 : 0u};
            ft_softmax<D / 4>(p, sacc, rm, binary_mask, mrow, slope, sh.cells[warp][it & 3], t, m_run, l_run, o, ph, pl);
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) ft_pv<D, NT>(o, ph[kk], pl[kk], Vs + (uint32_t) (16 * kk * ROW + 16 * NT * warp), lane);
            rm0 = rm1;
            rm1 = rm2;
            s = s == 2 ? 0 : s + 1;
            s2 = s2 == 2 ? 0 : s2 + 1;
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 1);
            l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 2);
            if (live[i]) ft_write<D, NT>(p, tok, head[i], split, i, o, m_run[i], l_run[i], t, NT * warp);
        }
    }
}

template <int D>
__global__ void __launch_bounds__(FT_THREADS, 3) fattn_tile_kernel(FattnParams p, int gqa_log2) {
    pdl_prologue();
    // the first rows of the grid take the listed tiles' tokens (their chains are the longest), the others a tile each that is not listed
    const bool spread = (int) blockIdx.y < p.spread_rows;
    const int info = spread ? *p.tcount : (p.tflags ? p.tflags[(int) blockIdx.y - p.spread_rows] : 0);
    if (p.vote == 2 && !fattn_tiled_chosen(p.plan)) return;   // the tokens share too few cells: the per-token kernel takes this ubatch
    constexpr int KS = D / 16;            // k-steps of S
    constexpr int NT = D / 8;             // n-tiles of O
    constexpr int ROW = D * 2 + 16;       // bytes of a staged K / V row (the pad spreads the 8 rows of a fragment over all banks)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int gqa = 1 << gqa_log2;
    const int tw = 16 >> gqa_log2;                      // tokens per warp
    const int64_t tok0 = (int64_t) ((int) blockIdx.y - p.spread_rows) * (4 * tw);   // first token of the tile
    const int hk = blockIdx.x;
    const int split = blockIdx.z, nsplit = p.nsplit;
    const bool binary_mask = p.words && p.plan && p.plan[2] == 0;   // only 0 / -inf in the mask: a row's bit says it all

    __shared__ union {
        FtTileShared tile;
        FtSpreadShared spread;
    } sh;
    int *const cell_list = sh.tile.cell_list;
    unsigned short *const cell_kb = sh.tile.cell_kb, *const uw_index = sh.tile.uw_index;
    unsigned long long (*const tile_words)[FT_RW] = sh.tile.tile_words, *const ubits = sh.tile.ubits;
    int *const wbase = sh.tile.wbase;
    unsigned (*const rmask)[FT_LIST / FT_CHUNK] = sh.tile.rmask;
    int &list_count = sh.tile.list_count;
    extern __shared__ __align__(16) uint8_t kv_s[];   // [stage][K, V][FT_CHUNK rows of ROW bytes] (dynamic: fattn_tile_smem_bytes)

    if (spread) {
        if (info > 0) ft_spread<D>(p, gqa_log2, sh.spread, kv_s);
        return;
    }
    if (info) return;

    // rows g and g + 8 of this warp: (token, head)
    int64_t tok[2];
    int head[2], tl[2];
    bool live[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = g + 8 * i;
        tl[i] = warp * tw + (r >> gqa_log2);   // token within the tile
        tok[i] = tok0 + tl[i];
        head[i] = hk * gqa + (r & (gqa - 1));
        live[i] = tok[i] < p.Nq;
    }
    // Q as A fragments: a0 = (row g, d 16 ks + 2t, +1), a1 = (row g + 8, same), a2 = (row g, d 16 ks + 8 + 2t, +1), a3 = (row g + 8, same)
    uint32_t qa[KS][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float *qp = reinterpret_cast<const float *>(reinterpret_cast<const char *>(p.q) + (live[i] ? tok[i] : 0) * p.q_nb_tok + (int64_t) head[i] * p.q_nb_head);
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            const float2 lo = live[i] ? *reinterpret_cast<const float2 *>(qp + 16 * ks + 2 * t) : make_float2(0.f, 0.f);
            const float2 hi = live[i] ? *reinterpret_cast<const float2 *>(qp + 16 * ks + 8 + 2 * t) : make_float2(0.f, 0.f);
            qa[ks][i] = pack_half2(lo.x, lo.y);
            qa[ks][2 + i] = pack_half2(hi.x, hi.y);
        }
    }
    float slope[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const uint32_t hh = (uint32_t) head[i];
        slope[i] = (p.max_bias > 0.0f) ? (hh < p.n_head_log2 ? powf(p.m0, (float) (hh + 1)) : powf(p.m1, (float) (2 * (hh - p.n_head_log2) + 1))) : 1.0f;
    }
    const __half *mrow[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) mrow[i] = (p.mask && live[i]) ? reinterpret_cast<const __half *>(p.mask + tok[i] * p.mask_nb_row) : nullptr;

    float o[NT][4];   // [nt][0,1]: row g, d = 8 nt + 2t, +1; [2,3]: row g + 8
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) o[nt][0] = o[nt][1] = o[nt][2] = o[nt][3] = 0.0f;
    float m_run[2] = {-CUDART_INF_F, -CUDART_INF_F}, l_run[2] = {0.0f, 0.0f};   // l: this lane's share of the row sum

    const char *kbase = p.k + (int64_t) hk * p.k_nb_head;
    const char *vbase = p.v + (int64_t) hk * p.v_nb_head;
    const uint32_t kv_u32 = (uint32_t) __cvta_generic_to_shared(kv_s);
    const int n_tile_tok = (int) min((int64_t) (4 * tw), p.Nq - tok0);

    const int n_uw = ft_union(p, tok0, n_tile_tok, sh.tile.bits, uw_index, sh.tile.warp_cnt);

    // one 16-byte piece of a K or V row per copy: D / 8 pieces per row, 32 rows of K then 32 of V.  A thread's copies sit at
    // fixed places of a stage: copy n of thread tid is piece (tid + 128 n) % PIECES of row ((tid + 128 n) / PIECES) % 32.
    constexpr int PIECES = D / 8, COPIES = 2 * FT_CHUNK * PIECES / FT_THREADS, K_COPIES = COPIES / 2;
    const int st_row0 = tid / PIECES, st_piece = tid % PIECES;   // 128 / PIECES rows apart from copy to copy
    const uint32_t st_dst0 = kv_u32 + (uint32_t) (st_row0 * ROW + st_piece * 16);
    auto stage = [&](int chunk, int count, int s) {
#pragma unroll
        for (int n = 0; n < COPIES; ++n) {
            const int which = n / K_COPIES, r = st_row0 + (n % K_COPIES) * (FT_THREADS / PIECES);
            const int64_t cell = cell_list[min(chunk * FT_CHUNK + r, count - 1)];
            const char *src = (which == 0 ? kbase + cell * p.k_nb_cell : vbase + cell * p.v_nb_cell) + st_piece * 16;
            ft_cp16(st_dst0 + (uint32_t) ((s * 2 + which) * (FT_CHUNK * ROW) + (n % K_COPIES) * (FT_THREADS / PIECES) * ROW), src);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    for (int r0 = 0; r0 < n_uw; r0 += FT_RW) {
        __syncthreads();   // the previous round's lists and stages are no longer read
        // ---- the round's words, token by token; their union; the cells in ascending order ----
        for (int e = tid; e < n_tile_tok * FT_RW; e += FT_THREADS) {
            const int j = e / FT_RW, k = e - j * FT_RW;
            unsigned long long w = 0;
            if (r0 + k < n_uw) {
                const int64_t wi = uw_index[r0 + k];
                if (p.words) w = p.words[(tok0 + j) * p.nw + wi];
                else {
                    const int64_t left = p.n_kv - wi * 64;
                    w = left >= 64 ? ~0ull : ((1ull << left) - 1ull);
                }
            }
            tile_words[j][k] = w;
        }
        __syncthreads();
        if (warp == 0) {
            unsigned long long bits = 0;
            if (lane < FT_RW)
                for (int j = 0; j < n_tile_tok; ++j) bits |= tile_words[j][lane];
            const int cnt = __popcll(bits);
            int pre = cnt;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, pre, off);
                if (lane >= off) pre += x;
            }
            if (lane < FT_RW) {
                ubits[lane] = bits;
                wbase[lane] = pre - cnt;
            }
            if (lane == 31) list_count = pre;
        }
        __syncthreads();
        const int count = list_count;
        for (int e = tid; e < FT_LIST; e += FT_THREADS) {
            const int k = e >> 6, b = e & 63;
            const unsigned long long bits = ubits[k];
            if ((bits >> b) & 1ull) {
                const int at = wbase[k] + __popcll(bits & ((1ull << b) - 1ull));
                cell_list[at] = (int) uw_index[r0 + k] * 64 + b;
                cell_kb[at] = (unsigned short) e;
            }
        }
        __syncthreads();
        const int n_chunks = (count + FT_CHUNK - 1) / FT_CHUNK;
        // this split's chunks: split, split + nsplit, ...; FT_STAGES - 1 of them are on their way while one is multiplied
        int issued = 0;
        auto issue = [&] {
            const int c = split + issued * nsplit;
            if (c < n_chunks) stage(c, count, issued % FT_STAGES);
            else asm volatile("cp.async.commit_group;\n" ::: "memory");
            ++issued;
        };
        for (int k = 0; k < FT_STAGES - 1; ++k) issue();
        // ---- which cells of each of this split's chunks every token attends to (while the first chunks travel) ----
        for (int c = split + warp * nsplit; c < n_chunks; c += 4 * nsplit) {   // a warp per chunk, a lane per cell
            const int idx = c * FT_CHUNK + lane, kb = cell_kb[min(idx, count - 1)];
#pragma unroll 4
            for (int j = 0; j < n_tile_tok; ++j) {
                const unsigned m = __ballot_sync(0xffffffffu, idx < count && ((tile_words[j][kb >> 6] >> (kb & 63)) & 1ull));
                if (lane == 0) rmask[j][c] = m;
            }
        }
        int it = 0;
        for (int ch = split; ch < n_chunks; ch += nsplit, ++it) {
            const int s = it % FT_STAGES;
            issue();
            asm volatile("cp.async.wait_group %0;\n" ::"n"(FT_STAGES - 1) : "memory");
            __syncthreads();   // the stage has landed for every thread (and, first time round, the row masks are written)
            const uint32_t Ks = kv_u32 + (uint32_t) ((s * 2) * (FT_CHUNK * ROW)), Vs = Ks + (uint32_t) (FT_CHUNK * ROW);
            unsigned rm[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) rm[i] = live[i] ? rmask[tl[i]][ch] : 0u;
            if (__any_sync(0xffffffffu, (rm[0] | rm[1]) != 0u)) {   // a chunk that none of the warp's rows attends to changes nothing
                float sacc[4][4];
                uint32_t ph[2][4], pl[2][4];
                ft_s<D>(sacc, qa, Ks, lane);
                ft_softmax<D>(p, sacc, rm, binary_mask, mrow, slope, cell_list + ch * FT_CHUNK, t, m_run, l_run, o, ph, pl);
#pragma unroll
                for (int kk = 0; kk < 2; ++kk) ft_pv<D>(o, ph[kk], pl[kk], Vs + (uint32_t) (16 * kk * ROW), lane);
            }
            __syncthreads();   // this stage may be refilled by the copy issued in the next step
        }
    }
    pdl_trigger();
    // ---- finish: every row's sum over its four lanes, then O / l (or the split's partial triple) ----
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 1);
        l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 2);
        if (live[i]) ft_write<D>(p, tok[i], head[i], split, i, o, m_run[i], l_run[i], t);
    }
}

}  // namespace b200
