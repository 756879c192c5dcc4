// Device-side pieces of the unified KV cache bookkeeping that the reference does on the host:
// the attention mask (llama_kv_cache_unified::set_input_kq_mask, cactus/llama-kv-cache.cpp:696-761),
// the K/V store into cache rows (cpy_k / cpy_v, :617-656) addressed by slot index, and greedy argmax over
// logits (the sampler step after llama_get_logits, cactus/cactus_completion.cpp:210).
#include <cooperative_groups.h>
#include <math_constants.h>

#include "common.cuh"

namespace b200 {

// mask[j][i] = 0 if cell i holds token j's sequence and cell_pos[i] <= tok_pos[j], else -inf; rows
// n_tokens..n_rows (the padding to a multiple of 64) are -inf.  One sequence id per cell.
__global__ void __launch_bounds__(256) kq_mask_kernel(const int32_t *__restrict__ cell_pos, const int32_t *__restrict__ cell_seq,
                                                     int64_t n_kv, const int32_t *__restrict__ tok_pos,
                                                     const int32_t *__restrict__ tok_seq, int64_t n_tokens, int64_t n_rows,
                                                     __half *__restrict__ mask, int64_t mask_nb_row) {
    const int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t j = blockIdx.y;
    if (i >= n_kv || j >= n_rows) return;
    unsigned short v = 0xFC00u;  // -inf
    if (j < n_tokens) {
        const int32_t cs = cell_seq[i];
        if (cs >= 0 && cs == tok_seq[j] && cell_pos[i] <= tok_pos[j]) v = 0;
    }
    reinterpret_cast<unsigned short *>(reinterpret_cast<char *>(mask) + j * mask_nb_row)[i] = v;
}

// The same for 8 cells per thread and MASK_ROWS rows per CTA, where 8 cells are 16 aligned bytes: the cells' positions and
// sequences are loaded once and the stores are 16 bytes wide (512 x 65536: 77.6 us with the kernel above, 15.5 with this one).
constexpr int MASK_ROWS = 16;
__global__ void __launch_bounds__(256) kq_mask8_kernel(const int32_t *__restrict__ cell_pos, const int32_t *__restrict__ cell_seq,
                                                      int64_t n_kv, const int32_t *__restrict__ tok_pos,
                                                      const int32_t *__restrict__ tok_seq, int64_t n_tokens, int64_t n_rows,
                                                      __half *__restrict__ mask, int64_t mask_nb_row) {
    pdl_prologue();
    const int64_t i = ((int64_t) blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (i >= n_kv) return;
    int32_t cs[8], cp[8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int4 s = *reinterpret_cast<const int4 *>(cell_seq + i + 4 * h), p = *reinterpret_cast<const int4 *>(cell_pos + i + 4 * h);
        cs[4 * h] = s.x; cs[4 * h + 1] = s.y; cs[4 * h + 2] = s.z; cs[4 * h + 3] = s.w;
        cp[4 * h] = p.x; cp[4 * h + 1] = p.y; cp[4 * h + 2] = p.z; cp[4 * h + 3] = p.w;
    }
    const int64_t j0 = (int64_t) blockIdx.y * MASK_ROWS, j1 = min(n_rows, j0 + MASK_ROWS);
#pragma unroll 4
    for (int64_t j = j0; j < j1; ++j) {
        const bool row = j < n_tokens;
        const int32_t ts = row ? tok_seq[j] : -1, tp = row ? tok_pos[j] : 0;
        uint32_t v[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const bool a = row && cs[2 * x] >= 0 && cs[2 * x] == ts && cp[2 * x] <= tp, b = row && cs[2 * x + 1] >= 0 && cs[2 * x + 1] == ts && cp[2 * x + 1] <= tp;
            v[x] = (a ? 0u : 0xFC00u) | (b ? 0u : 0xFC000000u);
        }
        *reinterpret_cast<uint4 *>(reinterpret_cast<char *>(mask) + j * mask_nb_row + i * 2) = make_uint4(v[0], v[1], v[2], v[3]);
    }
}

__global__ void __launch_bounds__(256) scatter_i32_kernel(int32_t *__restrict__ dst, const int32_t *__restrict__ idx,
                                                         const int32_t *__restrict__ src, int64_t n) {
    const int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[idx[i]] = src[i];
}

__global__ void __launch_bounds__(256) set_rows_f16_kernel(const float *__restrict__ x, int64_t x_nb_row,
                                                          const int32_t *__restrict__ slots, __half *__restrict__ dst,
                                                          int64_t dst_nb_row, int64_t d, int64_t rows) {
    const int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d * rows) return;
    const int64_t r = i / d, c = i - r * d;
    const float v = reinterpret_cast<const float *>(reinterpret_cast<const char *>(x) + r * x_nb_row)[c];
    reinterpret_cast<__half *>(reinterpret_cast<char *>(dst) + (int64_t) slots[r] * dst_nb_row)[c] = __float2half_rn(v);
}

// first index of the maximum of each row (ties: lowest index, as a linear scan finds it).  Bound by latency: the load of a thread's
// elements (16 bytes each where the row allows them) and the reduction.  A few long rows get a cluster of 8 CTAs each, which has 8 x 16 bytes of a
// thread for a vocabulary of 128256, all on their way at once; many rows fill the SMs with a CTA each, and the cluster's barriers only cost.
// us per launch on B200, rows beyond L2 in turn, a CTA of 1024 threads per row / a cluster: 128256 values, 1 row 5.4 / 3.4, 16 rows 10.7 / 6.4, 64 rows 11.9 /
// 8.9, 96 rows 12.7 / 14.2, 512 rows 42.9 / 56.4; 32000 values, 1 row 2.6 / 2.5, 64 rows 4.9 / 5.0, 512 rows 13.5 / 28.8; 320 values, 64 rows 1.8 / 3.5.
template <int CTAS, int THREADS>
__device__ __forceinline__ void argmax_row(const float *__restrict__ x, int64_t x_nb_row, int64_t d, int32_t *__restrict__ out, int64_t r, int part) {
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    if (CTAS > 1) cluster.barrier_arrive();   // (the first CTA's shared memory may be written once it has started: the wait is below)
    pdl_prologue();
    constexpr int WARPS = THREADS / 32, ALL = THREADS * CTAS, UNROLL = CTAS > 1 ? 8 : 4;
    const int tid = threadIdx.x, me = part * THREADS + tid;
    const float *row = reinterpret_cast<const float *>(reinterpret_cast<const char *>(x) + r * x_nb_row);
    float best = -CUDART_INF_F;
    int bi = 0x7fffffff;
    int64_t done = 0;
    if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {
        const int64_t n4 = d >> 2;
        const float4 *row4 = reinterpret_cast<const float4 *>(row);
#pragma unroll UNROLL
        for (int64_t i = me; i < n4; i += ALL) {
            const float4 v = __ldg(row4 + i);
            const int b = (int) (i << 2);
            if (v.x > best) { best = v.x; bi = b; }
            if (v.y > best) { best = v.y; bi = b + 1; }
            if (v.z > best) { best = v.z; bi = b + 2; }
            if (v.w > best) { best = v.w; bi = b + 3; }
        }
        done = n4 << 2;
    }
    for (int64_t i = done + me; i < d; i += ALL) {
        const float v = row[i];
        if (v > best) { best = v; bi = (int) i; }
    }
    // a thread's candidate is the first maximum among its own elements; between threads the lower index wins a tie
    auto fold = [&](int from) {
#pragma unroll
        for (int o = from; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
    };
    __shared__ float sv[WARPS];
    __shared__ int si[WARPS];
    __shared__ float cv[CTAS];   // of the cluster's first CTA: every CTA's candidate
    __shared__ int ci[CTAS];
    fold(16);
    if ((tid & 31) == 0) {
        sv[tid >> 5] = best;
        si[tid >> 5] = bi;
    }
    __syncthreads();
    if (CTAS > 1) cluster.barrier_wait();
    if (tid < 32) {
        best = sv[tid & (WARPS - 1)];
        bi = si[tid & (WARPS - 1)];
        fold(WARPS / 2);
        if (CTAS > 1 && tid == 0) {
            cluster.map_shared_rank(cv, 0)[part] = best;
            cluster.map_shared_rank(ci, 0)[part] = bi;
        }
    }
    if (CTAS > 1) {
        cluster.sync();
        if (tid < 32) {
            best = cv[tid & (CTAS - 1)];
            bi = ci[tid & (CTAS - 1)];
            fold(CTAS / 2);
        }
    }
    if (part == 0 && tid == 0) out[r] = bi == 0x7fffffff ? 0 : bi;   // nothing above -inf: a linear scan stays at index 0
}
constexpr int ARGMAX_CTAS = 8, ARGMAX_CLUSTER_THREADS = 512, ARGMAX_THREADS = 1024;
__global__ void __cluster_dims__(ARGMAX_CTAS, 1, 1) __launch_bounds__(ARGMAX_CLUSTER_THREADS)
argmax_rows_cluster_kernel(const float *__restrict__ x, int64_t x_nb_row, int64_t d, int32_t *__restrict__ out) {
    argmax_row<ARGMAX_CTAS, ARGMAX_CLUSTER_THREADS>(x, x_nb_row, d, out, blockIdx.y, blockIdx.x);
}
__global__ void __launch_bounds__(ARGMAX_THREADS) argmax_rows_kernel(const float *__restrict__ x, int64_t x_nb_row, int64_t d, int32_t *__restrict__ out) {
    argmax_row<1, ARGMAX_THREADS>(x, x_nb_row, d, out, blockIdx.x, 0);
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_kq_mask_build(const int32_t *cell_pos, const int32_t *cell_seq, int64_t n_kv, const int32_t *tok_pos,
                       const int32_t *tok_seq, int64_t n_tokens, void *mask, int64_t mask_nb_row, b200_stream_t stream) {
    B200_REQUIRE(cell_pos && cell_seq && tok_pos && tok_seq && mask && n_kv > 0 && n_tokens > 0, "bad kq_mask arguments");
    B200_REQUIRE(mask_nb_row % 2 == 0 && mask_nb_row >= n_kv * 2, "bad mask row stride");
    const int64_t n_rows = (n_tokens + 63) / 64 * 64;
    if (n_kv % 8 == 0 && mask_nb_row % 16 == 0 && is_aligned(mask, 16) && is_aligned(cell_pos, 16) && is_aligned(cell_seq, 16)) {
        launch_pdl(kq_mask8_kernel, dim3((unsigned) ((n_kv / 8 + 255) / 256), (unsigned) ((n_rows + MASK_ROWS - 1) / MASK_ROWS)), dim3(256), 0, (cudaStream_t) stream,
                   cell_pos, cell_seq, n_kv, tok_pos, tok_seq, n_tokens, n_rows, (__half *) mask, mask_nb_row);
        return check_launch("kq_mask");
    }
    dim3 grid((unsigned) ((n_kv + 255) / 256), (unsigned) n_rows);
    kq_mask_kernel<<<grid, 256, 0, (cudaStream_t) stream>>>(cell_pos, cell_seq, n_kv, tok_pos, tok_seq, n_tokens, n_rows,
                                                            (__half *) mask, mask_nb_row);
    return check_launch("kq_mask");
}

int b200_scatter_i32(int32_t *dst, const int32_t *idx, const int32_t *src, int64_t n, b200_stream_t stream) {
    B200_REQUIRE(dst && idx && src && n >= 0, "bad scatter arguments");
    if (n == 0) return B200_OK;
    scatter_i32_kernel<<<(unsigned) ((n + 255) / 256), 256, 0, (cudaStream_t) stream>>>(dst, idx, src, n);
    return check_launch("scatter_i32");
}

int b200_set_rows_f16(const float *x, int64_t x_nb_row, const int32_t *slots, void *dst, int64_t dst_nb_row, int64_t d,
                      int64_t rows, b200_stream_t stream) {
    B200_REQUIRE(x && slots && dst && d > 0 && rows >= 0 && x_nb_row % 4 == 0 && dst_nb_row % 2 == 0, "bad set_rows arguments");
    if (rows == 0) return B200_OK;
    set_rows_f16_kernel<<<(unsigned) ((d * rows + 255) / 256), 256, 0, (cudaStream_t) stream>>>(x, x_nb_row, slots, (__half *) dst,
                                                                                              dst_nb_row, d, rows);
    return check_launch("set_rows_f16");
}

int b200_argmax_rows(const float *x, int64_t x_nb_row, int64_t d, int64_t rows, int32_t *out, b200_stream_t stream) {
    B200_REQUIRE(x && out && d > 0 && rows >= 0 && x_nb_row % 4 == 0, "bad argmax arguments");
    if (rows == 0) return B200_OK;
    // (where the two cross: argmax_row)
    if (rows <= 64 && d >= 32768)
        launch_pdl(argmax_rows_cluster_kernel, dim3(ARGMAX_CTAS, (unsigned) rows), dim3(ARGMAX_CLUSTER_THREADS), 0, (cudaStream_t) stream, x, x_nb_row, d, out);
    else launch_pdl(argmax_rows_kernel, dim3((unsigned) rows), dim3(ARGMAX_THREADS), 0, (cudaStream_t) stream, x, x_nb_row, d, out);
    return check_launch("argmax_rows");
}

}  // extern "C"
