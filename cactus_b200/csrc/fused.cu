// Fused forms of the small ops between the mul_mats of a llama layer (llm_build_llama, cactus/llama-model.cpp:4517-4671).
// Each one computes exactly what the chain of separate ops computes -- same float operations in the same order -- and
// hands the result to the next mul_mat already quantised, so the intermediate f32 tensors need not be written:
//   residual ADD (ops.cpp:1283-1300) + RMS_NORM (ops.cpp:3268-3316) + MUL by the norm weight + quantize_row_q8_0
//   SILU (ops.cpp:2902-2981) * up + quantize_row_q8_0
//   ROPE of q and k (ops.cpp:5080-5362) + the f32 -> f16 stores of k and v into the cache rows (cpy_k / cpy_v,
//   cactus/llama-kv-cache.cpp:617-656)
#include <algorithm>

#include "common.cuh"

namespace b200 {

// One CTA per (padded) token row, one pass: a thread keeps its groups of 4 elements in registers from the load to the
// quantised store.  The sum of squares is accumulated in the order rms_norm_kernel uses (rms_block_sum), so the
// scale -- and with it every quantised value -- is bit-identical to the unfused chain.
// (x, res and h carry no __restrict__: a graph allocator may hand the same memory to the residual and to the normalised output)
// Bound by latency at few rows (load, reduce, 32 dependent double additions, scale), by memory at many.  One group per thread
// (GMAX 1: rows of up to 4096 elements) fits 32 registers, so two CTAs of 1024 threads share an SM, and the weight is loaded
// with the row; only the first warp adds up the warps' sums and works the scale out, with the exact reciprocal where d is a
// power of two (the same quotient), instead of all of them.  us per launch on B200, before / now: 512 x 4096 17.2 / 11.5, 512 x 2048 10.9 / 9.3.
template <int GMAX>   // groups of 4 elements per thread: d <= 4 GMAX blockDim.x
__global__ void __launch_bounds__(1024, GMAX == 1 ? 2 : 1) add_rms_norm_quantize_kernel(float *x, int64_t x_nb_row, const float *res,
                                                                    int64_t res_nb_row, const float *__restrict__ w, float *h,
                                                                    int64_t h_nb_row, int d, int64_t N, float eps, double inv_d, int64_t nb, int64_t nbp,
                                                                    uint8_t *__restrict__ out, size_t d_offset, int variant, int early) {
    pdl_prologue(early != 0);
    const int64_t n = blockIdx.x;
    const bool row_real = n < N;
    const int groups = d / 4, groups_padded = (int) nbp * 8;
    const bool w_vec = (reinterpret_cast<uintptr_t>(w) & 15) == 0;
    float v[GMAX][4];
    float4 wv[GMAX];
    double sum = 0.0;
    float *xr = row_real ? reinterpret_cast<float *>(reinterpret_cast<char *>(x) + n * x_nb_row) : nullptr;
    const float *rr = (row_real && res) ? reinterpret_cast<const float *>(reinterpret_cast<const char *>(res) + n * res_nb_row) : nullptr;
#pragma unroll
    for (int k = 0; k < GMAX; ++k) {
        const int gi = threadIdx.x + k * blockDim.x;
        v[k][0] = v[k][1] = v[k][2] = v[k][3] = 0.0f;
        wv[k] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        if (row_real && gi < groups) {
            const float4 a = *reinterpret_cast<const float4 *>(xr + gi * 4);
            const float4 b = rr ? *reinterpret_cast<const float4 *>(rr + gi * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (w) wv[k] = w_vec ? __ldg(reinterpret_cast<const float4 *>(w) + gi) : make_float4(w[gi * 4], w[gi * 4 + 1], w[gi * 4 + 2], w[gi * 4 + 3]);
            v[k][0] = a.x; v[k][1] = a.y; v[k][2] = a.z; v[k][3] = a.w;
            if (rr) {
                v[k][0] = v[k][0] + b.x; v[k][1] = v[k][1] + b.y; v[k][2] = v[k][2] + b.z; v[k][3] = v[k][3] + b.w;
                *reinterpret_cast<float4 *>(xr + gi * 4) = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) sum += (double) (v[k][i] * v[k][i]);
        }
    }
    __shared__ double red[32];
    __shared__ float sc_s;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) red[warp] = sum;
    __syncthreads();
    if (warp == 0) {
        double tot = 0.0;
        if (warps == 32) {
#pragma unroll
            for (int i = 0; i < 32; ++i) tot += red[i];
        } else {
#pragma unroll 4
            for (int i = 0; i < warps; ++i) tot += red[i];
        }
        const float mean = (float) (inv_d != 0.0 ? tot * inv_d : tot / (double) d);
        if (lane == 0) sc_s = 1.0f / sqrtf(mean + eps);
    }
    __syncthreads();
    pdl_trigger();
    const float sc = sc_s;
    float *hr = (h && row_real) ? reinterpret_cast<float *>(reinterpret_cast<char *>(h) + n * h_nb_row) : nullptr;
#pragma unroll
    for (int k = 0; k < GMAX; ++k) {
        const int gi = threadIdx.x + k * blockDim.x;
        if (gi >= groups_padded) continue;   // whole 8-lane block groups leave together
        const bool real = row_real && gi < groups;
        float o[4] = {0.f, 0.f, 0.f, 0.f};
        if (real) {
            const float wf[4] = {wv[k].x, wv[k].y, wv[k].z, wv[k].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] = (v[k][i] * sc) * wf[i];   // (without a weight: times one)
            if (hr) *reinterpret_cast<float4 *>(hr + gi * 4) = make_float4(o[0], o[1], o[2], o[3]);
        }
        q8_quantize_store<1>(o, out, d_offset, nb, nbp, n, gi >> 3, gi & 7, real, variant);
    }
}

// silu(gate) * up, quantised; the same index space as quantize_q8_0_kernel: a row per x, 256 groups of 4 elements per y (no
// 64-bit division per thread, which was most of the instructions: 64 x 14336 10.3 / 6.6 us before / now, 512 x 14336 23.6 / 20.3)
__global__ void __launch_bounds__(256) silu_mul_quantize_kernel(const float *gate, const float *up, int64_t nb_row,
                                                               float *dst, int64_t dst_nb_row,
                                                               int64_t N, int64_t nb, int64_t nbp,
                                                               uint8_t *__restrict__ out, size_t d_offset, int variant, int early) {
    pdl_prologue(early == 1);
    const int64_t n = blockIdx.x;
    for (int64_t at = blockIdx.y * 256 + threadIdx.x; at < nbp * 8; at += gridDim.y * 256) {   // whole groups of 8 lanes leave together
        const int j = (int) at & 7;
        const int64_t b = at >> 3;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        const bool real = (n < N) && (b < nb);
        if (real) {
            const float4 a = *reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(gate) + n * nb_row + at * 16);
            const float4 u = *reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(up) + n * nb_row + at * 16);
            const float ga[4] = {a.x, a.y, a.z, a.w}, ua[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float s = ga[i] / (1.0f + expf(-ga[i]));
                v[i] = s * ua[i];
            }
            if (dst) *reinterpret_cast<float4 *>(reinterpret_cast<char *>(dst) + n * dst_nb_row + at * 16) = make_float4(v[0], v[1], v[2], v[3]);
        }
        if (early == 2) pdl_trigger();
        q8_quantize_store<1>(v, out, d_offset, nb, nbp, n, b, j, real, variant);
    }
}

// One CTA per token: the angles as rope_norm_kernel builds them, q rotated into qo (which may be q itself, with the same
// strides), k rotated and stored as f16 into its cache row, v stored as f16 into its cache row.
__global__ void __launch_bounds__(512) rope_store_kernel(const float *q, float *qo, int64_t q_nb_head, int64_t q_nb_tok, const float *__restrict__ k,
                                                        int64_t k_nb_head, int64_t k_nb_tok, const float *__restrict__ v, int64_t v_nb_tok,
                                                        int64_t D, int64_t H, int64_t Hkv, int n_dims, const int32_t *__restrict__ pos,
                                                        const float *__restrict__ ff, float theta_scale, float freq_scale, float attn_factor,
                                                        const int32_t *__restrict__ slots, __half *__restrict__ kc, int64_t kc_nb_row,
                                                        __half *__restrict__ vc, int64_t vc_nb_row, int early) {
    pdl_prologue(early != 0);
    extern __shared__ float cs[];   // [n_dims/2] cos, [n_dims/2] sin
    const int64_t t = blockIdx.x;
    const int half_dims = n_dims / 2;
    const unsigned pairs = (unsigned) (D / 2), n_q = (unsigned) H, n_qk = (unsigned) (H + Hkv), total = (unsigned) (H + (v ? 2 : 1) * Hkv) * pairs;
    auto load = [&](unsigned i) -> float2 {
        const unsigned hh = i / pairs, p = i - hh * pairs;
        if (hh < n_q) return *(reinterpret_cast<const float2 *>(reinterpret_cast<const char *>(q) + t * q_nb_tok + hh * q_nb_head) + p);
        if (hh < n_qk) return *(reinterpret_cast<const float2 *>(reinterpret_cast<const char *>(k) + t * k_nb_tok + (hh - n_q) * k_nb_head) + p);
        return *(reinterpret_cast<const float2 *>(reinterpret_cast<const char *>(v) + t * v_nb_tok) + (hh - n_qk) * pairs + p);
    };
    // the rows travel while the angles are worked out
    constexpr int U = 6;   // 6 x 512 pairs: 32 + 2 x 8 heads of 128
    float2 x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const unsigned i = threadIdx.x + u * blockDim.x;
        x[u] = i < total ? load(i) : make_float2(0.f, 0.f);
    }
    const int64_t slot = slots ? (int64_t) slots[t] : t;   // no slot list: token t goes to row t of the cache pointers given
    for (int i = threadIdx.x; i < 2 * half_dims; i += blockDim.x) {   // first half of the threads: cosines, second half: sines
        const int a = i < half_dims ? i : i - half_dims;
        const float f = ff ? ff[a] : 1.0f;
        // theta_a = pos * theta_scale^a by repeated multiplication, as the reference builds it: every thread walks the chain
        // to its own angle (a multiplication per step, against a store and a barrier when one thread does it for all)
        float theta = (float) pos[t], mine = theta;
#pragma unroll 8
        for (int s = 0; s <= a; ++s) {
            mine = theta;
            theta *= theta_scale;
        }
        const float th = freq_scale * (mine / f);
        cs[i] = (i < half_dims ? cosf(th) : sinf(th)) * attn_factor;
    }
    __syncthreads();
    pdl_trigger();
    __half *krow = reinterpret_cast<__half *>(reinterpret_cast<char *>(kc) + slot * kc_nb_row);
    __half *vrow = reinterpret_cast<__half *>(reinterpret_cast<char *>(vc) + slot * vc_nb_row);
    auto finish = [&](unsigned i, float2 x) {
        const unsigned hh = i / pairs, p = i - hh * pairs;
        float2 r = x;
        if (hh < n_qk && p < (unsigned) half_dims) {
            const float c = cs[p], sn = cs[half_dims + p];
            r = make_float2(x.x * c - x.y * sn, x.x * sn + x.y * c);
        }
        if (hh < n_q) {
            if (p < (unsigned) half_dims || qo != q) *(reinterpret_cast<float2 *>(reinterpret_cast<char *>(qo) + t * q_nb_tok + hh * q_nb_head) + p) = r;
        } else {
            __half *to = hh < n_qk ? krow + (hh - n_q) * D : vrow + (hh - n_qk) * D;
            *reinterpret_cast<__half2 *>(to + 2 * p) = __halves2half2(__float2half_rn(r.x), __float2half_rn(r.y));
        }
    };
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const unsigned i = threadIdx.x + u * blockDim.x;
        if (i < total) finish(i, x[u]);
    }
    for (unsigned i = threadIdx.x + U * blockDim.x; i < total; i += blockDim.x) finish(i, load(i));
}

// The angles of a ubatch's tokens, [token][n_dims/2 cosines, n_dims/2 sines], for rope_store_angles_kernel: every layer rotates by the
// same ones.  theta_a = pos * theta_scale^a by repeated multiplication, as the reference builds it.  With `cell_pos` the tokens' cells are
// entered as well (b200_ubatch_begin): two launches less at the start of a step (with the mask index's plan, one less for a single token: 1B
// architecture, one sequence 694 / 689 us a step).
__global__ void __launch_bounds__(128) rope_angles_kernel(float *__restrict__ angles, int n_dims, const int32_t *__restrict__ pos, const float *__restrict__ ff,
                                                          float theta_scale, float freq_scale, float attn_factor, int32_t *__restrict__ cell_pos, int32_t *__restrict__ cell_seq,
                                                          const int32_t *__restrict__ slots, const int32_t *__restrict__ seq) {
    pdl_prologue();
    if (cell_pos && threadIdx.x == 0) {
        const int32_t slot = slots[blockIdx.x];
        cell_pos[slot] = pos[blockIdx.x];
        cell_seq[slot] = seq[blockIdx.x];
    }
    const int64_t t = blockIdx.x;
    const int half_dims = n_dims / 2;
    for (int i = threadIdx.x; i < n_dims; i += blockDim.x) {
        const int a = i < half_dims ? i : i - half_dims;
        const float f = ff ? ff[a] : 1.0f;
        float theta = (float) pos[t], mine = theta;
#pragma unroll 8
        for (int s = 0; s <= a; ++s) {
            mine = theta;
            theta *= theta_scale;
        }
        const float th = freq_scale * (mine / f);
        angles[t * n_dims + i] = (i < half_dims ? cosf(th) : sinf(th)) * attn_factor;
    }
}

// rope_store_kernel with the angles at hand: nothing to wait for but the rows.  Bound by latency: three CTAs per token for 48 heads of
// 128, and as many threads as a head has pairs (or a multiple), so that a thread needs one angle for all its pairs.  us per launch on
// B200, with the angles worked out in each launch / at hand: 64 tokens 6.4 / 4.1, 1 token 4.9 / 3.7.
constexpr int RA_UNROLL = 4;
__global__ void __launch_bounds__(256) rope_store_angles_kernel(float *q, int64_t q_nb_head, int64_t q_nb_tok, const float *__restrict__ k, int64_t k_nb_head, int64_t k_nb_tok,
                                                               const float *__restrict__ v, int64_t v_nb_tok, int pairs, int H, int Hkv, int n_dims,
                                                               const float *__restrict__ angles, const int32_t *__restrict__ slots, __half *__restrict__ kc, int64_t kc_nb_row,
                                                               __half *__restrict__ vc, int64_t vc_nb_row, int early) {
    if (early) pdl_trigger();
    const int64_t t = blockIdx.x;
    const int half_dims = n_dims / 2, p = threadIdx.x % pairs, per = blockDim.x / pairs;   // heads of one pass
    const int h0 = blockIdx.y * per * RA_UNROLL + threadIdx.x / pairs;
    pdl_prologue();
    const bool turns = p < half_dims;
    const float c = turns ? __ldg(angles + t * n_dims + p) : 1.0f, sn = turns ? __ldg(angles + t * n_dims + half_dims + p) : 0.0f;
    const int64_t slot = slots[t];
    float2 x[RA_UNROLL];
#pragma unroll
    for (int u = 0; u < RA_UNROLL; ++u) {
        const int h = min(h0 + u * per, H + 2 * Hkv - 1);   // (never conditional: a load behind a branch is waited for where it ends)
        const char *row = h < H ? reinterpret_cast<const char *>(q) + t * q_nb_tok + h * q_nb_head
                                : h < H + Hkv ? reinterpret_cast<const char *>(k) + t * k_nb_tok + (h - H) * k_nb_head
                                              : reinterpret_cast<const char *>(v) + t * v_nb_tok + (int64_t) (h - H - Hkv) * pairs * 8;
        x[u] = *(reinterpret_cast<const float2 *>(row) + p);
    }
    pdl_trigger();
#pragma unroll
    for (int u = 0; u < RA_UNROLL; ++u) {
        const int h = h0 + u * per;
        if (h >= H + 2 * Hkv) break;
        const float2 r = h < H + Hkv && turns ? rotate_pair(x[u], c, sn) : x[u];
        if (h < H) {
            if (turns) *(reinterpret_cast<float2 *>(reinterpret_cast<char *>(q) + t * q_nb_tok + h * q_nb_head) + p) = r;
        } else {
            char *row = h < H + Hkv ? reinterpret_cast<char *>(kc) + slot * kc_nb_row + (int64_t) (h - H) * pairs * 4 : reinterpret_cast<char *>(vc) + slot * vc_nb_row + (int64_t) (h - H - Hkv) * pairs * 4;
            *(reinterpret_cast<__half2 *>(row) + p) = __halves2half2(__float2half_rn(r.x), __float2half_rn(r.y));
        }
    }
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_add_rms_norm_quantize(float *x, int64_t x_nb_row, const float *residual, int64_t residual_nb_row, const float *w, float *h,
                               int64_t h_nb_row, int64_t d, int64_t rows, float eps, void *scratch, size_t scratch_bytes, int variant,
                               b200_stream_t stream) {
    B200_REQUIRE(x && scratch && d > 0 && d % 32 == 0 && rows > 0, "bad arguments");
    B200_REQUIRE(x_nb_row % 4 == 0 && residual_nb_row % 4 == 0 && h_nb_row % 4 == 0, "row strides must be multiples of 4 bytes");
    B200_REQUIRE(variant == B200_Q8_AVX2 || variant == B200_Q8_SCALAR, "unknown quantiser variant %d", variant);
    B200_REQUIRE(is_aligned(scratch, 256), "scratch must be 256-byte aligned");
    const ActDims a = act_dims(d, rows);
    if (scratch_bytes < a.total_bytes) return set_error(B200_E_SCRATCH, "scratch too small: %zu < %zu", scratch_bytes, a.total_bytes);
    B200_REQUIRE(d <= 16384, "rows of more than 16384 elements are not supported");
    B200_REQUIRE(x_nb_row % 16 == 0 && residual_nb_row % 16 == 0 && h_nb_row % 16 == 0 && is_aligned(x, 16) && (!residual || is_aligned(residual, 16)) &&
                     (!h || is_aligned(h, 16)) && (!w || is_aligned(w, 4)), "rows must be 16-byte aligned");
    const unsigned grid = (unsigned) (a.n_nt * 8);
    const unsigned threads = rms_threads(d);
    cudaStream_t st = (cudaStream_t) stream;
    const int early = rows <= pdl_early_rows() ? 1 : 0;
    const double inv_d = (d & (d - 1)) == 0 ? 1.0 / (double) d : 0.0;   // a power of two: multiplying by it is the same quotient
    launch_pdl(threads * 4 >= d ? add_rms_norm_quantize_kernel<1> : add_rms_norm_quantize_kernel<4>, dim3(grid), dim3(threads), 0, st, x, x_nb_row, residual, residual_nb_row,
               w, h, h_nb_row, (int) d, rows, eps, inv_d, a.nb, a.nbp, (uint8_t *) scratch, a.d_offset, variant, early);
    return check_launch("add_rms_norm_quantize");
}

int b200_silu_mul_quantize(const float *gate, const float *up, int64_t nb_row, float *dst, int64_t dst_nb_row, int64_t K, int64_t N,
                           void *scratch, size_t scratch_bytes, int variant, b200_stream_t stream) {
    B200_REQUIRE(gate && up && scratch && K > 0 && K % 32 == 0 && N > 0, "bad arguments");
    B200_REQUIRE(nb_row % 16 == 0 && is_aligned(gate, 16) && is_aligned(up, 16) && (!dst || (is_aligned(dst, 16) && dst_nb_row % 16 == 0)),
                 "rows must be 16-byte aligned");
    B200_REQUIRE(variant == B200_Q8_AVX2 || variant == B200_Q8_SCALAR, "unknown quantiser variant %d", variant);
    B200_REQUIRE(is_aligned(scratch, 256), "scratch must be 256-byte aligned");
    const ActDims a = act_dims(K, N);
    if (scratch_bytes < a.total_bytes) return set_error(B200_E_SCRATCH, "scratch too small: %zu < %zu", scratch_bytes, a.total_bytes);
    const dim3 grid((unsigned) (a.n_nt * 8), (unsigned) std::min<int64_t>(65535, (a.nbp * 8 + 255) / 256));
    cudaStream_t st = (cudaStream_t) stream;
    const int early = pdl_quantiser(N);
    launch_pdl(silu_mul_quantize_kernel, grid, dim3(256), 0, st, gate, up, nb_row, dst, dst_nb_row, N, a.nb, a.nbp, (uint8_t *) scratch, a.d_offset, variant, early);
    return check_launch("silu_mul_quantize");
}

int b200_rope_store(float *q, int64_t q_nb_head, int64_t q_nb_tok, const float *k, int64_t k_nb_head, int64_t k_nb_tok, const float *v,
                    int64_t v_nb_tok, int64_t D, int64_t H, int64_t Hkv, int64_t T, int n_dims, const int32_t *pos, const float *freq_factors,
                    float freq_base, float freq_scale, float attn_factor, const int32_t *slots, void *k_cache, int64_t k_cache_nb_row,
                    void *v_cache, int64_t v_cache_nb_row, b200_stream_t stream) {
    return b200_rope_store_to(q, q, q_nb_head, q_nb_tok, k, k_nb_head, k_nb_tok, v, v_nb_tok, D, H, Hkv, T, n_dims, pos, freq_factors, freq_base, freq_scale,
                              attn_factor, slots, k_cache, k_cache_nb_row, v_cache, v_cache_nb_row, stream);
}

int b200_rope_store_to(const float *q, float *q_dst, int64_t q_nb_head, int64_t q_nb_tok, const float *k, int64_t k_nb_head, int64_t k_nb_tok, const float *v,
                       int64_t v_nb_tok, int64_t D, int64_t H, int64_t Hkv, int64_t T, int n_dims, const int32_t *pos, const float *freq_factors,
                       float freq_base, float freq_scale, float attn_factor, const int32_t *slots, void *k_cache, int64_t k_cache_nb_row,
                       void *v_cache, int64_t v_cache_nb_row, b200_stream_t stream) {
    B200_REQUIRE(k && pos && k_cache && (H == 0 || (q && q_dst)) && (!v || v_cache), "null pointer");
    B200_REQUIRE(is_aligned(q_dst, 8), "pairs must be 8-byte aligned");
    B200_REQUIRE(D > 0 && D % 2 == 0 && H >= 0 && Hkv > 0 && T >= 0 && n_dims > 0 && n_dims <= D && n_dims % 2 == 0, "bad rope arguments");
    B200_REQUIRE(q_nb_head % 8 == 0 && q_nb_tok % 8 == 0 && k_nb_head % 8 == 0 && k_nb_tok % 8 == 0 && v_nb_tok % 8 == 0 && is_aligned(q, 8) &&
                     is_aligned(k, 8) && is_aligned(v, 8) && k_cache_nb_row % 4 == 0 && v_cache_nb_row % 4 == 0 && is_aligned(k_cache, 4) && is_aligned(v_cache, 4),
                 "pairs must be 8-byte aligned (f32) / 4-byte aligned (f16)");
    if (T == 0) return B200_OK;
    const float theta_scale = powf(freq_base, -2.0f / (float) n_dims);
    launch_pdl(rope_store_kernel, dim3((unsigned) T), dim3(512), (size_t) n_dims * sizeof(float), (cudaStream_t) stream,
        q, q_dst, q_nb_head, q_nb_tok, k, k_nb_head, k_nb_tok, v, v_nb_tok, D, H, Hkv, n_dims, pos, freq_factors, theta_scale, freq_scale, attn_factor,
        slots, (__half *) k_cache, k_cache_nb_row, (__half *) v_cache, v_cache_nb_row, T <= pdl_early_rows() ? 1 : 0);
    return check_launch("rope_store");
}

static int launch_rope_angles(float *angles, int64_t T, int n_dims, const int32_t *pos, const float *freq_factors, float freq_base, float freq_scale, float attn_factor,
                              int32_t *cell_pos, int32_t *cell_seq, const int32_t *slots, const int32_t *seq, b200_stream_t stream) {
    B200_REQUIRE(angles && pos && T > 0 && n_dims > 0 && n_dims % 2 == 0 && n_dims <= 8192 && is_aligned(angles, 4), "bad rope arguments");
    const float theta_scale = powf(freq_base, -2.0f / (float) n_dims);
    launch_pdl(rope_angles_kernel, dim3((unsigned) T), dim3(128), 0, (cudaStream_t) stream, angles, n_dims, pos, freq_factors, theta_scale, freq_scale, attn_factor,
               cell_pos, cell_seq, slots, seq);
    return check_launch("rope_angles");
}

int b200_rope_angles(float *angles, int64_t T, int n_dims, const int32_t *pos, const float *freq_factors, float freq_base, float freq_scale,
                     float attn_factor, b200_stream_t stream) {
    return launch_rope_angles(angles, T, n_dims, pos, freq_factors, freq_base, freq_scale, attn_factor, nullptr, nullptr, nullptr, nullptr, stream);
}

int b200_ubatch_begin(int32_t *cell_pos, int32_t *cell_seq, const int32_t *slots, const int32_t *pos, const int32_t *seq, int64_t T, float *angles, int n_dims,
                      const float *freq_factors, float freq_base, float freq_scale, float attn_factor, b200_stream_t stream) {
    B200_REQUIRE(cell_pos && cell_seq && slots && seq, "null pointer");
    return launch_rope_angles(angles, T, n_dims, pos, freq_factors, freq_base, freq_scale, attn_factor, cell_pos, cell_seq, slots, seq, stream);
}

int b200_rope_store_angles(float *q, int64_t q_nb_head, int64_t q_nb_tok, const float *k, int64_t k_nb_head, int64_t k_nb_tok, const float *v,
                           int64_t v_nb_tok, int64_t D, int64_t H, int64_t Hkv, int64_t T, int n_dims, const float *angles, const int32_t *slots,
                           void *k_cache, int64_t k_cache_nb_row, void *v_cache, int64_t v_cache_nb_row, b200_stream_t stream) {
    B200_REQUIRE(q && k && v && angles && slots && k_cache && v_cache && T > 0 && H > 0 && Hkv > 0 && H + 2 * Hkv <= 4096, "bad rope_store arguments");
    B200_REQUIRE((D == 64 || D == 128 || D == 256) && n_dims > 0 && n_dims % 2 == 0 && n_dims <= D, "head size %lld not supported (64, 128 or 256)", (long long) D);
    B200_REQUIRE(is_aligned(q, 8) && is_aligned(k, 8) && is_aligned(v, 8) && q_nb_head % 8 == 0 && q_nb_tok % 8 == 0 && k_nb_head % 8 == 0 && k_nb_tok % 8 == 0 && v_nb_tok % 8 == 0,
                 "rope rows must be 8-byte aligned");
    B200_REQUIRE(is_aligned(k_cache, 4) && is_aligned(v_cache, 4) && k_cache_nb_row % 4 == 0 && v_cache_nb_row % 4 == 0, "cache rows must be 4-byte aligned");
    const int pairs = (int) D / 2, per = 256 / pairs;
    const dim3 grid((unsigned) T, (unsigned) ((H + 2 * Hkv + per * RA_UNROLL - 1) / (per * RA_UNROLL)));
    launch_pdl(rope_store_angles_kernel, grid, dim3(256), 0, (cudaStream_t) stream, q, q_nb_head, q_nb_tok, k, k_nb_head, k_nb_tok, v, v_nb_tok, pairs, (int) H, (int) Hkv, n_dims,
               angles, slots, (__half *) k_cache, k_cache_nb_row, (__half *) v_cache, v_cache_nb_row, T <= pdl_early_rows() ? 1 : 0);
    return check_launch("rope_store_angles");
}

}  // extern "C"
