// C ABI of MUL_MAT: argument checks and the choice between the dp4a kernel (mmvq.cu), the streaming tensor-core kernel
// (mmq_stream.cu) and the tiled ones (mmq.cu, mmq_tc.cu).
#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "common.cuh"

namespace b200 {
int launch_mmq_tc(const TiledDims &d, const void *w, const ActDims &a, const void *aq, float *dst, int64_t dst_nb_row,
                  void *workspace, size_t workspace_bytes, cudaStream_t st);
size_t mmq_tc_workspace_bytes(int64_t M, int64_t N);
int tc_error_flag();
void tc_set_wait_limit(unsigned rounds);
bool mmq_sync_forced();
int launch_quantize_b8(const float *x, int64_t x_nb_row, int64_t K, int64_t N, void *scratch, int variant, int layout, cudaStream_t st);
int mmvq_max_n();
int launch_mmvq(int wtype, const TiledDims &d, const void *w, const ActDims &a, const void *aq, float *dst, int64_t dst_nb_row, const PeerDst &peers,
                const RopeStore *rope, cudaStream_t st);
int launch_mmq(int wtype, const TiledDims &d, const void *w, const ActDims &a, const void *aq, float *dst, int64_t dst_nb_row,
               void *workspace, size_t workspace_bytes, cudaStream_t st, const PeerDst &peers);
bool launch_mmq_stream(int wtype, const TiledDims &d, const void *w, const ActDims &a, const void *aq, float *dst, int64_t dst_nb_row, bool workspace, size_t workspace_bytes,
                       const RopeStore *rope, cudaStream_t st, int *rc);
int launch_peer_signal_wait(void *const *flags_of_rank, int rank, int g, cudaStream_t st);
size_t mmq_workspace_bytes(int wtype, int64_t K, int64_t M, int64_t N);
}  // namespace b200

using namespace b200;

// ---------------------------------------------------------------------------------------------
// Scratch for b200_mul_mat_q_noalloc: room for the quantised activations of up to 8 columns of
// B200_NOALLOC_MAX_K values (one 8-column tile of 256-byte block groups plus its scale plane).
// The array lives in every device that loads this library, from load until the process exits.
// In host code the name below is only a handle for cudaGetSymbolAddress, never a device address.
// ---------------------------------------------------------------------------------------------
constexpr size_t NOALLOC_SCRATCH_BYTES = (size_t) B200_NOALLOC_MAX_K / 32 * 256 + (size_t) B200_NOALLOC_MAX_K / 128 * 256;
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

// device address of the array on the current device, looked up once per device
static int noalloc_scratch_ptr(void **out) {
    static void *ptrs[64] = {nullptr};
    static std::mutex mu;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(B200_E_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= 64) return set_error(B200_E_INVALID, "device index %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (!ptrs[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) return set_error(B200_E_CUDA, "cudaGetSymbolAddress(scratch): %s", cudaGetErrorString(e));
        ptrs[dev] = p;
    }
    *out = ptrs[dev];
    return B200_OK;
}

static bool shape_ok(int wtype, int64_t K, int64_t M, int64_t N) {
    return (wtype == B200_TYPE_Q4_0 || wtype == B200_TYPE_Q8_0) && K > 0 && K % 32 == 0 && M > 0 && N > 0;
}

// b200_mul_mat_q alone chooses between the two tensor-core kernels: it knows the weights' shape when it quantises, and the
// tcgen05 kernel wants its operands laid out by the quantiser.  (Products of activations that are quantised on their own feed
// whole models and keep the mma.sync kernel.)
// Measured on B200, quantiser and product, weights larger than L2 in turn (us, tcgen05 / mma.sync, Q4_0):
//   K x M            N = 33       64           65           128          192          256          384          512
//   4096 x 28672     48.8 / 53.5  53.3 / 54.3  81.6 / 103   89.9 / 104   122 / 138    156 / 178    231 / 248    316 / 321
//   4096 x 20480     1.14         1.07         1.27         1.18         1.13         1.10         1.09         1.05   (ratios)
//   8192 x 16384     1.10         1.01         1.22         1.12         1.19         1.16         1.14         0.97
//   4096 x 14336     31.5 / 32.8  34.6 / 33.1  47.3 / 54.6  51.0 / 55.3  68.5 / 78.7  88.4 / 103   121 / 138    156 / 178
//   4096 x 10240     0.96         0.89         1.18         1.11         1.04         1.18         1.14         1.10
//   8192 x 8192      33.6 / 32.6  36.3 / 32.9  52.1 / 56.8  57.0 / 57.7  74.0 / 82.5  93.7 / 105   134 / 158    184 / 201
//   4096 x 8192      0.85         0.79         0.99         0.94         1.06         1.01         1.15         1.07
//   14336 x 4096     36.5 / 30.1  39.0 / 30.5  48.2 / 50.2  52.9 / 51.7  86.8 / 71.5  91.8 / 96.3  124 / 134    167 / 183
//   4096 x 6144      20.8 / 18.4  23.2 / 18.8  31.1 / 25.7  34.2 / 28.0  34.8 / 33.1  46.5 / 49.4  55.8 / 56.1  76.6 / 86.8
//   4096 x 4096      18.8 / 14.7  20.9 / 14.9  23.1 / 19.1  24.5 / 19.7  34.0 / 28.3  34.8 / 33.1  46.7 / 50.3  56.4 / 56.6
//   2048 x 16384     21.6 / 20.8  24.0 / 21.2  31.4 / 30.4  34.3 / 30.9  48.7 / 50.8  60.5 / 56.6  83.8 / 81.6  105 / 95.5
// The tcgen05 kernel needs about 5 us to fill and empty a CTA's pipeline and pays per 256 rows x 64 columns x K, so it wants
// a long K and enough row groups that no SM waits: hence the lines below.  Beyond 100 G multiply-adds it falls behind again
// (8192 x 32768 at 320 / 384 / 448 / 512 columns: 434 / 453, 535 / 531, 670 / 624, 762 / 675).
// Q8_0 never: a stage of its ring holds twice the weights, so that two fit instead of three and copies and MMAs hardly overlap
// (4096 x 28672 at 65 / 256 / 512 columns 95.8 / 101, 193 / 175, 371 / 310; 4096 x 14336 54.2 / 53.8, 100 / 101, 182 / 176;
// 14336 x 4096 55.4 / 49.9, 109 / 94.0, 179 / 177; 8192 x 32768 191 / 193, 419 / 347, 869 / 651).
// B200_MMQ_TC decides by hand for Q4_0 (0: never, else from 9 columns on).
static bool use_tc(int wtype, int64_t K, int64_t M, int64_t N) {
    static const int forced = [] {
        const char *e = getenv("B200_MMQ_TC");
        return e ? atoi(e) : -1;
    }();
    if (wtype != B200_TYPE_Q4_0 || forced == 0 || N < 9 || mmq_sync_forced()) return false;
    if (forced > 0) return true;
    if (N <= 32 || K < 4096 || (double) M * K * N > 1e11) return false;
    if (N <= 64) return M >= 20480;
    if (N <= 192) return M >= 10240;
    return M >= 4096 && M * K >= (24 << 20);
}

// Up to 8 columns the kernel that streams tiles into registers (mmq_stream.cu): from 3 columns on where it is faster than the mma.sync
// kernel, whose result it has to the last bit (ms_pays there).  At one and two columns it adds in another order than the dp4a kernel
// (whose short CTAs start and end faster), so only what is taken for an output head streams: a layer's sums are quantised again, and with
// 4096 x 28672 streaming the logits of one sequence of the 8B architecture moved by 1.4e-2 of their norm (16.3 us against 19.5).
// Quantiser and product, us on B200, dp4a / stream at one and two columns (K x M): Q4_0 4096 x 128256 60.7 / 51.1, 63.5 / 52.6; 4096 x 65536 36.3 / 29.4,
// 36.9 / 30.4; 1024 x 65536 12.2 / 11.6, 13.6 / 12.3; Q8_0 2048 x 128256 50.0 / 45.0, 50.0 / 47.1; 4096 x 128256 88.1 / 83.9, 90.7 / 85.4; 1024 x 128256
// 31.2 / 25.9, 25.5 / 26.8.  Below 32768 tiles (16 rows x 128 values) nothing is won: Q4_0 512 x 65536 8.1, 256 x 128256 11.4, for the dp4a kernel.
static bool use_stream(int wtype, const TiledDims &d, int64_t N) {
    if (N > 8 || mmq_sync_forced()) return false;
    if (N > 2) return N > mmvq_max_n();
    return d.M >= HEAD_ROWS && d.n_rt * d.n_bg >= 32768 && (wtype == B200_TYPE_Q4_0 || N == 1 || d.n_bg >= 16);
}

extern "C" {

int b200_kernel_status(void) { return tc_error_flag() ? 2 : 0; }
void b200_kernel_set_wait_limit(unsigned rounds) { tc_set_wait_limit(rounds); }

size_t b200_mul_mat_workspace_bytes(int wtype, int64_t K, int64_t M, int64_t N) {
    if (!shape_ok(wtype, K, M, N)) return 0;
    return mmq_workspace_bytes(wtype, K, M, N);
}

size_t b200_mul_mat_scratch_bytes(int wtype, int64_t K, int64_t M, int64_t N) {
    if (!shape_ok(wtype, K, M, N)) return 0;
    const ActDims a = act_dims(K, N);
    return a.total_bytes + (use_tc(wtype, K, M, N) ? a.b_bytes + mmq_tc_workspace_bytes(M, N) : mmq_workspace_bytes(wtype, K, M, N));
}

static int mul_mat_prequant(int wtype, const void *w, int64_t K, int64_t M, const void *act, int64_t N, float *dst, int64_t dst_row_stride_bytes,
                            void *workspace, size_t workspace_bytes, const PeerDst &peers, b200_stream_t stream);

int b200_mul_mat_q_prequant(int wtype, const void *w, int64_t K, int64_t M, const void *act, int64_t N, float *dst,
                            int64_t dst_row_stride_bytes, void *workspace, size_t workspace_bytes, b200_stream_t stream) {
    return mul_mat_prequant(wtype, w, K, M, act, N, dst, dst_row_stride_bytes, workspace, workspace_bytes, PeerDst{}, stream);
}

static int rowsplit_impl(int wtype, const void *w, int64_t K, int64_t M, const void *act, int64_t N, int rank, int g, void *const *dst_of_rank,
                         int64_t dst_row_stride_bytes, int64_t first_column, PeerDst peers, void *workspace, size_t workspace_bytes,
                         void *const *flags_of_rank, b200_stream_t stream);

int b200_mul_mat_q_rowsplit(int wtype, const void *w, int64_t K, int64_t M, const void *act, int64_t N, int rank, int g, void *const *dst_of_rank,
                            int64_t dst_row_stride_bytes, int64_t first_column, void *workspace, size_t workspace_bytes,
                            void *const *flags_of_rank, b200_stream_t stream) {
    return rowsplit_impl(wtype, w, K, M, act, N, rank, g, dst_of_rank, dst_row_stride_bytes, first_column, PeerDst{}, workspace, workspace_bytes,
                         flags_of_rank, stream);
}

int b200_mul_mat_q_rowsplit_stacked(int wtype, const void *w, int64_t K, int64_t M, const void *act, int64_t N, int rank, int g,
                                    void *const *dst_of_rank, int64_t dst_row_stride_bytes, int n_parts, const int64_t *part_rows,
                                    const int64_t *part_first_column, void *workspace, size_t workspace_bytes, void *const *flags_of_rank,
                                    b200_stream_t stream) {
    B200_REQUIRE(n_parts >= 1 && n_parts <= 3 && part_rows && part_first_column, "a stacked weight has 1 to 3 parts");
    PeerDst peers = {};
    peers.n_seg = n_parts;
    int64_t row = 0;
    for (int i = 0; i < n_parts; ++i) {
        B200_REQUIRE(part_rows[i] > 0 && part_first_column[i] >= 0 && (i == n_parts - 1 || part_rows[i] % 16 == 0), "parts but the last hold a multiple of 16 rows");
        // a plain mapping puts local row r at column part_first_column[0] + r
        peers.seg_shift[i] = (part_first_column[i] - (part_first_column[0] + row)) * 4;
        row += part_rows[i];
        if (i < 2) peers.seg_end[i] = (int) row;
    }
    B200_REQUIRE(row == M, "the parts hold %lld rows, the weight %lld", (long long) row, (long long) M);
    return rowsplit_impl(wtype, w, K, M, act, N, rank, g, dst_of_rank, dst_row_stride_bytes, part_first_column[0], peers, workspace, workspace_bytes,
                         flags_of_rank, stream);
}

static int rowsplit_impl(int wtype, const void *w, int64_t K, int64_t M, const void *act, int64_t N, int rank, int g, void *const *dst_of_rank,
                         int64_t dst_row_stride_bytes, int64_t first_column, PeerDst peers, void *workspace, size_t workspace_bytes,
                         void *const *flags_of_rank, b200_stream_t stream) {
    B200_REQUIRE(dst_of_rank && flags_of_rank && g >= 1 && g <= 8 && rank >= 0 && rank < g && first_column >= 0, "bad row-split arguments");
    float *own = nullptr;
    for (int r = 0; r < g; ++r) {
        B200_REQUIRE(dst_of_rank[r] && flags_of_rank[r], "null buffer of rank %d", r);
        float *p = reinterpret_cast<float *>(dst_of_rank[r]) + first_column;
        if (r == rank) own = p;
        else peers.p[peers.n++] = p;
    }
    if (int e = mul_mat_prequant(wtype, w, K, M, act, N, own, dst_row_stride_bytes, workspace, workspace_bytes, peers, stream)) return e;
    return launch_peer_signal_wait(flags_of_rank, rank, g, (cudaStream_t) stream);
}

static int mul_mat_prequant(int wtype, const void *w, int64_t K, int64_t M, const void *act, int64_t N, float *dst, int64_t dst_row_stride_bytes,
                            void *workspace, size_t workspace_bytes, const PeerDst &peers, b200_stream_t stream) {
    B200_REQUIRE(shape_ok(wtype, K, M, N), "bad mul_mat shape/type: type %d K %lld M %lld N %lld", wtype, (long long) K, (long long) M, (long long) N);
    B200_REQUIRE(w && act && dst, "null pointer");
    B200_REQUIRE(is_aligned(w, 16) && is_aligned(act, 256) && is_aligned(dst, 4), "misaligned pointer");
    B200_REQUIRE(dst_row_stride_bytes % 4 == 0 && dst_row_stride_bytes >= M * 4, "bad dst row stride");
    B200_REQUIRE(!workspace || is_aligned(workspace, 256), "workspace must be 256-byte aligned");
    const TiledDims d = tiled_dims(wtype, K, M);
    const ActDims a = act_dims(K, N);
    if (peers.n == 0 && peers.n_seg <= 1 && use_stream(wtype, d, N)) {
        int rc = 0;
        if (launch_mmq_stream(wtype, d, w, a, act, dst, dst_row_stride_bytes, workspace != nullptr, workspace_bytes, nullptr, (cudaStream_t) stream, &rc)) return rc;
    }
    if (N <= mmvq_max_n()) return launch_mmvq(wtype, d, w, a, act, dst, dst_row_stride_bytes, peers, nullptr, (cudaStream_t) stream);
    return launch_mmq(wtype, d, w, a, act, dst, dst_row_stride_bytes, workspace, workspace_bytes, (cudaStream_t) stream, peers);
}

int b200_mul_mat_qkv_rope(int wtype, const void *w, int64_t K, const void *act, int64_t N, float *qkv, int64_t qkv_row_stride_bytes, int64_t D, int64_t H, int64_t Hkv,
                          int n_dims, const float *angles, const int32_t *slots, void *k_cache, int64_t k_cache_nb_row, void *v_cache, int64_t v_cache_nb_row,
                          void *workspace, size_t workspace_bytes, b200_stream_t stream) {
    B200_REQUIRE((D == 64 || D == 128 || D == 256) && H > 0 && Hkv > 0 && H + 2 * Hkv <= 4096, "bad heads: %lld and 2 x %lld of %lld", (long long) H, (long long) Hkv, (long long) D);
    const int64_t M = (H + 2 * Hkv) * D;
    B200_REQUIRE(shape_ok(wtype, K, M, N), "bad mul_mat shape/type: type %d K %lld M %lld N %lld", wtype, (long long) K, (long long) M, (long long) N);
    B200_REQUIRE(w && act && qkv && angles && slots && k_cache && v_cache && n_dims > 0 && n_dims % 2 == 0 && n_dims <= D, "null pointer or bad rope arguments");
    B200_REQUIRE(is_aligned(w, 16) && is_aligned(act, 256) && is_aligned(qkv, 8) && is_aligned(k_cache, 4) && is_aligned(v_cache, 4), "misaligned pointer");
    B200_REQUIRE(qkv_row_stride_bytes % 8 == 0 && qkv_row_stride_bytes >= M * 4 && k_cache_nb_row % 4 == 0 && v_cache_nb_row % 4 == 0, "bad row stride");
    const TiledDims d = tiled_dims(wtype, K, M);
    const ActDims a = act_dims(K, N);
    const RopeStore rope = {angles, slots, (__half *) k_cache, (__half *) v_cache, k_cache_nb_row, v_cache_nb_row, (int) (H * D), (int) ((H + Hkv) * D), (int) D / 2 - 1, n_dims / 2};
    if (use_stream(wtype, d, N)) {
        int rc = 0;
        if (launch_mmq_stream(wtype, d, w, a, act, qkv, qkv_row_stride_bytes, workspace != nullptr, workspace_bytes, &rope, (cudaStream_t) stream, &rc)) return rc;
    } else if (N <= std::min(2, mmvq_max_n())) {
        return launch_mmvq(wtype, d, w, a, act, qkv, qkv_row_stride_bytes, PeerDst{}, &rope, (cudaStream_t) stream);
    }
    if (int e = b200_mul_mat_q_prequant(wtype, w, K, M, act, N, qkv, qkv_row_stride_bytes, workspace, workspace_bytes, stream)) return e;
    return b200_rope_store_angles(qkv, D * 4, qkv_row_stride_bytes, qkv + H * D, D * 4, qkv_row_stride_bytes, qkv + (H + Hkv) * D, qkv_row_stride_bytes, D, H, Hkv, N, n_dims, angles, slots,
                                  k_cache, k_cache_nb_row, v_cache, v_cache_nb_row, stream);
}

int b200_mul_mat_q_prequant_multi(int wtype, int n_weights, const void *const *w, const int64_t *M, int64_t K, const void *act, int64_t N,
                                  float *const *dst, int64_t dst_row_stride_bytes, void *workspace, size_t workspace_bytes, b200_stream_t stream) {
    B200_REQUIRE(n_weights >= 1 && n_weights <= 3 && w && M && dst, "1 to 3 weights");
    int64_t total = 0;
    bool whole_groups = true;
    for (int i = 0; i < n_weights; ++i) {
        B200_REQUIRE(w[i] && dst[i] && M[i] > 0 && is_aligned(w[i], 16) && is_aligned(dst[i], 4), "null or misaligned weight / destination %d", i);
        whole_groups = whole_groups && (i == n_weights - 1 || M[i] % 128 == 0);
        total += M[i];
    }
    // one launch needs whole row groups per tensor and the tensor-core kernel; otherwise one product after the other
    if (n_weights == 1 || !whole_groups || N <= mmvq_max_n()) {
        for (int i = 0; i < n_weights; ++i)
            if (int e = b200_mul_mat_q_prequant(wtype, w[i], K, M[i], act, N, dst[i], dst_row_stride_bytes, workspace, workspace_bytes, stream)) return e;
        return B200_OK;
    }
    B200_REQUIRE(shape_ok(wtype, K, total, N), "bad mul_mat shape/type: type %d K %lld M %lld N %lld", wtype, (long long) K, (long long) total, (long long) N);
    B200_REQUIRE(act && is_aligned(act, 256), "null or misaligned activations");
    B200_REQUIRE(dst_row_stride_bytes % 4 == 0, "bad dst row stride");
    B200_REQUIRE(!workspace || is_aligned(workspace, 256), "workspace must be 256-byte aligned");
    PeerDst segs = {};
    segs.n_seg = n_weights;
    segs.n_wseg = n_weights;
    int64_t row = 0;
    for (int i = 0; i < n_weights; ++i) {
        B200_REQUIRE(dst_row_stride_bytes >= M[i] * 4, "bad dst row stride");
        segs.wseg[i] = (const unsigned char *) w[i];
        segs.wseg_qs[i] = (unsigned long long) tiled_dims(wtype, K, M[i]).qs_bytes;
        // a plain mapping puts row r of the stacked product at dst[0] + r floats
        segs.seg_shift[i] = (int64_t) ((const char *) dst[i] - (const char *) dst[0]) - row * 4;
        row += M[i];
        if (i < 2) segs.seg_end[i] = (int) row;
    }
    const TiledDims d = tiled_dims(wtype, K, total);
    const ActDims a = act_dims(K, N);
    return launch_mmq(wtype, d, w[0], a, act, dst[0], dst_row_stride_bytes, workspace, workspace_bytes, (cudaStream_t) stream, segs);
}

int b200_mul_mat_q(int wtype, const void *w, int64_t K, int64_t M, const float *x, int64_t x_row_stride_bytes, int64_t N,
                   float *dst, int64_t dst_row_stride_bytes, void *scratch, size_t scratch_bytes, int variant, b200_stream_t stream) {
    B200_REQUIRE(shape_ok(wtype, K, M, N), "bad mul_mat shape/type: type %d K %lld M %lld N %lld", wtype, (long long) K, (long long) M, (long long) N);
    const ActDims a = act_dims(K, N);
    const bool tc = use_tc(wtype, K, M, N);
    const size_t ab = a.total_bytes + (tc ? a.b_bytes : 0), wb = tc ? mmq_tc_workspace_bytes(M, N) : mmq_workspace_bytes(wtype, K, M, N);
    if (!scratch || scratch_bytes < ab + wb) return set_error(B200_E_SCRATCH, "scratch too small: %zu < %zu", scratch_bytes, ab + wb);
    if (!tc) {
        if (int e = b200_quantize_activations(x, x_row_stride_bytes, K, N, scratch, ab, variant, stream)) return e;
        return b200_mul_mat_q_prequant(wtype, w, K, M, scratch, N, dst, dst_row_stride_bytes, wb ? (char *) scratch + ab : nullptr, wb, stream);
    }
    B200_REQUIRE(w && x && dst && is_aligned(w, 16) && is_aligned(x, 4) && is_aligned(dst, 4) && is_aligned(scratch, 256), "null or misaligned pointer");
    B200_REQUIRE(x_row_stride_bytes % 4 == 0 && dst_row_stride_bytes % 4 == 0 && dst_row_stride_bytes >= M * 4, "bad row stride");
    B200_REQUIRE(variant == B200_Q8_AVX2 || variant == B200_Q8_SCALAR, "unknown quantiser variant %d", variant);
    if (int e = launch_quantize_b8(x, x_row_stride_bytes, K, N, scratch, variant, 2, (cudaStream_t) stream)) return e;
    return launch_mmq_tc(tiled_dims(wtype, K, M), w, a, scratch, dst, dst_row_stride_bytes, (char *) scratch + ab, wb, (cudaStream_t) stream);
}

int b200_mul_mat_q_noalloc(int wtype, const void *w, int64_t K, int64_t M, const float *x, int64_t x_row_stride_bytes, int64_t N,
                           float *dst, int64_t dst_row_stride_bytes, int variant, b200_stream_t stream) {
    B200_REQUIRE(shape_ok(wtype, K, M, N), "bad mul_mat shape/type: type %d K %lld M %lld N %lld", wtype, (long long) K, (long long) M, (long long) N);
    B200_REQUIRE(N <= B200_NOALLOC_MAX_N, "b200_mul_mat_q_noalloc handles at most %d columns, got %lld", B200_NOALLOC_MAX_N, (long long) N);
    B200_REQUIRE(K <= B200_NOALLOC_MAX_K, "b200_mul_mat_q_noalloc handles rows of at most %d values, got %lld", B200_NOALLOC_MAX_K, (long long) K);
    const size_t ab = b200_act_bytes(K, N);
    B200_REQUIRE(ab <= NOALLOC_SCRATCH_BYTES, "built-in scratch too small for K %lld", (long long) K);
    void *scratch = nullptr;
    if (int e = noalloc_scratch_ptr(&scratch)) return e;
    // the quantiser rewrites every byte of the region it uses (padding included), so nothing has to be cleared
    if (int e = b200_quantize_activations(x, x_row_stride_bytes, K, N, scratch, ab, variant, stream)) return e;
    return b200_mul_mat_q_prequant(wtype, w, K, M, scratch, N, dst, dst_row_stride_bytes, nullptr, 0, stream);
}

}  // extern "C"
