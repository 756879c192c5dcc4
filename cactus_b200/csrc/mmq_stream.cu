// MUL_MAT for a handful of activation columns (up to 8): int8 tensor-core MMAs on weights that go from global memory straight
// to registers.
//
// lm_ggml_compute_forward_mul_mat (cactus/ggml-cpu/ggml-cpu.c:1257-1449) with the arithmetic of mmq.cu: exact integer block dots,
// t = d_a * dot rounded once, y = fma(d_w, t, y).
//
// What bounds it: the weight stream, and at these widths the latency in front of and behind it.  A T16 tile is in the order
// of an MMA A fragment, so a warp needs no shared memory for weights: it keeps RING tiles on their way in registers (16 warps
// an SM: 74 KB).  Weights may be what the kernel ahead writes (an upload, a copy that stacks them), so none is read before the wait for it,
// and asking for the first tiles in L2 ahead of it (cp.async.bulk.prefetch.L2) is slower the more are asked for: quantiser and product of
// 8 columns, Q4_0 4096 x 28672, with 32 / 16 / 8 / 4 / 1 / 0 tiles of a warp 22.2 / 21.3 / 20.4 / 19.6 / 19.3 / 19.3 us, 4096 x 4096 7.7 / 7.7 / 7.7 / 7.7 / 7.3 / 7.2.
// mmq.cu copies through a shared-memory ring with a barrier per block group, works 128 rows at a time and stays the kernel for
// more columns (16 columns here: two column tiles per weight tile are bound by instructions, 16.6 us against 13.6 at 14336 x 4096).
// us on B200, mmq.cu / this kernel at 8 columns (K x M, weights larger than L2 in turn): Q4_0 4096 x 28672 24.6 / 16.9, 4096 x 6144
// 8.6 / 6.8, 4096 x 4096 7.6 / 5.4, 14336 x 4096 13.4 / 11.1, 4096 x 128256 72.3 / 54.9 (5.4 TB/s), 2048 x 2048 4.4 / 3.8; Q8_0
// 2048 x 128256 51.1 / 49.2.
//
// Work split: one CTA of 16 warps per SM with an equal share of the row tiles; 2^cl warps share the K range of a row tile, and
// their parts are added in K order through shared memory, so sums do not depend on timing.  Cutting K over clusters as well was
// slower at every shape (4096 x 6144: 8.3 us with two CTAs, 4096 x 4096 7.3), two CTAs of 8 warps per SM too (4096 x 28672 21.7), and
// so was an early trigger for the next kernel (7 sequences of the 8B architecture 2907 us a step, 2715 without).

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "mma_s8.cuh"

namespace b200 {

constexpr int MS_LOG_WARPS = 4, MS_WARPS = 1 << MS_LOG_WARPS, MS_THREADS = MS_WARPS * 32, MS_SMEM = 216 * 1024;
constexpr int MS_SLOT = 160;   // floats of a partial tile: [column][16 rows], columns 20 apart (32 lanes, 32 banks)

struct MsPlan {
    int cl, chunk_bg;   // 2^cl warps share a row tile, block groups of each
    int slots_at;       // in shared memory, behind the activations
};

template <int WTYPE>
struct MsTile {   // a T16 tile as a lane holds it
    uint4 q[WTYPE == B200_TYPE_Q4_0 ? 2 : 4];
    uint2 sa, sb;
};

template <int WTYPE, bool ROPE>   // ROPE: the rows are those of q, k and v (RopeStore)
__global__ void __launch_bounds__(MS_THREADS, 1) mmq_stream_kernel(TiledDims dims, const uint8_t *__restrict__ w, ActDims act, const uint8_t *__restrict__ aq,
                                                                float *__restrict__ dst, int64_t dst_nb_row, MsPlan plan, RopeStore rope) {
    constexpr int RING = WTYPE == B200_TYPE_Q4_0 ? 4 : 2, TB = WTYPE == B200_TYPE_Q4_0 ? 1024 : 2048;
    constexpr float WS = WTYPE == B200_TYPE_Q4_0 ? 0.0625f : 1.0f;   // Q4_0 quants are used as 16 * value
    extern __shared__ __align__(128) uint8_t smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int n_bg = (int) dims.n_bg, n_rt = (int) dims.n_rt;
    const int r0 = (int) ((uint64_t) blockIdx.x * (unsigned) n_rt / gridDim.x), n_r = (int) ((uint64_t) (blockIdx.x + 1) * (unsigned) n_rt / gridDim.x) - r0;
    const int cl = plan.cl, chunk = warp & ((1 << cl) - 1), step = MS_WARPS >> cl, b0 = chunk * plan.chunk_bg, len = min(plan.chunk_bg, n_bg - b0), r_first = warp >> cl;
    const bool idle = len <= 0 || r_first >= n_r;
    // the next tile to load: pointers of this lane, which jump from the end of a row tile to the next one of the warp
    const int64_t at0 = idle ? 0 : (int64_t) (r0 + r_first) * n_bg + b0;
    const uint8_t *lq = w + at0 * TB + lane * (WTYPE == B200_TYPE_Q4_0 ? 32 : 16), *ld = w + dims.qs_bytes + at0 * 128 + g * 8;
    const int jump = step * n_bg - len;
    const int n_mine = idle ? 0 : (n_r - r_first + step - 1) >> (MS_LOG_WARPS - cl);   // row tiles of this warp
    int left = n_mine * len, to_end = len;   // tiles to load, of this row tile
    MsTile<WTYPE> ring[RING];
    // (never conditional: a load behind a branch is waited for where the branch ends.  The last tile is loaded again instead.)
    auto load = [&](MsTile<WTYPE> &f) {
        if (WTYPE == B200_TYPE_Q4_0) {
            f.q[0] = __ldg(reinterpret_cast<const uint4 *>(lq));
            f.q[1] = __ldg(reinterpret_cast<const uint4 *>(lq) + 1);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) f.q[j % (WTYPE == B200_TYPE_Q4_0 ? 2 : 4)] = __ldg(reinterpret_cast<const uint4 *>(lq + j * 512));
        }
        f.sa = __ldg(reinterpret_cast<const uint2 *>(ld));
        f.sb = __ldg(reinterpret_cast<const uint2 *>(ld + 64));
        --left;
        --to_end;
        const int64_t go = left <= 0 ? 0 : to_end == 0 ? 1 + jump : 1;
        to_end = to_end == 0 ? len : to_end;
        lq += go * TB;
        ld += go * 128;
    };
    pdl_prologue();
#pragma unroll
    for (int k = 0; k < RING; ++k) load(ring[k]);
    const int q_bytes = n_bg * 1024;
    {   // into shared memory, with their scales: one piece (a single column tile)
        const uint4 *q = reinterpret_cast<const uint4 *>(aq);
#pragma unroll 4
        for (int i = tid; i < n_bg * 80; i += MS_THREADS) reinterpret_cast<uint4 *>(smem)[i] = __ldg(q + i);
    }
    __syncthreads();
    float *const slots = reinterpret_cast<float *>(smem + plan.slots_at);
    {
        const uint8_t *qb = smem + b0 * 1024 + lane * 8, *sb = smem + q_bytes + b0 * 256 + t * 16;
        float *slot = slots + ((r_first << cl) + chunk) * MS_SLOT + 40 * t + g;
        uint64_t y0 = 0ull, y1 = 0ull;   // rows g, g + 8, columns 2t, 2t + 1
        int todo = n_mine * len, i = 0;
        while (todo > 0) {
#pragma unroll
            for (int k = 0; k < RING; ++k) {
                if (todo <= 0) break;
                --todo;
                const MsTile<WTYPE> &f = ring[k];
                uint2 b[4];
                uint4 sc[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    b[j] = *reinterpret_cast<const uint2 *>(qb + i * 1024 + j * 256);
                    sc[j] = *reinterpret_cast<const uint4 *>(sb + i * 256 + j * 64);
                }
                uint64_t p01[4], p23[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint32_t a0, a1, a2, a3;
                    if (WTYPE == B200_TYPE_Q4_0) {
                        const uint32_t wa = j == 0 ? f.q[0].x : j == 1 ? f.q[0].y : j == 2 ? f.q[0].z : f.q[0].w, wb = j == 0 ? f.q[1].x : j == 1 ? f.q[1].y : j == 2 ? f.q[1].z : f.q[1].w;
                        a0 = (wa << 4) & 0xF0F0F0F0u; a2 = wa & 0xF0F0F0F0u;
                        a1 = (wb << 4) & 0xF0F0F0F0u; a3 = wb & 0xF0F0F0F0u;
                    } else {
                        const uint4 u = f.q[j % (WTYPE == B200_TYPE_Q4_0 ? 2 : 4)];
                        a0 = u.x; a1 = u.y; a2 = u.z; a3 = u.w;
                    }
                    mma_s8_magic2(p01[j], p23[j], a0, a1, a2, a3, b[j].x, b[j].y);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t ha = j < 2 ? f.sa.x : f.sa.y, hb = j < 2 ? f.sb.x : f.sb.y;
                    const __half2 h2a = *reinterpret_cast<const __half2 *>(&ha), h2b = *reinterpret_cast<const __half2 *>(&hb);
                    const uint32_t ua = __float_as_uint(j & 1 ? __high2float(h2a) : __low2float(h2a)), ub = __float_as_uint(j & 1 ? __high2float(h2b) : __low2float(h2b));
                    const uint64_t da = pack2(sc[j].x, sc[j].y), nda = pack2(sc[j].z, sc[j].w);
                    y0 = fma2(fma2(p01[j], da, nda), pack2(ua, ua), y0);
                    y1 = fma2(fma2(p23[j], da, nda), pack2(ub, ub), y1);
                }
                load(ring[k]);
                if (++i == len) {
                    i = 0;
                    float v0, v1, v2, v3;
                    unpack2(y0, v0, v1);
                    unpack2(y1, v2, v3);
                    slot[0] = v0 * WS; slot[20] = v1 * WS; slot[8] = v2 * WS; slot[28] = v3 * WS;
                    y0 = y1 = 0ull;
                    slot += MS_WARPS * MS_SLOT;   // (step << cl is the number of warps)
                }
            }
        }
    }
    // The chunks of a row tile, in K order.  Threads go over [column][rows], the rows padded to a power of two.
    const int chunks = min(1 << cl, (n_bg + plan.chunk_bg - 1) / plan.chunk_bg), rows = n_r * 16, lg = 32 - __clz(rows - 1), n_e = (int) act.N << lg;
    auto angle_of = [&](int e) { return rope_angle(rope, min(e >> lg, (int) act.N - 1), r0 * 16 + (e & ((1 << lg) - 1))); };
    float2 angle = make_float2(1.0f, 0.0f);
    int64_t slot = 0;
    if (ROPE) {   // of the first round; the loads travel while the last warps finish
        angle = angle_of(tid);
        slot = rope.slots[min(tid >> lg, (int) act.N - 1)];
    }
    pdl_trigger();
    __syncthreads();
    for (int e = tid; e < (n_e + 31 & ~31); e += MS_THREADS) {   // whole warps
        const int col = e >> lg, rr = e & ((1 << lg) - 1);
        const int64_t row = (int64_t) r0 * 16 + rr;
        const bool real = e < n_e && rr < rows && row < dims.M;
        float v = 0.0f;
        if (real) {
            const float *s = slots + ((rr >> 4) << cl) * MS_SLOT + col * 20 + (rr & 15);
#pragma unroll 4
            for (int c = 0; c < chunks; ++c) v += s[c * MS_SLOT];
        }
        if (ROPE) {
            const float other = __shfl_down_sync(0xffffffffu, v, 1);   // (an even number of rows)
            if (e >= MS_THREADS) {
                angle = angle_of(e);
                slot = rope.slots[min(col, (int) act.N - 1)];
            }
            if (real && !(e & 1)) rope_store_pair(rope, dst, dst_nb_row, col, (int) row, make_float2(v, other), angle, slot);
        } else if (real) {
            *reinterpret_cast<float *>(reinterpret_cast<char *>(dst) + col * dst_nb_row + row * 4) = v;
        }
    }
}

static int ms_sm_count() {   // every device of a process is the same model; the kernels' attribute is per device
    static int n[64] = {0};
    static std::mutex mu;
    int dev = 0;
    cudaGetDevice(&dev);
    dev &= 63;
    std::lock_guard<std::mutex> lock(mu);
    if (!n[dev]) {
        cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
        if (n[dev] <= 0) n[dev] = 148;
        cudaFuncSetAttribute(mmq_stream_kernel<B200_TYPE_Q4_0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MS_SMEM);
        cudaFuncSetAttribute(mmq_stream_kernel<B200_TYPE_Q4_0, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MS_SMEM);
        cudaFuncSetAttribute(mmq_stream_kernel<B200_TYPE_Q8_0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MS_SMEM);
        cudaFuncSetAttribute(mmq_stream_kernel<B200_TYPE_Q8_0, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MS_SMEM);
    }
    return n[dev];
}

// false: the activations and partial tiles do not fit into shared memory (K above some 21000), or nothing does; *rc: how the launch went.
// rope: the rows are those of q, k and v, see there
bool launch_mmq_stream(int wtype, const TiledDims &d, const void *w, const ActDims &a, const void *aq, float *dst, int64_t dst_nb_row, const RopeStore *rope, cudaStream_t st,
                       int *rc) {
    if (a.n_nt != 1 || d.n_rt * d.n_bg >= (1ll << 31)) return false;
    const int64_t ctas = std::min<int64_t>(ms_sm_count(), d.n_rt), rt = (d.n_rt + ctas - 1) / ctas, act = d.n_bg * 1280;
    // The most warps a row tile (all work to the end) whose partial tiles fit: tiles of the busiest warp, and what a row tile's end costs
    MsPlan p = {};
    int64_t best = -1;
    size_t smem = 0;
    for (int cl = MS_LOG_WARPS; cl >= 0; --cl) {
        const int64_t chunk = (d.n_bg + (1 << cl) - 1) >> cl, step = MS_WARPS >> cl, rounds = (rt + step - 1) / step;
        const int64_t bytes = act + rounds * MS_WARPS * MS_SLOT * 4, cost = rounds * (chunk * 4 + 1);
        if (bytes > MS_SMEM || (best >= 0 && cost >= best)) continue;
        best = cost;
        p.cl = cl;
        p.chunk_bg = (int) chunk;
        p.slots_at = (int) act;
        smem = (size_t) bytes;
    }
    if (best < 0) return false;
    const bool q4 = wtype == B200_TYPE_Q4_0;
    const auto kernel = rope ? (q4 ? mmq_stream_kernel<B200_TYPE_Q4_0, true> : mmq_stream_kernel<B200_TYPE_Q8_0, true>) : (q4 ? mmq_stream_kernel<B200_TYPE_Q4_0, false> : mmq_stream_kernel<B200_TYPE_Q8_0, false>);
    launch_pdl(kernel, dim3((unsigned) ctas), dim3(MS_THREADS), smem, st, d, (const uint8_t *) w, a, (const uint8_t *) aq, dst, dst_nb_row, p, rope ? *rope : RopeStore{});
    *rc = check_launch("mmq_stream");
    return true;
}

}  // namespace b200
