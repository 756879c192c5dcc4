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
// Quantiser and product on B200, us with mmq.cu / with this kernel at 8 columns (K x M, weights larger than L2 in turn): Q4_0 4096 x 28672
// 25.7 / 19.3, 4096 x 6144 9.3 / 8.4, 4096 x 4096 7.9 / 7.3, 14336 x 4096 15.1 / 13.5, 4096 x 128256 71.6 / 54.3, 2048 x 2048 5.3 / 4.9; Q8_0 2048 x 128256
// 50.9 / 48.7.  ms_pays has the sizes where it is not faster.
//
// Work split: one CTA of 16 warps per SM with an equal share of the row tiles; the K range of a row tile is cut into parts, which
// are the warps' tasks, and the parts are added in K order through shared memory, so sums do not depend on timing.  Cutting K over
// clusters as well was slower at every shape (4096 x 6144: 8.3 us with two CTAs, 4096 x 4096 7.3), two CTAs of 8 warps per SM too (4096 x
// 28672 21.7), and so was an early trigger for the next kernel (7 sequences of the 8B architecture 2907 us a step, 2715 without).
// K is cut where mmq.cu cuts it (KSplit), so that both give the same bits.  The cuts that suit this kernel best (FREE) are left to output
// heads, whose result nothing quantises again: in the layers they moved a step's logits by 1.3e-2 of their norm.  They are some faster:
// quantiser and product of 8 columns, Q4_0 14336 x 4096 12.8 us against 13.5, 4096 x 28672 18.9 against 19.3.  12 warps with 7 tiles on their way
// each and 8 with 12 are slower (4096 x 28672 22.8 and 23.3 us where 16 with 4 took 20.4), a table of the tasks in shared memory as well (14336 x
// 4096 14.4 us).

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "mma_s8.cuh"

namespace b200 {

constexpr int MS_WARPS = 16, MS_THREADS = MS_WARPS * 32, MS_SMEM = 216 * 1024;
constexpr int MS_SLOT = 160;   // floats of a partial tile: [column][16 rows], columns 20 apart (32 lanes, 32 banks)

struct MsPlan {
    int ks, per;        // the K range of a row tile is ks tasks of `per` block groups (the last one shorter)
    // A stream-K deal cuts some row groups' last task once more: what is behind the first n_bg - unit block groups of all row groups, laid
    // end to end, is dealt out evenly to `share` CTAs (0: no further cut)
    int unit, share, group_tiles, groups;
    int parts;          // at most, of a row tile: the tasks that are not empty, and one more with a further cut
    int slots_at, cuts_at;   // in shared memory, behind the activations
};
// the block group at which row group ct's last task is cut once more, n_bg where it is not
__device__ __forceinline__ int ms_cut(const MsPlan &p, int ct, int n_bg) {
    const uint64_t all = (uint64_t) p.groups * p.unit, at = (uint64_t) ct * p.unit;
    const uint64_t j = ((at + 1) * p.share + all - 1) / all;   // the first CTA whose range starts behind the row group's
    const uint64_t pos = j * all / p.share - at;
    return n_bg - p.unit + (int) min(pos, (uint64_t) p.unit);
}

template <int WTYPE>
struct MsTile {   // a T16 tile as a lane holds it
    uint4 q[WTYPE == B200_TYPE_Q4_0 ? 2 : 4];
    uint2 sa, sb;
};

// FREE: ks divides MS_WARPS and no part is cut.  ROPE: the rows are those of q, k and v (RopeStore)
template <int WTYPE, bool FREE, bool ROPE>
__global__ void __launch_bounds__(MS_THREADS, 1) mmq_stream_kernel(TiledDims dims, const uint8_t *__restrict__ w, ActDims act, const uint8_t *__restrict__ aq,
                                                                float *__restrict__ dst, int64_t dst_nb_row, MsPlan plan, RopeStore rope) {
    constexpr int RING = WTYPE == B200_TYPE_Q4_0 ? 4 : 2, TB = WTYPE == B200_TYPE_Q4_0 ? 1024 : 2048;
    constexpr float WS = WTYPE == B200_TYPE_Q4_0 ? 0.0625f : 1.0f;   // Q4_0 quants are used as 16 * value
    extern __shared__ __align__(128) uint8_t smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int n_bg = (int) dims.n_bg, n_rt = (int) dims.n_rt;
    const int r0 = (int) ((uint64_t) blockIdx.x * (unsigned) n_rt / gridDim.x), n_r = (int) ((uint64_t) (blockIdx.x + 1) * (unsigned) n_rt / gridDim.x) - r0;
    // Task i of the CTA is part i / n_r of row tile i % n_r (FREE: part i % ks of row tile i / ks, 2 % faster at the heads, 6 % slower at 14336 x 4096
    // in 13 parts); a warp takes tasks warp, warp + MS_WARPS, ...
    const int ks = plan.ks, per = plan.per, n_tasks = n_r * ks, d_r = FREE ? MS_WARPS / ks : MS_WARPS % n_r, d_c = FREE ? 0 : MS_WARPS / n_r;
    const bool idle = warp >= n_tasks || (FREE && warp % ks * per >= n_bg);   // (FREE: the last parts may be empty)
    const int r_first = idle ? 0 : FREE ? warp / ks : warp % n_r, c_first = idle ? 0 : FREE ? warp % ks : warp / n_r;
    auto next = [&](int &r, int &c) {   // false: that was the last
        r += d_r;
        c += d_c;
        if (!FREE && r >= n_r) {
            r -= n_r;
            ++c;
        }
        return FREE ? r < n_r : c < ks;
    };
    // the next tile to load: where its quants and scales are, counted from the CTA's first
    const uint8_t *const wq = w + (int64_t) r0 * n_bg * TB, *const ws = w + dims.qs_bytes + (int64_t) r0 * n_bg * 128;
    int lr = r_first, lc = c_first, lend, lgo = 1;
    uint32_t lq, ls;
    auto load_from = [&] {
        const int at = lr * n_bg + lc * per;
        lend = min(per, n_bg - lc * per);
        lq = at * TB + lane * (WTYPE == B200_TYPE_Q4_0 ? 32 : 16);
        ls = at * 128 + g * 8;
    };
    MsTile<WTYPE> ring[RING];
    // (never conditional: a load behind a branch is waited for where the branch ends.  Behind the warp's last tile it is loaded again.)
    auto load = [&](MsTile<WTYPE> &f) {
        if (WTYPE == B200_TYPE_Q4_0) {
            f.q[0] = __ldg(reinterpret_cast<const uint4 *>(wq + lq));
            f.q[1] = __ldg(reinterpret_cast<const uint4 *>(wq + lq + 16));
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) f.q[j % (WTYPE == B200_TYPE_Q4_0 ? 2 : 4)] = __ldg(reinterpret_cast<const uint4 *>(wq + lq + j * 512));
        }
        f.sa = __ldg(reinterpret_cast<const uint2 *>(ws + ls));
        f.sb = __ldg(reinterpret_cast<const uint2 *>(ws + ls + 64));
        if (--lend == 0) {   // on to the warp's next task
            if (next(lr, lc)) load_from();
            else lgo = 0;
        } else {
            lq += lgo * TB;
            ls += lgo * 128;
        }
    };
    int *const cuts = reinterpret_cast<int *>(smem + plan.cuts_at);
    if (!FREE && plan.share) {
        for (int i = tid; i < n_r; i += MS_THREADS) cuts[i] = ms_cut(plan, (r0 + i) / plan.group_tiles, n_bg);
    }

    pdl_prologue();
    load_from();
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
        float *const slot0 = slots + 40 * t + g;
        uint64_t y0 = 0ull, y1 = 0ull;   // rows g, g + 8, columns 2t, 2t + 1
        int r = r_first, c = c_first, part, i_q, i_s, left;   // where in the activations, block groups to the part's end
        auto begin = [&] {
            const int b = c * per, end = !FREE && plan.share != 0 && c == ks - 1 ? cuts[r] : min(b + per, n_bg);
            part = c;
            left = end - b;
            i_q = b * 1024 + lane * 8;
            i_s = q_bytes + b * 256 + t * 16;
        };
        bool work = !idle;
        if (work) begin();
        while (work) {
#pragma unroll
            for (int k = 0; k < RING; ++k) {
                const MsTile<WTYPE> &f = ring[k];
                uint2 b[4];
                uint4 sc[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    b[j] = *reinterpret_cast<const uint2 *>(smem + i_q + j * 256);
                    sc[j] = *reinterpret_cast<const uint4 *>(smem + i_s + j * 64);
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
                i_q += 1024;
                i_s += 256;
                if (--left == 0) {
                    float v0, v1, v2, v3;
                    unpack2(y0, v0, v1);
                    unpack2(y1, v2, v3);
                    float *const slot = slot0 + (r * plan.parts + part) * MS_SLOT;
                    slot[0] = v0 * WS; slot[20] = v1 * WS; slot[8] = v2 * WS; slot[28] = v3 * WS;
                    y0 = y1 = 0ull;
                    if (!FREE && plan.share != 0 && part == ks - 1 && cuts[r] < n_bg) {   // a cut inside the task
                        part = ks;
                        left = n_bg - cuts[r];
                    } else {
                        work = next(r, c);
                        if (!work) break;
                        begin();
                    }
                }
            }
        }
    }
    // The parts of a row tile, in K order.  Threads go over [column][rows], the rows padded to a power of two.
    const int rows = n_r * 16, lg = 32 - __clz(rows - 1), n_e = (int) act.N << lg;
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
            const float *s = slots + (rr >> 4) * plan.parts * MS_SLOT + col * 20 + (rr & 15);
            const int parts = FREE ? plan.parts : plan.share != 0 && cuts[rr >> 4] < n_bg ? ks + 1 : ks;
#pragma unroll 4
            for (int c = 0; c < parts; ++c) v += s[c * MS_SLOT];
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

KSplit mmq_k_split(int wtype, const TiledDims &d, const ActDims &a, bool streamk, bool workspace, size_t workspace_bytes);

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
        const auto allow = [](auto kernel) { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MS_SMEM); };
        allow(mmq_stream_kernel<B200_TYPE_Q4_0, false, false>);
        allow(mmq_stream_kernel<B200_TYPE_Q4_0, false, true>);
        allow(mmq_stream_kernel<B200_TYPE_Q4_0, true, false>);
        allow(mmq_stream_kernel<B200_TYPE_Q8_0, false, false>);
        allow(mmq_stream_kernel<B200_TYPE_Q8_0, false, true>);
        allow(mmq_stream_kernel<B200_TYPE_Q8_0, true, false>);
    }
    return n[dev];
}

// Where this kernel is faster than mmq.cu with the same cuts of K.  Quantiser and product, us on B200, mmq.cu / this at 8 columns (3 columns differ by a
// few per cent):
//   a stream-K deal             Q4_0 4096 x 28672 25.4 / 19.3, 2048 x 32768 16.9 / 11.9, Q8_0 8192 x 32768 1.15 times (8192 x 28672 1.00)
//   one part for all of K       Q4_0 256 x 2048 3.6 / 3.9, 1024 x 32768 9.0 / 10.3, Q8_0 512 x 32768 7.1 / 8.0: few and short row tiles per warp
//   several parts, Q4_0         4096 x 4096 7.9 / 7.3, 14336 x 4096 15.0 / 13.5, 512 x 512 4.6 / 3.8, 4096 x 20480 18.3 / 18.2
//     few rows of a long K      14336 x 256 7.6 / 8.3: 16 SMs copy all the activations, where mmq.cu has 32 CTAs
//   several parts, Q8_0         2048 x 2048 6.1 / 5.2, 4096 x 4096 1.06 times, 2048 x 8192 8.2 / 8.0; beyond some 8192 tiles two of them on their way per
//                               warp are too few: 4096 x 20480 22.9 / 24.4, 8192 x 6144 14.4 / 16.3, 14336 x 6144 21.0 / 26.0; 512 x 24576 6.8 / 7.3
static bool ms_pays(int wtype, const TiledDims &d, const KSplit &s) {
    if (s.sk_ctas) return true;
    if (s.ks == 1 || (d.n_rt <= 32 && d.n_bg > 64)) return false;
    return wtype == B200_TYPE_Q4_0 || (d.n_rt * d.n_bg <= 8192 && d.n_rt <= 1024);
}

// false: mmq.cu is faster, or the activations and partial tiles do not fit into shared memory (K above some 21000); *rc: how the launch went.
// workspace: what mmq.cu would have for its split.  rope: the rows are those of q, k and v, see there
bool launch_mmq_stream(int wtype, const TiledDims &d, const void *w, const ActDims &a, const void *aq, float *dst, int64_t dst_nb_row, bool workspace, size_t workspace_bytes,
                       const RopeStore *rope, cudaStream_t st, int *rc) {
    const int64_t ctas = std::min<int64_t>(ms_sm_count(), d.n_rt), rt = (d.n_rt + ctas - 1) / ctas, act = d.n_bg * 1280, n_bg = d.n_bg;
    if (a.n_nt != 1 || d.n_rt * n_bg >= (1ll << 31) || rt * n_bg * d.tile_bytes >= (1ll << 31)) return false;
    const bool free = d.M >= HEAD_ROWS;
    MsPlan p = {};
    if (free) {
        if (rope) return false;
        // The most warps a row tile (all work to the end) whose partial tiles fit: tiles of the busiest warp, and what a row tile's end costs
        int64_t best = -1;
        for (int ks = MS_WARPS; ks >= 1; ks /= 2) {
            const int64_t chunk = (n_bg + ks - 1) / ks, rounds = (rt * ks + MS_WARPS - 1) / MS_WARPS, cost = rounds * (chunk * 4 + 1);
            if (act + rt * ks * MS_SLOT * 4 > MS_SMEM || (best >= 0 && cost >= best)) continue;
            // (not understood, but steep: with 63 row tiles and more to a CTA four parts take 119 us at Q8_0 4096 x 151936, 1 column, two 101; up to 55 row
            // tiles four are as good as two or better: 4096 x 128256 84.0 / 84.2, 2048 x 102400 Q4_0 24.6 / 25.5)
            if (ks == 4 && rt > 60) continue;
            best = cost;
            p.ks = ks;
            p.per = (int) chunk;
        }
        if (best < 0) return false;
    } else {
        const KSplit s = mmq_k_split(wtype, d, a, true, workspace, workspace_bytes);
        if (!ms_pays(wtype, d, s)) return false;
        p.per = (int) (s.sk_ctas ? (s.sk_head ? s.sk_head : n_bg) : (n_bg + s.ks - 1) / s.ks);
        p.ks = (int) ((n_bg + p.per - 1) / p.per);
        if (s.sk_ctas) {
            p.unit = (int) n_bg - s.sk_head;
            p.group_tiles = s.group_tiles;
            p.groups = (int) (d.n_rt / s.group_tiles);
            p.share = s.sk_head ? s.sk_ctas - p.groups : s.sk_ctas;
        }
    }
    p.parts = (int) ((n_bg + p.per - 1) / p.per) + (p.share ? 1 : 0);
    p.slots_at = (int) act;
    const int64_t cuts_at = act + rt * p.parts * MS_SLOT * 4, bytes = cuts_at + (p.share ? rt * 4 : 0);
    if (bytes > MS_SMEM) return false;
    p.cuts_at = (int) cuts_at;
    const bool q4 = wtype == B200_TYPE_Q4_0;
    const auto kernel = free ? (q4 ? mmq_stream_kernel<B200_TYPE_Q4_0, true, false> : mmq_stream_kernel<B200_TYPE_Q8_0, true, false>)
                        : rope ? (q4 ? mmq_stream_kernel<B200_TYPE_Q4_0, false, true> : mmq_stream_kernel<B200_TYPE_Q8_0, false, true>)
                               : (q4 ? mmq_stream_kernel<B200_TYPE_Q4_0, false, false> : mmq_stream_kernel<B200_TYPE_Q8_0, false, false>);
    launch_pdl(kernel, dim3((unsigned) ctas), dim3(MS_THREADS), (size_t) bytes, st, d, (const uint8_t *) w, a, (const uint8_t *) aq, dst, dst_nb_row, p, rope ? *rope : RopeStore{});
    *rc = check_launch("mmq_stream");
    return true;
}

}  // namespace b200
