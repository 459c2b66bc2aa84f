// Implicit-GEMM convolution for launches that do not fill the GPU: one tile per cluster, the K loop cut across it.
//
// The persistent kernel (conv_tc.cu) keeps 148 SMs busy when there are many tiles.  At one or a few images a layer is a
// handful of tiles with a long K loop (taps x channel blocks): a few SMs work for a long time.  Here every output tile is
// the work of a cluster of S CTAs (2 S with CTA pairs).  CTA s runs K iterations [s*K/S, (s+1)*K/S) into its own TMEM
// accumulator and dumps it, raw, into its own shared memory, over the operand ring its MMAs have finished with; after a
// cluster barrier each CTA finishes the 1/S of the tile's pixels that is its share: it adds the S partial sums of every
// value through distributed shared memory, in rank order (results do not depend on timing), and runs the epilogue (folded
// batchnorm or bias, activation, fused residual or [yolo] logistic, rounding) straight to global memory.  Nothing spins
// on memory: the cluster barrier is the only meeting point, and every wait before it is bounded.
//
// What bounds a launch here is latency, not bandwidth: (set-up + first loads) + K/S iterations + reduction.  So
//  * weights, which no earlier kernel writes, are requested for the whole ring before griddepcontrol.wait: their trip from
//    HBM overlaps the tail of the layer before;
//  * nothing is persistent and nothing is double-buffered: one accumulator, one pass;
//  * tiles are any wt x ht x bt <= 128 box (19 x 6 pixels of a 19x19 map, not 32 x 4): less padded work where tiles are few;
//  * the reduction goes through distributed shared memory (one dump, S loads per value), not through L2 and a counter.
// Measured in a chain of launches: 512 -> 1024 3x3 filters at 19x19, one image, 31 -> 15.4 us (the persistent kernel with
// partial sums through L2: 36 us); 256 -> 256 at 16x16, one image, 16.5 -> 6.8 us.
//
// Replaces forward_convolutional_layer_gpu (src/convolutional_kernels.cu:73-135 of the reference) at small batches.
#include <cuda.h>

#include <atomic>
#include <mutex>

#include "common.h"
#include "conv.h"
#include "device_utils.cuh"
#include "tc_ptx.cuh"

namespace dnb {

constexpr int SP_THREADS = 320;       // a load warp, an MMA warp, eight that drain the accumulator; all ten finish the tile
constexpr int SP_MAX_STAGES = 12;

struct SplitShared {
    uint64_t full[SP_MAX_STAGES];
    uint64_t empty[SP_MAX_STAGES];
    uint64_t acc_full;
    uint32_t tmem_base;
    int abort_flag;
    int pixel[128];            // output pixel ((b * out_h) + oh) * out_w + ow of a tile row, -1 outside the output
    int res_pixel[128];        // pixel of the fused residual that is added there
    long long nchw[128];       // offset of that pixel in Darknet's layout, filter 0
};

enum { SP_WAIT_EMPTY = 101, SP_WAIT_FULL = 102, SP_WAIT_ACC_FULL = 104, SP_BAD_SMEM_BASE = 106 };

__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ uint4 ld_cluster16(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
// both CTAs of this CTA's pair, whatever the size of the cluster
__device__ __forceinline__ void umma_commit_pair_at(uint32_t bar, uint32_t even_rank)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)(3u << even_rank)) : "memory");
}

__device__ __forceinline__ float split_act(float x, int act)
{
    if (act == DNB_LEAKY) return fmaxf(x, 0.1f * x);
    if (act == DNB_LINEAR) return x;
    if (act == DNB_RELU) return x > 0.f ? x : 0.f;
    return activate_call(x, act);
}

// KIND: operand kind (TF32 on f32, bf16, int8 signs).  PAIR: the CTAs of a cluster work in pairs (cta_group::2): a pair
// multiplies two adjacent pixel tiles by one 256-filter tile, each CTA loading its own pixels and half of the filters.
// MAXS: upper bound of S (4 or 8).  What is left after the barrier is a chain of latencies (partial sums, residual, store)
// per value, so a thread keeps its filters' scale and shift and has ROWS_AT_ONCE pixels' loads in flight together.
template <int KIND, bool PAIR, int MAXS>
__global__ void __launch_bounds__(SP_THREADS, 1)
conv_tc_split_kernel(const __grid_constant__ SplitArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t ring = smem_u32(smem_raw);
    if (ring & 1023u) {   // uniform over the cluster: every CTA's window starts at the same offset
        if (threadIdx.x == 0) atomicCAS(a.status, 0, SP_BAD_SMEM_BASE);
        return;
    }
    constexpr bool OUT_BF16 = KIND == MMA_BF16;
    const int stages = a.stages, bn = a.bn, splits = a.splits;
    const uint32_t stage_bytes = a.a_bytes + a.b_bytes, a_bytes = a.a_bytes;
    SplitShared *sh = reinterpret_cast<SplitShared *>(smem_raw + a.work_bytes);
    volatile int *abort_flag = &sh->abort_flag;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int cluster = PAIR ? 2 * splits : splits;
    const int tile = (int)(blockIdx.x / cluster), rank = (int)blockIdx.x - tile * cluster;   // cluster ranks follow blockIdx.x
    const int split = PAIR ? rank >> 1 : rank, parity = PAIR ? rank & 1 : 0;
    const bool leader = parity == 0;

    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(smem_u32(&sh->full[s]), 1);
            mbar_init(smem_u32(&sh->empty[s]), 1);
        }
        mbar_init(smem_u32(&sh->acc_full), 1);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    const uint32_t tmem_cols = (uint32_t)a.tmem_cols;
    if (warp == 1) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();   // the partner's barriers exist before anything is signalled across the pair
    tc_fence_after();
    launch_dependents();            // the next layer's CTAs may take free SMs, run this far and fetch their weights
    const uint32_t tmem_base = sh->tmem_base;

    const int taps = a.taps, c_blocks = a.c_blocks, k_iters = taps * c_blocks;
    const int k0 = split * k_iters / splits, k1 = (split + 1) * k_iters / splits;
    const int n_tiles = a.n_tiles, tiles_w = a.tiles_w, tiles_h = a.tiles_h;
    const int nt = tile % n_tiles, pt = PAIR ? 2 * (tile / n_tiles) + parity : tile / n_tiles;
    const int ow0 = (pt % tiles_w) * a.wt, oh0 = ((pt / tiles_w) % tiles_h) * a.ht, b0 = (pt / (tiles_w * tiles_h)) * a.bt;
    const long long wait_limit = a.wait_limit;
    int *const status = a.status;

    if (warp == 0) {
        // ---------------- loads: the whole warp in step, one elected lane issues
        const int ksize = a.g.size, cstride = a.g.stride, cpad = a.g.pad, bk = a.bk;
        const CUtensorMap *maps = a.tmx, *wmap = &a.tmw;
        const uint32_t tx_bytes = (uint32_t)a.rows * a.row_bytes + (uint32_t)(PAIR ? bn >> 1 : bn) * a.row_bytes;
        const uint32_t full0 = smem_u32(&sh->full[0]), empty0 = smem_u32(&sh->empty[0]);
        const int n0 = nt * bn + (PAIR ? parity * (bn >> 1) : 0);
        const bool withhold = (a.debug & 32) != 0;
        const int ahead = min(stages, k1 - k0);
        {   // the first ring's worth of weights, before the layer before this one has finished
            int tap = k0 / c_blocks, cb = k0 - tap * c_blocks;
            for (int s = 0; s < ahead; ++s) {
                if (elect_one()) {
                    const uint32_t bar = full0 + 8 * s, dst = ring + s * stage_bytes + a_bytes;
                    if (PAIR) {
                        if (leader) mbar_expect_tx(bar, 2u * tx_bytes);
                        tma_load_3d_pair(dst, wmap, bar, cb * bk, n0, tap);
                    } else {
                        mbar_expect_tx(bar, tx_bytes);
                        tma_load_3d(dst, wmap, bar, cb * bk, n0, tap);
                    }
                }
                if (++cb == c_blocks) { cb = 0; ++tap; }
            }
        }
        grid_dependency_wait();
        int ki = k0, tap = k0 / c_blocks, cb = k0 - tap * c_blocks;
        int kh = tap / ksize, kw = tap - kh * ksize, stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        while (ki < k1 && ok) {
            const int dh = kh - cpad, dw = kw - cpad;
            int ph = 0, qh = dh, pw = 0, qw = dw;
            if (cstride == 2) { ph = dh & 1; qh = (dh - ph) >> 1; pw = dw & 1; qw = (dw - pw) >> 1; }
            const CUtensorMap *mx = maps + (ph * cstride + pw);
            const int iw0 = ow0 + qw, ih0 = oh0 + qh, kend = min(k1, ki + c_blocks - cb);
            for (; ki < kend; ++ki, ++cb) {
                const bool first = ki - k0 < ahead;   // the weights of these slots are on their way already
                if (!first) {
                    ok = mbar_wait_warp(empty0 + 8 * stage, phase ^ 1, abort_flag, status, SP_WAIT_EMPTY, wait_limit);
                    if (!ok) break;
                }
                if (withhold && ki == k1 - 1) { ok = false; break; }   // wait-expiry test: the last load is never requested
                if (elect_one()) {
                    const uint32_t bar = full0 + 8 * stage, sa = ring + stage * stage_bytes;
                    if (PAIR) {
                        if (!first && leader) mbar_expect_tx(bar, 2u * tx_bytes);
                        tma_load_4d_pair(sa, mx, bar, cb * bk, iw0, ih0, b0);
                        if (!first) tma_load_3d_pair(sa + a_bytes, wmap, bar, cb * bk, n0, tap);
                    } else {
                        if (!first) mbar_expect_tx(bar, tx_bytes);
                        tma_load_4d(sa, mx, bar, cb * bk, iw0, ih0, b0);
                        if (!first) tma_load_3d(sa + a_bytes, wmap, bar, cb * bk, n0, tap);
                    }
                }
                if (++stage == stages) { stage = 0; phase ^= 1; }
            }
            cb = 0; ++tap;
            if (++kw == ksize) { kw = 0; ++kh; }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMAs
        const uint32_t idesc = mma_idesc<KIND>(PAIR ? 256u : 128u, (uint32_t)bn);
        const int k_steps = a.row_bytes / 32, kn = k1 - k0;
        const uint64_t da0 = make_smem_desc(ring, a.row_bytes), db0 = make_smem_desc(ring + a_bytes, a.row_bytes);
        const uint64_t slot_step = stage_bytes >> 4;
        const uint32_t full0 = smem_u32(&sh->full[0]), empty0 = smem_u32(&sh->empty[0]);
        const uint32_t even = (uint32_t)(rank & ~1);
        int stage = 0;
        uint32_t phase = 0;
        uint64_t da = da0, db = db0;
        bool ok = leader;
        grid_dependency_wait();   // only so that the bounds of the waits below count this launch's own time
        for (int ki = 0; ki < kn && ok; ++ki) {
            ok = mbar_wait_warp(full0 + 8 * stage, phase, abort_flag, status, SP_WAIT_FULL, wait_limit);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                if (PAIR) {
                    umma_pair<KIND>(tmem_base, da, db, idesc, ki != 0);
                    umma_pair<KIND>(tmem_base, da + 2, db + 2, idesc, 1u);
                    umma_pair<KIND>(tmem_base, da + 4, db + 4, idesc, 1u);
                    umma_pair<KIND>(tmem_base, da + 6, db + 6, idesc, 1u);
                    umma_commit_pair_at(empty0 + 8 * stage, even);
                } else {
                    if (k_steps == 4) {
                        umma<KIND>(tmem_base, da, db, idesc, ki != 0);
                        umma<KIND>(tmem_base, da + 2, db + 2, idesc, 1u);
                        umma<KIND>(tmem_base, da + 4, db + 4, idesc, 1u);
                        umma<KIND>(tmem_base, da + 6, db + 6, idesc, 1u);
                    } else {
                        for (int k = 0; k < k_steps; ++k) umma<KIND>(tmem_base, da + 2 * k, db + 2 * k, idesc, (ki | k) != 0);
                    }
                    umma_commit(empty0 + 8 * stage);
                }
            }
            da += slot_step; db += slot_step;
            if (++stage == stages) { stage = 0; phase ^= 1; da = da0; db = db0; }
        }
        if (ok && elect_one()) {
            if (PAIR) umma_commit_pair_at(smem_u32(&sh->acc_full), even); else umma_commit(smem_u32(&sh->acc_full));
        }
        __syncwarp();
    }
    // ---------------- partial sums: TMEM -> shared memory rows of bn + 4 words (the pad spreads a column over the banks)
    const int pitch = bn + 4;
    uint32_t *const part = reinterpret_cast<uint32_t *>(smem_raw);
    const ConvGeom &g = a.g;
    const int r0 = split * a.rows / splits, r1 = (split + 1) * a.rows / splits, R = r1 - r0, qn = bn >> 2;
    const int n_base = nt * bn, n_end = a.n_write;     // channels written: the layer's own, padded to 8 for channels-last output
    // Who finishes what.  Channels-last: a thread keeps four filters and walks pixels, consecutive threads on consecutive
    // filters.  Darknet's layout: consecutive threads on consecutive pixels of one plane; a thread keeps its pixel.
    const bool by_pixel = a.y_nchw != nullptr;
    const int lanes = by_pixel ? (R > 0 ? R : 1) : qn, groups = SP_THREADS / lanes, mine = tid % lanes, first = tid / lanes;
    const int total = first < groups && R > 0 && b0 < g.batch ? (by_pixel ? qn : R) : 0;   // items of this thread's walk
    float4 sc = make_float4(0.f, 0.f, 0.f, 0.f), sf = sc;
    if (warp >= 2) {
        const int quarter = warp & 3, m = quarter * 32 + lane, half = (warp - 2) >> 2;
        if (half == 0) {   // where this row goes, while the MMAs run
            const int wl = m % a.wt, t = m / a.wt, hl = t % a.ht, bl = t / a.ht;
            const int ow = ow0 + wl, oh = oh0 + hl, b = b0 + bl;
            const bool in = m < a.rows && ow < g.out_w && oh < g.out_h && b < g.batch;
            sh->pixel[m] = in ? (b * g.out_h + oh) * g.out_w + ow : -1;
            if (a.ep.residual) {   // (g may hold a 1x1 layer's pixels in one row: back to the map's own rows)
                const int px = in ? sh->pixel[m] : 0, rx = px % a.ep.res_out_w, t2 = px / a.ep.res_out_w, ry = t2 % a.ep.res_out_h, rb = t2 / a.ep.res_out_h;
                sh->res_pixel[m] = (rb * a.ep.res_h + ry * a.ep.res_stride) * a.ep.res_w + rx * a.ep.res_stride;
            }
            sh->nchw[m] = in ? (long long)b * g.n * g.out_h * g.out_w + oh * g.out_w + ow : 0;
        }
        grid_dependency_wait();
        mbar_wait(smem_u32(&sh->acc_full), 0, abort_flag, status, SP_WAIT_ACC_FULL, 0, wait_limit);
        tc_fence_after();
        if (!*abort_flag) {   // (an aborted CTA's loads may still be landing where the dump goes; its tile is incomplete anyway)
            const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
            uint32_t *row = part + (size_t)m * pitch;
#pragma unroll 1
            for (int c0 = 32 * half; c0 < bn; c0 += 64) {
                uint32_t v[32];
                tmem_ld16(t_row + c0, *reinterpret_cast<uint32_t(*)[16]>(&v[0]));
                if (c0 + 16 < bn) tmem_ld16(t_row + c0 + 16, *reinterpret_cast<uint32_t(*)[16]>(&v[16]));
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (q < 4 || c0 + 16 < bn) *reinterpret_cast<uint4 *>(row + c0 + 4 * q) = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            }
        }
        tc_fence_before();
    }
    __syncwarp();
    if (total && !by_pixel && n_base + 4 * mine < n_end) {       // parameters: no earlier kernel writes them
        sc = __ldg(reinterpret_cast<const float4 *>(a.ep.scale + n_base + 4 * mine));
        sf = __ldg(reinterpret_cast<const float4 *>(a.ep.shift + n_base + 4 * mine));
    }
    __syncwarp();
    cluster_sync_all();
    grid_dependency_wait();   // the residual is read and the output written from here on

    // ---------------- this CTA's share of the tile's pixels
    if (total) {
        constexpr int ROWS_AT_ONCE = MAXS <= 4 ? 4 : 2;
        uint32_t peer[MAXS];
        const uint32_t part_addr = smem_u32(part);
#pragma unroll
        for (int s = 0; s < MAXS; ++s) peer[s] = s < splits ? map_to_rank(part_addr, (uint32_t)(PAIR ? 2 * s + parity : s)) : part_addr;
        const int act = a.ep.activation, act2 = a.ep.activation2, do_round = a.ep.round_tf32, yolo = a.ep.yolo_entries;
        const size_t plane = (size_t)g.out_h * g.out_w;
        for (int i0 = first; i0 < total; i0 += groups * ROWS_AT_ONCE) {
            uint4 p[ROWS_AT_ONCE][MAXS];
            uint4 res[ROWS_AT_ONCE];
            int pixel[ROWS_AT_ONCE];
#pragma unroll
            for (int u = 0; u < ROWS_AT_ONCE; ++u) {
                const int i = i0 + u * groups;
                const int row = r0 + (by_pixel ? mine : i), q = by_pixel ? i : mine;
                pixel[u] = i < total && n_base + 4 * q < n_end ? sh->pixel[row] : -1;
                if (pixel[u] < 0) continue;
                const uint32_t off = (uint32_t)(row * pitch + 4 * q) * 4u;
#pragma unroll
                for (int s = 0; s < MAXS; ++s)
                    if (s < splits) {   // this CTA's own sums by a plain load: distributed shared memory moves about 15 bytes per clock and SM
                        if (s == split) p[u][s] = *reinterpret_cast<const uint4 *>(part + (size_t)row * pitch + 4 * q);
                        else p[u][s] = ld_cluster16(peer[s] + off);
                    }
                res[u] = make_uint4(0u, 0u, 0u, 0u);
                if (a.ep.residual && n_base + 4 * q < a.ep.res_c) {   // channels beyond the residual's get no addend
                    const size_t at = (size_t)sh->res_pixel[row] * a.ep.res_cpitch + n_base + 4 * q;
                    if (!OUT_BF16) res[u] = __ldg(reinterpret_cast<const uint4 *>(reinterpret_cast<const float *>(a.ep.residual) + at));
                    else { const uint2 r = __ldg(reinterpret_cast<const uint2 *>(reinterpret_cast<const __nv_bfloat16 *>(a.ep.residual) + at)); res[u].x = r.x; res[u].y = r.y; }
                }
            }
#pragma unroll
            for (int u = 0; u < ROWS_AT_ONCE; ++u) {
                if (pixel[u] < 0) continue;
                const int i = i0 + u * groups;
                const int row = r0 + (by_pixel ? mine : i), q = by_pixel ? i : mine, n = n_base + 4 * q;
                uint32_t sum[4] = {p[u][0].x, p[u][0].y, p[u][0].z, p[u][0].w};
#pragma unroll
                for (int s = 1; s < MAXS; ++s)
                    if (s < splits) {
                        const uint32_t w[4] = {p[u][s].x, p[u][s].y, p[u][s].z, p[u][s].w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) sum[e] = KIND == MMA_I8 ? sum[e] + w[e] : __float_as_uint(__uint_as_float(sum[e]) + __uint_as_float(w[e]));
                    }
                if (by_pixel) {
                    sc = __ldg(reinterpret_cast<const float4 *>(a.ep.scale + n));
                    sf = __ldg(reinterpret_cast<const float4 *>(a.ep.shift + n));
                }
                const float scv[4] = {sc.x, sc.y, sc.z, sc.w}, sfv[4] = {sf.x, sf.y, sf.z, sf.w};
                float o[4], rv[4];
                if (!OUT_BF16) { rv[0] = __uint_as_float(res[u].x); rv[1] = __uint_as_float(res[u].y); rv[2] = __uint_as_float(res[u].z); rv[3] = __uint_as_float(res[u].w); }
                else { rv[0] = __uint_as_float(res[u].x << 16); rv[1] = __uint_as_float(res[u].x & 0xffff0000u); rv[2] = __uint_as_float(res[u].y << 16); rv[3] = __uint_as_float(res[u].y & 0xffff0000u); }
                int entry = yolo > 0 ? n % yolo : 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float acc = KIND == MMA_I8 ? (float)(int)sum[e] : __uint_as_float(sum[e]);
                    float v = split_act(fmaf(acc, scv[e], sfv[e]), act);
                    if (yolo > 0) {   // forward_yolo_layer_gpu (src/yolo_layer.c:351-357): logistic on x, y, objectness, classes
                        if (entry < 2 || entry >= 4) v = __fdividef(1.f, 1.f + __expf(-v));
                        if (++entry == yolo) entry = 0;
                    }
                    if (a.ep.residual) v = split_act(a.ep.alpha * v + a.ep.beta * rv[e], act2);
                    if (!OUT_BF16 && do_round) v = round_tf32(v);
                    o[e] = n + e < g.n ? v : 0.f;
                    if (KIND == MMA_I8 && a.ep.raw_acc) o[e] = __uint_as_float(sum[e]);   // the integer sums themselves
                }
                uint2 h = make_uint2(0u, 0u);
                if (OUT_BF16) {
                    __nv_bfloat162 lo = __floats2bfloat162_rn(o[0], o[1]), hi = __floats2bfloat162_rn(o[2], o[3]);
                    h = make_uint2(*reinterpret_cast<uint32_t *>(&lo), *reinterpret_cast<uint32_t *>(&hi));
                }
                if (a.y_nhwc) {
                    const size_t at = (size_t)pixel[u] * a.y_cpitch + n;
                    if (!OUT_BF16) *reinterpret_cast<float4 *>(reinterpret_cast<float *>(a.y_nhwc) + at) = make_float4(o[0], o[1], o[2], o[3]);
                    else *reinterpret_cast<uint2 *>(reinterpret_cast<__nv_bfloat16 *>(a.y_nhwc) + at) = h;
                }
                if (KIND == MMA_I8 && a.sign_out) {   // the next xnor layer's operand: +1 where > 0, else -1, 0 beyond the layer's filters
                    uint32_t w = 0;
#pragma unroll
                    for (int e = 0; e < 4; ++e) w |= (n + e < g.n ? (o[e] > 0.f ? 0x01u : 0xFFu) : 0u) << (8 * e);
                    *reinterpret_cast<uint32_t *>(reinterpret_cast<int8_t *>(a.sign_out) + (size_t)pixel[u] * a.sign_cpitch + n) = w;
                }
                if (a.y_nchw) {
                    float *dst = a.y_nchw + sh->nchw[row] + (size_t)n * plane;
                    if (OUT_BF16) {   // what the channels-last copy holds
                        o[0] = __uint_as_float(h.x << 16); o[1] = __uint_as_float(h.x & 0xffff0000u);
                        o[2] = __uint_as_float(h.y << 16); o[3] = __uint_as_float(h.y & 0xffff0000u);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (n + e < g.n) dst[(size_t)e * plane] = o[e];
                }
            }
        }
    }
    __syncwarp();
    cluster_sync_all();   // nobody's shared memory, barriers or TMEM go away while a peer may use them

    // ---------------- teardown (also the abort path)
    if (*abort_flag) {   // loads still in flight land before shared memory is released
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000LL) { }
    }
    __syncthreads();
    if (PAIR) cluster_sync_all();
    if (warp == 1) {
        tc_fence_after();
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
    if (PAIR) cluster_sync_all();
}

// ------------------------------------------------------------------ host side
size_t conv_tc_split_smem(int stages, int stage_bytes, int bn, int *work_bytes)
{
    size_t work = (size_t)stages * stage_bytes, dump = (size_t)128 * (bn + 4) * 4;
    if (dump > work) work = dump;
    int cols = 32;
    while (cols < bn) cols *= 2;
    work = (work + 15) / 16 * 16;
    if (work_bytes) *work_bytes = (int)work;
    return tmem_smem(work + sizeof(SplitShared) + 16, cols);
}

typedef void (*SplitKernel)(SplitArgs);
static int split_class(int splits) { return splits <= 4 ? 0 : 1; }
template <int KIND, bool PAIR>
static SplitKernel kernel_of_class(int cls)
{
    return cls == 0 ? conv_tc_split_kernel<KIND, PAIR, 4> : conv_tc_split_kernel<KIND, PAIR, 8>;
}
static SplitKernel kernel_of(int kind, int pair, int cls)
{
    if (kind == 1) return pair ? kernel_of_class<MMA_BF16, true>(cls) : kernel_of_class<MMA_BF16, false>(cls);
    if (kind == 2) return pair ? kernel_of_class<MMA_I8, true>(cls) : kernel_of_class<MMA_I8, false>(cls);
    return pair ? kernel_of_class<MMA_TF32, true>(cls) : kernel_of_class<MMA_TF32, false>(cls);
}

// The kernel's attributes, set once per kernel and device (twice, where two threads come at once: harmless).
static int prepare_kernel(int kind, int pair, int cls)
{
    static std::atomic<bool> done[64][3][2][2];
    int dev = 0;
    DNB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) DNB_FAIL(DNB_ECUDA, "conv_tc_split: device %d", dev);
    std::atomic<bool> &d = done[dev][kind][pair ? 1 : 0][cls];
    if (d.load(std::memory_order_acquire)) return DNB_OK;
    const SplitKernel kern = kernel_of(kind, pair, cls);
    DNB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, conv_tc_max_smem()));
    DNB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    d.store(true, std::memory_order_release);
    return DNB_OK;
}

// Clusters of `cluster` CTAs, each with an SM to itself, that the device holds at once (0: none).  Asked once per size and
// device: every plan of a network compares a few dozen splits.
int conv_tc_split_resident(int pair, int cluster)
{
    static std::mutex lock;
    static int known[64][2][17];   // answer + 1
    int dev = 0;
    if (cluster < 1 || cluster > 16 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    std::lock_guard<std::mutex> guard(lock);
    int &slot = known[dev][pair ? 1 : 0][cluster];
    if (slot) return slot - 1;
    if (prepare_kernel(0, pair, 1) != DNB_OK) return 0;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)cluster * 512u);
    cfg.blockDim = dim3(SP_THREADS);
    cfg.dynamicSmemBytes = (size_t)conv_tc_max_smem();
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel_of(0, pair, 1), &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
    slot = n + 1;
    return n;
}

int launch_conv_tc_split(const SplitArgs &a, cudaStream_t s)
{
    if (a.kind < 0 || a.kind > 2) DNB_FAIL(DNB_EINVAL, "conv_tc_split: operand kind %d", a.kind);
    if (a.splits < 2 || a.splits > 8 || a.stages < 2 || a.stages > SP_MAX_STAGES || a.bn < 16 || a.bn > 256 || a.bn % 16 || a.rows < 1 || a.rows > 128)
        DNB_FAIL(DNB_EINVAL, "conv_tc_split: plan out of range (splits %d, stages %d, bn %d, rows %d)", a.splits, a.stages, a.bn, a.rows);
    if (a.pair && (a.bn != 256 || a.row_bytes != 128)) DNB_FAIL(DNB_EINVAL, "conv_tc_split: pairs run 256-filter tiles over 128-byte rows");
    const int cls = split_class(a.splits);
    DNB_TRY(prepare_kernel(a.kind, a.pair, cls));
    const unsigned cluster = (unsigned)(a.pair ? 2 * a.splits : a.splits);
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = cluster; attrs[1].val.clusterDim.y = 1; attrs[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)a.tiles * cluster);
    cfg.blockDim = dim3(SP_THREADS);
    cfg.dynamicSmemBytes = conv_tc_split_smem(a.stages, a.a_bytes + a.b_bytes, a.bn, nullptr);
    cfg.stream = s;
    cfg.attrs = attrs;
    cfg.numAttrs = 2;
    DNB_CUDA(cudaLaunchKernelEx(&cfg, kernel_of(a.kind, a.pair, cls), a));
    DNB_LAUNCH_CHECK("conv_tc_split");
    return DNB_OK;
}

}  // namespace dnb
