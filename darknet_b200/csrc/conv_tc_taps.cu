// 3x3 convolutions with stride 1 and padding 1 on the sm_100a tensor cores: one load of pixels serves all nine taps.
//
// conv_tc.cu loads 128 pixels and a filter tile for every tap and block of channels.  With pairs over 256 filters that is 32 KB a CTA for MMAs of 512
// clocks, which is what an SM's way from L2 carries (64 bytes a clock): the tensor pipe waits for operands.  Here the map is walked as if it had one column
// of zeros before each row and one row of zeros before each image: output pixels are consecutive positions of that order, and a tap is a
// constant distance, kh * (w + 1) + kw.  A tile of 128 positions needs 128 + 2 * (w + 1) + 2 of them, whatever the map and however many images it spans;
// one TMA load in im2col mode brings them (its bounding box is the map with that column and row, its fill is their zeros), and the nine taps'
// MMAs start their A descriptors kh * (w + 1) + kw rows further down (the 128-byte swizzle is a function of the shared-memory address, so a
// descriptor may start at any row).  What is left to load for a tap and 32 channels (TF32) is the filters: 16 KB for half of 256, and a ninth of the pixels.
// Positions of the extra column and row are multiplied like any other and not stored: (w + 1)(h + 1) / (w h) of the work, less than
// the boxes of conv_tc.cu pad on most maps.
//
// Roles (352 threads, CTA pairs with cta_group::2 MMAs): warp 0 loads filters, warp 10 pixels, warp 1 of the even CTA issues the MMAs, warps 2..9 drain the
// accumulator: each a chunk of 128 bytes of every pixel of its 32, staged in rows of its own, stored eight lanes a pixel.  No two epilogue warps meet.
// Where the layer's filters fit shared memory beside two boxes they are loaded once (64 -> 64 in TF32).
// Wide maps are cut into boxes of 8 x 16 pixels instead (boxes): a load is one of 10 x 18, eight-row groups of the A operand are ten rows apart, and what a row
// of such a load costs is a third of what one of an im2col load does (1.1 ns, 3.7), of which a map of 304 columns would want 740 a tile.
// 1x1 layers run here too (ONE): a position is a pixel of the batch, a plain load of 128 of them serves a block of channels; what is gained there is that the
// filters stay in shared memory (512 -> 256 in bf16: 128 KB of each CTA of a pair) and the stores in Darknet's layout.
// K runs over blocks of channels, then taps (conv_tc.cu and conv_tc_split.cu: taps, then blocks).
//
// Replaces forward_convolutional_layer_gpu (src/convolutional_kernels.cu:73-135 of the reference), and the shortcut layer after it
// (src/shortcut_layer.c:75-80), for these layers.
#include <cuda.h>

#include <map>
#include <mutex>
#include <tuple>

#include "common.h"
#include "conv.h"
#include "device_utils.cuh"
#include "tc_ptx.cuh"

namespace dnb {

constexpr int TAPS_THREADS = 352;
constexpr int TAPS_RES_ROWS = 3;   // sets of staged rows of a warp where a residual lands in them

struct TapsShared {
    uint64_t x_full[TAPS_MAX_X], x_empty[TAPS_MAX_X];
    uint64_t w_full[TAPS_MAX_W], w_empty[TAPS_MAX_W];
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    int abort_flag;
};

enum { TAPS_WAIT_EMPTY = 101, TAPS_WAIT_FULL = 102, TAPS_WAIT_ACC_EMPTY = 103, TAPS_WAIT_ACC_FULL = 104, TAPS_BAD_SMEM_BASE = 106 };

constexpr int TAPS_YOLO = -3;   // linear, then the logistic of a [yolo] layer on every entry but w and h of each anchor (1x1 layers, Darknet's layout)

template <int ACT>
__device__ __forceinline__ float taps_act(float x)
{
    return ACT == DNB_LEAKY ? fmaxf(x, 0.1f * x) : x;
}

// RES: a residual of the output's shape is added, then ACT2 (the other of the two activations).
// ONE: a 1x1 layer: positions are the pixels of the whole batch, a block of channels has one tap.
template <int ACT, bool BF16, bool RES, bool ONE>
__global__ void __launch_bounds__(TAPS_THREADS, 1)
conv_tc_taps_kernel(const __grid_constant__ TapsArgs a)
{
    constexpr int KIND = BF16 ? MMA_BF16 : MMA_TF32, OES = BF16 ? 2 : 4, CPC = 128 / OES;   // CPC: columns of a chunk
    constexpr int ACT2 = ACT == DNB_LEAKY ? DNB_LINEAR : DNB_LEAKY, TAPS = ONE ? 1 : 9;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t ring = smem_u32(smem_raw);
    if (ring & 1023u) {   // uniform over the pair: both CTAs' windows start at the same offset
        if (threadIdx.x == 0) atomicCAS(a.status, 0, TAPS_BAD_SMEM_BASE);
        return;
    }
    const uint32_t w_ring = ring + a.x_stages * a.x_slot;
    uint8_t *const stage_out = smem_raw + a.x_stages * a.x_slot + a.w_stages * a.w_bytes;
    float *const s_scale = reinterpret_cast<float *>(stage_out + a.staged_bytes);
    float *const s_shift = s_scale + a.table;
    TapsShared *const sh = reinterpret_cast<TapsShared *>(s_shift + a.table);
    volatile int *const abort_flag = &sh->abort_flag;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t cta_rank = cluster_ctarank();
    const bool leader = cta_rank == 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < TAPS_MAX_X; ++s) { mbar_init(smem_u32(&sh->x_full[s]), 1); mbar_init(smem_u32(&sh->x_empty[s]), 1); }
        for (int s = 0; s < TAPS_MAX_W; ++s) { mbar_init(smem_u32(&sh->w_full[s]), 1); mbar_init(smem_u32(&sh->w_empty[s]), 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&sh->acc_full[i]), 1); mbar_init(smem_u32(&sh->acc_empty[i]), 16); }   // the epilogue warps of both CTAs
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    const uint32_t tmem_cols = (uint32_t)a.tmem_cols, acc_stride = tmem_cols / 2;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    // scale and shift of all filters, which no kernel of the stream writes
    for (int i = threadIdx.x; i < a.table; i += TAPS_THREADS) {
        s_scale[i] = i < a.n_pad ? __ldg(a.ep.scale + i) : 0.f;
        s_shift[i] = i < a.n_pad ? __ldg(a.ep.shift + i) : 0.f;
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the other CTA's barriers are initialised before anything is signalled across the pair
    tc_fence_after();
    launch_dependents();
    const uint32_t tmem_base = sh->tmem_base;

    const int c_blocks = a.c_blocks, n_tiles = a.n_tiles, total_tiles = a.total_tiles, bn = a.bn, pitch = a.pitch;
    const bool boxes = !ONE && a.boxes != 0;
    const int tile_step = (int)(gridDim.x >> 1), first_tile = (int)(blockIdx.x >> 1);
    const long long wait_limit = a.wait_limit;
    int *const status = a.status;
    auto pixel_tile = [&](int tile) { return 2 * (tile / n_tiles) + (int)cta_rank; };

    if (warp == 0) {
        // ---------------- filters: the whole warp runs the loop, an elected lane issues
        const CUtensorMap *const map = &a.tmw;
        const int bk = a.bk, stages = a.w_stages, half = bn >> 1;
        const uint32_t bytes = (uint32_t)half * 128u, slot_bytes = a.w_bytes;
        const uint32_t full0 = smem_u32(&sh->w_full[0]), empty0 = smem_u32(&sh->w_empty[0]);
        const bool resident = a.resident != 0, withhold = (a.debug & 32) != 0;
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        // resident: once each of the filter tiles that this pair's tiles have (they come round in a cycle), in the slot that is its own.  No other: nobody
        // would wait for its load, which could still be on its way when the CTA's shared memory is given back.
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
            const int nt = tile % n_tiles, n0 = nt * bn + (int)cta_rank * half;
            if (resident && tile != first_tile && nt == first_tile % n_tiles) break;
            if (resident) { stage = nt * c_blocks * TAPS; phase = 0; }
            for (int cb = 0; cb < c_blocks && ok; ++cb)
                for (int tap = 0; tap < TAPS; ++tap) {
                    ok = mbar_wait_warp(empty0 + 8 * stage, phase ^ 1, abort_flag, status, TAPS_WAIT_EMPTY, wait_limit);
                    if (!ok) break;
                    if (withhold && tile == first_tile && cb == c_blocks - 1 && tap == TAPS - 1) { ok = false; break; }   // wait-expiry test
                    if (elect_one()) {
                        const uint32_t bar = full0 + 8 * stage;
                        if (leader) mbar_expect_tx(bar, 2u * bytes);
                        tma_load_3d_pair(w_ring + stage * slot_bytes, map, bar, cb * bk, n0, tap);
                    }
                    __syncwarp();
                    if (++stage == stages) { stage = 0; phase ^= 1; }
                }
        }
        __syncwarp();
    } else if (warp == 10) {
        // ---------------- pixels: one load of `rows` positions per block of channels
        const CUtensorMap *const map = &a.tmx;
        const int bk = a.bk, stages = a.x_stages, h1 = a.g.h + 1, last = a.ptiles - 1;
        const uint32_t bytes = (uint32_t)a.rows * 128u, slot_bytes = a.x_slot;
        const uint32_t full0 = smem_u32(&sh->x_full[0]), empty0 = smem_u32(&sh->x_empty[0]);
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        grid_dependency_wait();
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
            const int pt = min(pixel_tile(tile), last);   // the second CTA of the last of an odd number of pixel tiles does the first's again, and stores nothing
            int at = pt * 128, x0 = 0, y0 = 0, img = 0;
            if (!ONE && boxes) {
                const int tw = pt % a.tiles_w, t = pt / a.tiles_w, th = t % a.tiles_h;
                x0 = 8 * tw - 1; y0 = 16 * th - 1; img = t / a.tiles_h;
            } else if (!ONE) {
                const int row = at / pitch;
                img = row / h1;
                x0 = at - row * pitch - 1; y0 = row - img * h1 - 1;
            }
            for (int cb = 0; cb < c_blocks; ++cb) {
                ok = mbar_wait_warp(empty0 + 8 * stage, phase ^ 1, abort_flag, status, TAPS_WAIT_EMPTY, wait_limit);
                if (!ok) break;
                if (elect_one()) {
                    const uint32_t bar = full0 + 8 * stage;
                    if (leader) mbar_expect_tx(bar, 2u * bytes);
                    if (ONE) tma_load_3d_pair(ring + stage * slot_bytes, map, bar, cb * bk, at, 0);
                    else if (boxes) tma_load_4d_pair(ring + stage * slot_bytes, map, bar, cb * bk, x0, y0, img);
                    else tma_load_im2col_4d_pair(ring + stage * slot_bytes, map, bar, cb * bk, x0, y0, img);
                }
                __syncwarp();
                if (++stage == stages) { stage = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMAs of both CTAs, by the even one: the same descriptors address either's shared memory
        if (leader) {
            const uint32_t idesc = mma_idesc<KIND>(256u, (uint32_t)bn);
            const int w_stages = a.w_stages, x_stages = a.x_stages;
            uint64_t dx0 = make_smem_desc(ring, 128);
            if (boxes) dx0 = (dx0 & ~((uint64_t)0x3FFF << 32)) | ((uint64_t)(pitch * 8) << 32);   // groups of eight rows: a box's rows apart
            const uint64_t dw0 = make_smem_desc(w_ring, 128);
            const uint64_t x_step = a.x_slot >> 4, w_step = a.w_bytes >> 4, row_step = (uint64_t)(pitch - 2) * 8;   // from tap (kh, 2) to (kh + 1, 0)
            const uint32_t xf = smem_u32(&sh->x_full[0]), xe = smem_u32(&sh->x_empty[0]), wf = smem_u32(&sh->w_full[0]), we = smem_u32(&sh->w_empty[0]);
            const bool resident = a.resident != 0, no_mma = (a.debug & 16) != 0;
            int xs = 0, ws = 0, it = 0;
            uint32_t xp = 0, wp = 0;
            uint64_t dx = dx0, dw = dw0;
            bool ok = true;
            grid_dependency_wait();   // only so that the bounds of the waits below count this launch's own time
            for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step, ++it) {
                const int acc = it & 1;
                ok = mbar_wait_warp(smem_u32(&sh->acc_empty[acc]), ((it >> 1) & 1) ^ 1, abort_flag, status, TAPS_WAIT_ACC_EMPTY, wait_limit);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * acc_stride;
                if (resident && n_tiles > 1) { ws = (tile % n_tiles) * c_blocks * TAPS; dw = dw0 + (uint64_t)ws * w_step; }
                for (int cb = 0; cb < c_blocks && ok; ++cb) {
                    ok = mbar_wait_warp(xf + 8 * xs, xp, abort_flag, status, TAPS_WAIT_FULL, wait_limit);
                    if (!ok) break;
                    uint64_t da = dx;
                    for (int kh = 0; kh < (ONE ? 1 : 3) && ok; ++kh, da += row_step)
                        for (int kw = 0; kw < (ONE ? 1 : 3); ++kw) {
                            ok = mbar_wait_warp(wf + 8 * ws, wp, abort_flag, status, TAPS_WAIT_FULL, wait_limit);
                            if (!ok) break;
                            tc_fence_after();
                            if (elect_one()) {
                                if (!no_mma) {
                                    umma_pair<KIND>(d_tmem, da, dw, idesc, (uint32_t)((cb | kh | kw) != 0));
                                    umma_pair<KIND>(d_tmem, da + 2, dw + 2, idesc, 1u);
                                    umma_pair<KIND>(d_tmem, da + 4, dw + 4, idesc, 1u);
                                    umma_pair<KIND>(d_tmem, da + 6, dw + 6, idesc, 1u);
                                }
                                if (!resident) umma_commit_pair(we + 8 * ws);
                            }
                            if (!ONE && kw < 2) da += 8;
                            dw += w_step;
                            if (++ws == w_stages) { ws = 0; wp ^= resident ? 0u : 1u; dw = dw0; }
                        }
                    if (!ok) break;
                    if (elect_one()) umma_commit_pair(xe + 8 * xs);
                    dx += x_step;
                    if (++xs == x_stages) { xs = 0; xp ^= 1; dx = dx0; }
                }
                if (ok && elect_one()) umma_commit_pair(smem_u32(&sh->acc_full[acc]));
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue: TMEM lanes 32 * (warp % 4) .. + 31; of the sequence of a CTA's chunks a group of four warps takes every other one
        grid_dependency_wait();
        const int group = (warp - 2) >> 2, quarter = warp & 3, chunks = (bn + CPC - 1) / CPC;
        const ConvGeom g = a.g;
        const int h1 = g.h + 1, plane = g.h * g.w, ptiles = a.ptiles, y_chan = a.y_chan, do_round = a.ep.round_tf32;
        uint8_t *const y_nhwc = reinterpret_cast<uint8_t *>(a.y_nhwc);
        float *const y_nchw = a.y_nchw;
        const size_t y_pix = (size_t)a.y_cpitch * OES, res_pix = RES ? (size_t)a.ep.res_cpitch * OES : 0;
        const uint8_t *const res_base = reinterpret_cast<const uint8_t *>(a.ep.residual);
        const float alpha = a.ep.alpha, beta = a.ep.beta;
        const int dbg = a.debug, yolo_entries = ACT == TAPS_YOLO ? a.ep.yolo_entries : 1;
        uint8_t *const staged0 = stage_out + (size_t)(warp - 2) * (RES ? TAPS_RES_ROWS * 4096 : 4096);
        // the pixel of this lane's position of a tile, -1 for one of the extra column or row, or past the batch
        auto pixel_of = [&](int tile, int &b, int &y, int &x) {
            const int pt = pixel_tile(tile);
            if (ONE) {   // (b and x: the image and the pixel of its plane, for Darknet's layout only)
                const int f = pt * 128 + quarter * 32 + lane;
                b = y = 0;
                x = f;
                if (y_nchw) { b = f / plane; x = f - b * plane; }
                return pt < ptiles && f < a.pixels ? f : -1;
            }
            if (boxes) {
                const int m = quarter * 32 + lane, tw = pt % a.tiles_w, t = pt / a.tiles_w, th = t % a.tiles_h;
                b = t / a.tiles_h;
                x = 8 * tw + (m & 7); y = 16 * th + (m >> 3);
                return pt < ptiles && x < g.w && y < g.h ? (b * g.h + y) * g.w + x : -1;
            }
            const int f = pt * 128 + pitch + 1 + quarter * 32 + lane, row = f / pitch;
            x = f - row * pitch - 1;
            b = row / h1;
            y = row - b * h1 - 1;
            return pt < ptiles && x >= 0 && y >= 0 && b < g.batch ? (b * g.h + y) * g.w + x : -1;
        };
        const int piece = lane & 7, sub = lane >> 3, q_xor = lane & 7;

        // Residual: 128 bytes of each of the warp's 32 pixels, eight lanes a pixel, into the staged rows, two chunks ahead and across tiles.
        int pf_tile = first_tile, pf_c = group, pf_pixel = -1, pf_at = -1;
        uint32_t pf_rows = 0, rows_now = 0;   // which of the staged rows the next request, this chunk has
        auto request_residual = [&]() {
            while (pf_c >= chunks) { pf_c -= chunks; pf_tile += tile_step; }
            if (pf_tile < total_tiles && !(dbg & 1)) {
                if (pf_at != pf_tile) {
                    int b, y, x;
                    pf_pixel = pixel_of(pf_tile, b, y, x);
                    pf_at = pf_tile;
                }
                const int ch = (pf_tile % n_tiles) * bn + pf_c * CPC + piece * (16 / OES);
                const uint32_t dst = smem_u32(staged0 + pf_rows * 4096);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = 4 * i + sub, px = __shfl_sync(0xffffffffu, pf_pixel, r);
                    const bool in = px >= 0 && ch < y_chan;
                    cp_async16(dst + r * 128 + ((piece ^ (r & 7)) << 4), in ? res_base + (size_t)px * res_pix + (size_t)ch * OES : res_base, in);
                }
            }
            pf_c += 2;
            if (++pf_rows == TAPS_RES_ROWS) pf_rows = 0;
            cp_async_commit();
        };
        if (RES)
            for (int i = 1; i < TAPS_RES_ROWS; ++i) request_residual();

        int it = 0, c = group;
        for (int tile = first_tile; tile < total_tiles; tile += tile_step, ++it) {
            const int acc = it & 1, nt = tile % n_tiles;
            int b, y, x;
            const int pixel = pixel_of(tile, b, y, x);
            if (!mbar_wait(smem_u32(&sh->acc_full[acc]), (it >> 1) & 1, abort_flag, status, TAPS_WAIT_ACC_FULL, 0, wait_limit)) break;
            tc_fence_after();
            const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * acc_stride;
#pragma unroll 1
            for (; c < chunks; c += 2) {
                const int c0 = c * CPC;
                if (dbg & 8) continue;
                uint8_t *const staged = staged0 + rows_now * 4096, *const row = staged + lane * 128;
                if (RES && ++rows_now == TAPS_RES_ROWS) rows_now = 0;
                if (RES) {
                    cp_async_wait<TAPS_RES_ROWS - 2>();
                    __syncwarp();            // ... of all lanes; and their stores have read the last chunk's rows
                    request_residual();
                }
                uint32_t r[CPC];
#pragma unroll
                for (int u = 0; u < CPC / 16; ++u) {
                    if (c0 + 16 * u < bn) {
                        tmem_ld16(t_row + c0 + 16 * u, *reinterpret_cast<uint32_t(*)[16]>(&r[16 * u]));
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j) r[16 * u + j] = 0u;
                    }
                }
                tmem_ld_wait();
                const int nl0 = nt * bn + c0;
                int entry = ACT == TAPS_YOLO ? nl0 % yolo_entries : 0;   // of the chunk's first column: the same for the whole warp
                const float4 *const sc4 = reinterpret_cast<const float4 *>(s_scale + nl0), *const sf4 = reinterpret_cast<const float4 *>(s_shift + nl0);
#pragma unroll
                for (int q = 0; q < CPC / 4; ++q) {
                    const float4 sc = sc4[q], sf = sf4[q];
                    const float scv[4] = {sc.x, sc.y, sc.z, sc.w}, sfv[4] = {sf.x, sf.y, sf.z, sf.w};
                    uint4 rv = make_uint4(0u, 0u, 0u, 0u);
                    if (RES && !(dbg & 1)) {
                        if (!BF16) rv = *reinterpret_cast<const uint4 *>(row + ((q ^ q_xor) << 4));
                        else {
                            const uint2 h = *reinterpret_cast<const uint2 *>(row + (((q >> 1) ^ q_xor) << 4) + 8 * (q & 1));
                            rv = make_uint4(h.x << 16, h.x & 0xffff0000u, h.y << 16, h.y & 0xffff0000u);
                        }
                    }
                    const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        float t = taps_act<ACT>(fmaf(__uint_as_float(r[4 * q + e]), scv[e], sfv[e]));
                        if (ACT == TAPS_YOLO) {   // forward_yolo_layer_gpu (src/yolo_layer.c:351-357)
                            if (entry < 2 || entry >= 4) t = __fdividef(1.f, 1.f + __expf(-t));
                            if (++entry == yolo_entries) entry = 0;
                        }
                        if (RES) t = taps_act<ACT2>(alpha * t + beta * __uint_as_float(rw[e]));
                        r[4 * q + e] = __float_as_uint(!BF16 && do_round ? round_tf32(t) : t);
                    }
                }
                if (y_nhwc) {
                    __syncwarp();            // the last chunk's rows have been read
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        uint4 v;
                        if (!BF16) v = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
                        else {
                            uint32_t w[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[(8 * q + 2 * e) % CPC]), __uint_as_float(r[(8 * q + 2 * e + 1) % CPC]));
                                w[e] = *reinterpret_cast<const uint32_t *>(&h);
                            }
                            v = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                        *reinterpret_cast<uint4 *>(row + ((q ^ q_xor) << 4)) = v;
                    }
                    __syncwarp();
                    const int ch = nl0 + piece * (16 / OES);
                    const bool in = ch < y_chan && !(dbg & 2);
                    uint8_t *const dst = y_nhwc + (size_t)ch * OES;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int rr = 4 * i + sub, px = __shfl_sync(0xffffffffu, pixel, rr);
                        const uint4 v = *reinterpret_cast<const uint4 *>(staged + rr * 128 + ((piece ^ (rr & 7)) << 4));
                        if (in && px >= 0) *reinterpret_cast<uint4 *>(dst + (size_t)px * y_pix) = v;
                    }
                }
                if (y_nchw && pixel >= 0) {
                    // Darknet's layout: this lane's pixel, a store per filter plane; a warp's positions are runs of rows of the plane
                    float *dst = y_nchw + ((size_t)b * g.n + nl0) * plane + (size_t)y * g.w + x;
                    const int cols = min(min(CPC, bn - c0), g.n - nl0);
#pragma unroll
                    for (int j = 0; j < CPC; ++j)
                        if (j < cols) {
                            float v = __uint_as_float(r[j]);
                            if (BF16) v = __bfloat162float(__float2bfloat16_rn(v));   // what the channels-last copy holds
                            dst[(size_t)j * plane] = v;
                        }
                }
            }
            c -= chunks;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(smem_u32(&sh->acc_empty[acc]));
        }
        if (RES) cp_async_wait<0>();
    }

    // ---------------- teardown (also the abort path)
    if (*abort_flag) {   // loads that are still in flight land before shared memory is released
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000LL) { }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // a pair leaves together: every wait above is bounded, so both CTAs get here
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
    cluster_sync_all();
}

// ------------------------------------------------------------------ host side
size_t conv_tc_taps_fixed_smem(const TapsArgs &a) { return a.staged_bytes + 2 * sizeof(float) * (size_t)a.table + sizeof(TapsShared); }

size_t conv_tc_taps_smem(const TapsArgs &a)
{
    return tmem_smem((size_t)a.x_stages * a.x_slot + (size_t)a.w_stages * a.w_bytes + conv_tc_taps_fixed_smem(a), a.tmem_cols);
}

typedef void (*TapsKernel)(TapsArgs);
template <int ACT>
static TapsKernel taps_kernel_of(bool bf16, bool res, bool one)
{
    if (one) return bf16 ? conv_tc_taps_kernel<ACT, true, false, true> : conv_tc_taps_kernel<ACT, false, false, true>;
    return bf16 ? (res ? conv_tc_taps_kernel<ACT, true, true, false> : conv_tc_taps_kernel<ACT, true, false, false>)
                : (res ? conv_tc_taps_kernel<ACT, false, true, false> : conv_tc_taps_kernel<ACT, false, false, false>);
}

// Resident pairs of a kernel with `smem` bytes, kept for each kernel, size and device.
static int taps_resident(TapsKernel kern, size_t smem)
{
    static std::mutex lock;
    static std::map<std::tuple<TapsKernel, size_t, int>, int> known;
    int device = 0;
    cudaGetDevice(&device);
    const auto key = std::make_tuple(kern, smem, device);
    std::lock_guard<std::mutex> guard(lock);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (unsigned)(sm_count() / 2));
    cfg.blockDim = dim3(TAPS_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) { cudaGetLastError(); n = sm_count() / 2; }
    known[key] = n;
    return n;
}

int launch_conv_tc_taps(const TapsArgs &a, cudaStream_t s)
{
    const int act2 = a.ep.activation == DNB_LEAKY ? DNB_LINEAR : DNB_LEAKY;
    const bool yolo = a.ep.yolo_entries > 0;
    if ((a.ep.activation != DNB_LEAKY && a.ep.activation != DNB_LINEAR) || (a.ep.residual && (a.ep.activation2 != act2 || !a.y_nhwc || a.taps == 1)) ||
        (yolo && (a.ep.activation != DNB_LINEAR || a.ep.residual || a.y_nhwc || a.taps != 1)))
        DNB_FAIL(DNB_EINVAL, "conv_tc_taps: no variant of this epilogue");
    if (a.bn < 32 || a.bn > 256 || a.bn % 32 || a.x_stages < 2 || a.x_stages > TAPS_MAX_X || a.w_stages < 1 || a.w_stages > TAPS_MAX_W || a.rows > 1024)
        DNB_FAIL(DNB_EINVAL, "conv_tc_taps: plan out of range (bn %d, stages %d and %d, rows %d)", a.bn, a.x_stages, a.w_stages, a.rows);
    const TapsKernel kern = yolo ? (a.bf16 ? conv_tc_taps_kernel<TAPS_YOLO, true, false, true> : conv_tc_taps_kernel<TAPS_YOLO, false, false, true>)
                                 : a.ep.activation == DNB_LEAKY ? taps_kernel_of<DNB_LEAKY>(a.bf16 != 0, a.ep.residual != nullptr, a.taps == 1)
                                                                : taps_kernel_of<DNB_LINEAR>(a.bf16 != 0, a.ep.residual != nullptr, a.taps == 1);
    const size_t smem = conv_tc_taps_smem(a);
    DNB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, conv_tc_max_smem()));
    const int most = taps_resident(kern, smem);
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = 2; attrs[1].val.clusterDim.y = 1; attrs[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2u * (unsigned)(a.total_tiles < most ? a.total_tiles : most));
    cfg.blockDim = dim3(TAPS_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attrs;
    cfg.numAttrs = 2;
    DNB_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
    DNB_LAUNCH_CHECK("conv_tc_taps");
    return DNB_OK;
}

}  // namespace dnb
