// First-layer convolution on the sm_100a tensor cores: 3x3 filters over at most 3 input channels (the RGB stems of YOLOv3,
// YOLOv3-tiny and Darknet-19), 5x5 and 7x7 filters over RGB (ResNet's 7x7 stride-2 first layer).
//
// No im2col row is ever written.  A tile's patch of the image lies in shared memory with one 16-byte cell per pixel, its
// channels as TF32 values followed by zeros, and 16 bytes x 8 rows is exactly the core matrix of an operand without swizzle: the cells
// of 8 neighbouring pixels are the core matrix of one tap, and the next tap's is the same cells one pixel on.  So tcgen05.mma
// reads its rows straight from the patch: K = 8 TF32 values are two taps, the distance between their cells is the
// descriptor's leading byte offset, the pitch of the patch its stride byte offset.
//  * a tile is 8 x 16 output pixels of one image (16 groups of 8 rows of the MMA, at a constant distance).  For stride 2 the
//    patch keeps the even columns of a row first and the odd ones behind them, so that neighbouring pixels of a tap stay
//    neighbours.  The taps, an odd number, are paired in the order of their cells; the last but one takes part
//    in two pairs with half its weight each (exact), so that nothing outside the receptive field meets even a zero weight.
//  * builder warps fetch the next patch into registers a tile ahead and write it, rounded once, zero outside the
//    image (the padding), as one 16-byte cell per pixel; one of them issues the MMAs.
//  * warps 0..3 drain the accumulator of the tile before (two accumulators in TMEM): folded batchnorm / bias, activation,
//    staged rows, one TMA store per 128 bytes of row and warp, clipped by the unit at the output's edges.
// What bounds it: 16 x 608 x 608, 3x3, 32 filters takes 205 us where its bytes take 126; 155 without the stores, 156 without the
// fetches, 208 without the MMAs, and the same with 3 to 6 CTAs an SM: the two streams of requests, not the arithmetic.
// ResNet's 7x7 at 64 x 224 x 224 takes 97 us (37 for its bytes); building swizzled im2col rows from the patch by
// threads (147 shared-memory loads a pixel) took 136 us, fetching every tap from global memory 260.
//
// Every mbarrier wait is bounded; on expiry the CTA records a code in the status word and leaves.
//
// Replaces forward_convolutional_layer_gpu (src/convolutional_kernels.cu:73-135 of the reference) for size 3, groups 1,
// c <= 3 or size 5 or 7, c = 3, with n a multiple of 16 up to 64 and channels-last output; weights in the im2col order
// c*size*size + kh*size + kw as in src/im2col.c:15-39.
#include "common.h"
#include "conv.h"
#include "device_utils.cuh"
#include "tc_ptx.cuh"

namespace dnb {

constexpr int ST_EPI = 128;
constexpr int ST_TW = 8, ST_TH = 16;    // output pixels of a tile
// Builder threads, and CTAs that share an SM: enough of both that the fetches of one CTA and the epilogues of the others overlap,
// within the register file.  A 3x3 stride-1 patch is 180 pixels, the others 240 to 777.
__host__ __device__ constexpr int stem_build(int size, int stride) { return size == 3 && stride == 1 ? 64 : 128; }
__host__ __device__ constexpr int stem_threads(int size, int stride) { return ST_EPI + stem_build(size, stride); }
__host__ __device__ constexpr int stem_ctas(int size) { return size == 3 ? 4 : 2; }

struct StemShared {
    uint64_t mma_done[2];   // the MMAs that read patch i have retired
    uint64_t acc_full[2];
    uint64_t acc_empty[2];
    uint32_t tmem_base;
    int abort_flag;
};

enum { ST_WAIT_ROWS = 101, ST_WAIT_ACC_EMPTY = 103, ST_WAIT_ACC = 104, ST_BAD_SMEM_BASE = 106 };
enum { ST_ACT_GENERIC = -1 };

template <int ACT>
__device__ __forceinline__ float stem_act(float x, int runtime_act)
{
    if (ACT == DNB_LINEAR) return x;
    if (ACT == DNB_LEAKY) return fmaxf(x, 0.1f * x);
    return activate_call(x, runtime_act);
}

// The builders meet, and learn whether any of them has given up: they leave their loop together.
template <int THREADS>
__device__ __forceinline__ bool builders_meet(bool failed)
{
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred p, 1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(any) : "r"((uint32_t)failed), "n"(THREADS) : "memory");
    return any != 0;
}

// Position of a CTA's current tile, advanced by the grid's size with carries instead of divisions.
struct StemTile {
    int tx, ty, b;
    __device__ __forceinline__ StemTile(int tile, int tiles_w, int tiles_h) : tx(tile % tiles_w), ty(tile / tiles_w % tiles_h), b(tile / tiles_w / tiles_h) {}
    __device__ __forceinline__ void advance(const StemTile &by, int tiles_w, int tiles_h)
    {
        tx += by.tx; ty += by.ty; b += by.b;
        if (tx >= tiles_w) { tx -= tiles_w; ++ty; }
        if (ty >= tiles_h) { ty -= tiles_h; ++b; }
    }
};

// The patch of one tile, and the taps in the order of their cells.
template <int KS, int S>
struct StemPatch {
    static constexpr int W = (ST_TW - 1) * S + KS, H = (ST_TH - 1) * S + KS;
    static constexpr int EVEN = (W + 1) / 2, HALF = (EVEN + 3) / 8 * 8 + 4;   // stride 2: first odd column's cell, 4 modulo 8: 8 columns in 8 bank groups
    static constexpr int PITCH = S == 1 ? W : HALF + W / 2;
    static constexpr int CELLS = H * PITCH, BUILD = stem_build(KS, S), PER_THREAD = (W * H + BUILD - 1) / BUILD;
    static constexpr int TAPS = KS * KS, PAIRS = (TAPS + 1) / 2;
    static_assert(HALF >= EVEN && TAPS % 2 == 1 && CELLS < 32768 && W < 256 && H < 256, "layout of the patch");
    static __host__ __device__ constexpr int column(int x) { return S == 1 ? x : (x & 1) * HALF + (x >> 1); }
    // tap `slot` (0 or 1) of pair p; the last pair starts one tap back
    static __host__ __device__ constexpr int tap(int p, int slot) { return 2 * p + slot - (p == PAIRS - 1 ? 1 : 0); }
    static __host__ __device__ constexpr int tap_kh(int i) { return i / KS; }
    static __host__ __device__ constexpr int tap_kw(int i) { return S == 1 ? i % KS : (i % KS < (KS + 1) / 2 ? 2 * (i % KS) : 2 * (i % KS - (KS + 1) / 2) + 1); }
    static __host__ __device__ constexpr int cell(int i) { return tap_kh(i) * PITCH + column(tap_kw(i)); }
};

// Descriptor of a K-major operand without swizzle: 8-row x 16-byte core matrices, `lead` bytes apart along K, `stride` bytes
// apart along the rows.
__device__ __forceinline__ uint64_t plain_smem_desc(uint32_t addr, uint32_t lead, uint32_t stride)
{
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(lead >> 4) << 16 | (uint64_t)(stride >> 4) << 32 | (uint64_t)1 << 46;
}

// KS: filter size; S: stride; ACT: activation folded at compile time or ST_ACT_GENERIC; OUT_BF16: storage type of the
// channels-last output.
// POOL: the output is that of the 2x2 maxpool with stride 2 after the layer.  A warp's 32 pixels are four rows of eight, two rows of four
// windows: it stages them as ever, takes the largest of each four staged pieces and stores eight pixels.
template <int KS, int S, int ACT, bool OUT_BF16, bool POOL>
__global__ void __launch_bounds__(stem_threads(KS, S), stem_ctas(KS))
conv_stem_tc_kernel(const __grid_constant__ StemTcArgs a)
{
    using P = StemPatch<KS, S>;
    constexpr int ST_THREADS = stem_threads(KS, S), BUILD = P::BUILD;
    extern __shared__ __align__(1024) uint8_t smem[];
    if (smem_u32(smem) & 1023u) {   // the swizzle pattern repeats every 1024 bytes
        if (threadIdx.x == 0) atomicCAS(a.status, 0, ST_BAD_SMEM_BASE);
        return;
    }
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int n_pad = a.n_pad;
    const uint32_t seg_bytes = (uint32_t)a.seg_bytes, segs = (uint32_t)a.segs, out_bytes = segs * 128u * seg_bytes;
    uint8_t *const sO = smem;                                        // staged output rows
    uint8_t *const sB = sO + out_bytes;                              // PAIRS blocks of n_pad filters x 2 taps x 4 channels
    float4 *const patch0 = reinterpret_cast<float4 *>(sB + P::PAIRS * n_pad * 32);   // two patches
    float *const s_scale = reinterpret_cast<float *>(patch0 + 2 * P::CELLS), *const s_shift = s_scale + n_pad;
    StemShared *const sh = reinterpret_cast<StemShared *>(s_shift + n_pad);
    volatile int *abort_flag = &sh->abort_flag;
    const ConvGeom g = a.g;

    // filters, rounded to TF32: block p holds the core matrices of 8 filters x one tap, the pair's two taps side by side; zero beyond
    // the layer's channels and filters
    for (int i = tid; i < P::PAIRS * 2 * n_pad; i += ST_THREADS) {
        const int p = i / (2 * n_pad), r = i - p * 2 * n_pad, slot = r / n_pad, f = r - slot * n_pad;
        const int tap = P::tap(p, slot), k = P::tap_kh(tap) * KS + P::tap_kw(tap);
        const float part = tap == P::TAPS - 2 ? 0.5f : 1.f;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 3; ++c)
            if (c < g.c && f < g.n) v[c] = part * round_tf32(__ldg(a.w + (size_t)(c * P::TAPS + k) * a.npg_pad + f));
        *reinterpret_cast<float4 *>(sB + p * n_pad * 32 + (f >> 3) * 256 + slot * 128 + (f & 7) * 16) = make_float4(v[0], v[1], v[2], v[3]);
    }
    for (int i = tid; i < n_pad; i += ST_THREADS) {
        s_scale[i] = i < g.n ? __ldg(a.ep.scale + i) : 0.f;
        s_shift[i] = i < g.n ? __ldg(a.ep.shift + i) : 0.f;
    }
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&sh->mma_done[i]), 1);
            mbar_init(smem_u32(&sh->acc_full[i]), 1);
            mbar_init(smem_u32(&sh->acc_empty[i]), 4);   // one arrival per epilogue warp
        }
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem_cols = (uint32_t)a.tmem_cols, acc_stride = tmem_cols / 2;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();   // the filter rows are read by the tensor cores
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = sh->tmem_base;
    grid_dependency_wait();   // up to here only the layer's own parameters were read
    launch_dependents();

    // register copies: every asm statement below is a compiler memory barrier
    const int tiles = a.tiles, tiles_w = a.tiles_w, tiles_h = a.tiles_h;
    int *const status = a.status;
    const long long wait_limit = a.wait_limit;
    const StemTile step(gridDim.x, tiles_w, tiles_h);
    bool ok = true;
    int it = 0;
    if (warp >= 4) {
        // ---------------- builders
        const int bt = tid - ST_EPI;
        const float *const x = a.x;
        const long long xs_b = a.xs_b, xs_c = a.xs_c;
        const int xs_h = (int)a.xs_h, xs_w = (int)a.xs_w, pad = g.pad, img_h = g.h, img_w = g.w;
        const bool two = g.c > 1, three = g.c > 2;
        // the pixels this thread carries: where they come from (from the patch's corner) and which cell they go to
        float v[P::PER_THREAD][3];
        int from[P::PER_THREAD], yx[P::PER_THREAD];
#pragma unroll
        for (int i = 0; i < P::PER_THREAD; ++i) {
            const int e = bt + i * BUILD, py = e / P::W, px = e - py * P::W;
            from[i] = py * xs_h + px * xs_w;
            yx[i] = e < P::W * P::H ? (py << 8) | px | ((py * P::PITCH + P::column(px)) << 16) : -1;
        }
        StemTile at(blockIdx.x, tiles_w, tiles_h);        // the tile whose patch is fetched next
        StemTile got = at;                                // ... and the one whose patch was
        auto fetch = [&]() {
            const int ix0 = at.tx * ST_TW * S - pad, iy0 = at.ty * ST_TH * S - pad;
            const float *xp = x + (size_t)at.b * xs_b + (long long)iy0 * xs_h + (long long)ix0 * xs_w;   // dereferenced only inside the image
#pragma unroll
            for (int i = 0; i < P::PER_THREAD; ++i) {
                const int iy = iy0 + ((yx[i] >> 8) & 255), ix = ix0 + (yx[i] & 255);
                const bool in = yx[i] >= 0 && (unsigned)iy < (unsigned)img_h && (unsigned)ix < (unsigned)img_w;
                const float *p = xp + from[i];
                v[i][0] = in ? __ldg(p) : 0.f;
                v[i][1] = in && two ? __ldg(p + xs_c) : 0.f;
                v[i][2] = in && three ? __ldg(p + 2 * xs_c) : 0.f;
            }
            got = at;
            at.advance(step, tiles_w, tiles_h);
        };
        float *const keep = POOL ? a.keep : nullptr;
        const uint32_t idesc = mma_idesc<MMA_TF32>(128u, (uint32_t)n_pad);
        const uint64_t da0 = plain_smem_desc(smem_u32(patch0), 0, S * P::PITCH * 16), db0 = plain_smem_desc(smem_u32(sB), 128, 256);
        const uint64_t b_step = (uint64_t)(n_pad * 2);
        const uint32_t done0 = smem_u32(&sh->mma_done[0]), full0 = smem_u32(&sh->acc_full[0]), empty0 = smem_u32(&sh->acc_empty[0]);
        if ((int)blockIdx.x < tiles) fetch();
        bool stop = false;
        for (int tile = blockIdx.x; tile < tiles && !stop; tile += gridDim.x, ++it) {
            const int buf = it & 1, use = it >> 1;
            if (use > 0 && !mbar_wait(done0 + 8 * buf, (uint32_t)(use - 1) & 1u, abort_flag, status, ST_WAIT_ROWS, 0, wait_limit)) ok = false;
            float4 *const patch = patch0 + buf * P::CELLS;
#pragma unroll
            for (int i = 0; i < P::PER_THREAD; ++i)
                if (yx[i] >= 0) patch[yx[i] >> 16] = make_float4(round_tf32(v[i][0]), round_tf32(v[i][1]), round_tf32(v[i][2]), 0.f);
            fence_async_smem();   // cells visible to the tensor cores
            if (POOL && keep) {   // a copy of the images: the patch's inner pixels (stride 1, padding 1)
#pragma unroll
                for (int i = 0; i < P::PER_THREAD; ++i) {
                    const int py = (yx[i] >> 8) & 255, px = yx[i] & 255, iy = got.ty * ST_TH - pad + py, ix = got.tx * ST_TW - pad + px;
                    if (yx[i] < 0 || px < pad || px >= pad + ST_TW || py < pad || py >= pad + ST_TH || iy >= img_h || ix >= img_w) continue;
                    float *p = keep + (size_t)got.b * xs_b + (long long)iy * xs_h + ix;
                    p[0] = v[i][0];
                    if (two) p[xs_c] = v[i][1];
                    if (three) p[2 * xs_c] = v[i][2];
                }
            }
            if (tile + (int)gridDim.x < tiles) fetch();   // a whole tile's time to arrive
            stop = builders_meet<BUILD>(!ok);
            if (warp == 4 && !stop) {
                if (!mbar_wait_warp(empty0 + 8 * buf, (uint32_t)(use & 1) ^ 1u, abort_flag, status, ST_WAIT_ACC_EMPTY, wait_limit)) ok = false;
                if (ok && elect_one()) {
                    tc_fence_after();
                    const uint32_t d = tmem_base + buf * acc_stride;
                    const uint64_t da = da0 + (uint64_t)(buf * P::CELLS);   // addresses in the descriptor count cells
#pragma unroll
                    for (int p = 0; p < P::PAIRS; ++p) {
                        const int c0 = P::cell(P::tap(p, 0)), c1 = P::cell(P::tap(p, 1));
                        umma<MMA_TF32>(d, da + (uint64_t)c0 + ((uint64_t)(c1 - c0) << 16), db0 + p * b_step, idesc, p != 0 ? 1u : 0u);
                    }
                    umma_commit(done0 + 8 * buf);
                    umma_commit(full0 + 8 * buf);
                }
                __syncwarp();
            }
        }
    } else {
        // ---------------- epilogue: warp w owns TMEM lanes and tile pixels 32*w .. +31 (four rows of 8)
        const int runtime_act = a.ep.activation, do_round = a.ep.round_tf32;
        const CUtensorMap *ymap = &a.tmy;
        const uint32_t q_mask = seg_bytes / 16 - 1;
        const uint32_t m = (uint32_t)tid, q_xor = (seg_bytes == 128 ? m : (seg_bytes == 64 ? m >> 1 : m >> 2)) & q_mask;
        const uint32_t full0 = smem_u32(&sh->acc_full[0]), empty0 = smem_u32(&sh->acc_empty[0]);
        const int seg_chan = (int)seg_bytes / (OUT_BF16 ? 2 : 4);
        StemTile at(blockIdx.x, tiles_w, tiles_h);
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {
            const int acc = it & 1;
            if (!mbar_wait(full0 + 8 * acc, (uint32_t)((it >> 1) & 1), abort_flag, status, ST_WAIT_ACC, 0, wait_limit)) break;
            tc_fence_after();
            const uint32_t t_row = tmem_base + ((uint32_t)(warp * 32) << 16) + acc * acc_stride;
            if (lane == 0) tma_store_wait_read0();   // this warp's last store has read its rows
            __syncwarp();
#pragma unroll 1
            for (int c0 = 0; c0 < n_pad; c0 += 16) {
                uint32_t r[16];
                tmem_ld16(t_row + c0, r);
                tmem_ld_wait();
                float o[16];
                const float4 *sc4 = reinterpret_cast<const float4 *>(s_scale + c0);
                const float4 *sf4 = reinterpret_cast<const float4 *>(s_shift + c0);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 sc = sc4[q], sf = sf4[q];
                    const float scv[4] = {sc.x, sc.y, sc.z, sc.w}, sfv[4] = {sf.x, sf.y, sf.z, sf.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int j = 4 * q + e;
                        float f = stem_act<ACT>(fmaf(__uint_as_float(r[j]), scv[e], sfv[e]), runtime_act);
                        if (do_round) f = round_tf32(f);
                        // beyond the layer's filters scale and shift are zero: only an activation with f(0) != 0 needs the mask
                        o[j] = (ACT == ST_ACT_GENERIC && c0 + j >= g.n) ? 0.f : f;
                    }
                }
                // these 16 columns inside the pixel's staged row, which is cut into segments of at most 128 bytes
                const uint32_t byte0 = (uint32_t)c0 * (OUT_BF16 ? 2u : 4u), seg = byte0 / seg_bytes, q0 = (byte0 - seg * seg_bytes) >> 4;
                uint8_t *srow = sO + seg * 128u * seg_bytes + m * seg_bytes;
                if (!OUT_BF16) {
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        *reinterpret_cast<float4 *>(srow + (((q0 + q) ^ q_xor) << 4)) = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
                } else {
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        uint32_t pk[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            __nv_bfloat162 h = __floats2bfloat162_rn(o[8 * q + 2 * e], o[8 * q + 2 * e + 1]);
                            pk[e] = *reinterpret_cast<uint32_t *>(&h);
                        }
                        *reinterpret_cast<uint4 *>(srow + (((q0 + q) ^ q_xor) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                    }
                }
            }
            tc_fence_before();
            if (POOL) {
                // one segment; lane's piece of pooled pixel (rows of 32, 64 or 128 bytes: 16, 32 or 64 pieces)
                __syncwarp();
                uint8_t *const mine = sO + (uint32_t)(warp * 32) * seg_bytes;
                const uint32_t pieces = seg_bytes >> 4;
                auto swizzled = [&](uint32_t row, uint32_t q) { return row * seg_bytes + ((q ^ ((seg_bytes == 128 ? row : seg_bytes == 64 ? row >> 1 : row >> 2) & q_mask)) << 4); };
                uint4 best[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t e = lane + 32 * h, pp = e / pieces, q = e - pp * pieces;
                    if (e >= 8 * pieces) continue;
                    const uint32_t top = (pp >> 2) * 16 + (pp & 3) * 2;
                    uint4 v[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const uint4 *>(mine + swizzled(top + (i & 1) + (i >> 1) * 8, q));
                    best[h] = largest_of_four<OUT_BF16>(v);
                }
                __syncwarp();
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t e = lane + 32 * h, pp = e / pieces, q = e - pp * pieces;
                    if (e < 8 * pieces) *reinterpret_cast<uint4 *>(mine + swizzled(pp, q)) = best[h];
                }
            }
            fence_async_smem();
            __syncwarp();
            if (POOL && lane == 0) {
                mbar_arrive(empty0 + 8 * acc);
                if (at.ty * ST_TH + 4 * warp < g.out_h) tma_store_4d(ymap, smem_u32(sO) + (uint32_t)(warp * 32) * seg_bytes, 0, at.tx * (ST_TW / 2), at.ty * (ST_TH / 2) + 2 * warp, at.b);
                tma_store_commit();
            } else if (lane == 0) {
                mbar_arrive(empty0 + 8 * acc);
                for (uint32_t sg = 0; sg < segs && at.ty * ST_TH + 4 * warp < g.out_h; ++sg)   // (rows below the map: nothing to store)
                    tma_store_4d(ymap, smem_u32(sO) + sg * 128u * seg_bytes + (uint32_t)(warp * 32) * seg_bytes, (int)sg * seg_chan, at.tx * ST_TW, at.ty * ST_TH + 4 * warp, at.b);
                tma_store_commit();
            }
            at.advance(step, tiles_w, tiles_h);
        }
        if (lane == 0) tma_store_wait_all();
    }

    // ---------------- teardown (also the abort path)
    if (*abort_flag) {   // give MMAs that may still read shared memory time to retire
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000LL) { }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
}

// ------------------------------------------------------------------ host side
bool conv_stem_tc_covers(const ConvGeom &g)
{
    const bool narrow = g.size == 3 && g.c >= 1 && g.c <= 3, wide = g.c == 3 && (g.size == 5 || g.size == 7);
    return (narrow || wide) && g.groups == 1 && g.n % 16 == 0 && g.n <= 64 && g.stride >= 1 && g.stride <= 2;
}

// The maxpool after it in the same launch: 3x3 layers with stride 1 and padding 1, whole windows, pixels of at most 128 bytes, the leaky activation.
bool conv_stem_pool_covers(const ConvGeom &g, int y_dtype, int activation)
{
    return conv_stem_tc_covers(g) && g.size == 3 && g.stride == 1 && g.pad == 1 && g.out_h % 2 == 0 && g.out_w % 2 == 0 && g.n * (y_dtype == DNB_BF16 ? 2 : 4) <= 128 && activation == DNB_LEAKY;
}

template <int KS, int S, int ACT, bool OBF, bool POOL = false>
static int launch_stem(const StemTcArgs &a, cudaStream_t s)
{
    using P = StemPatch<KS, S>;
    auto kern = conv_stem_tc_kernel<KS, S, ACT, OBF, POOL>;
    size_t smem = (size_t)a.segs * 128 * a.seg_bytes + (size_t)P::PAIRS * a.n_pad * 32 + 2 * sizeof(float4) * P::CELLS + 2 * sizeof(float) * a.n_pad + sizeof(StemShared) + 16;
    smem = tmem_smem(smem, a.tmem_cols);
    const size_t sm_bytes = 228 * 1024, reserved = 1024;   // per SM, and per resident CTA
    DNB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // all of the SM's configurable memory as shared memory, so that several CTAs are resident
    DNB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    int per_sm = (int)(sm_bytes / (smem + reserved));
    if (per_sm > stem_ctas(KS)) per_sm = stem_ctas(KS);   // the kernel's register budget (__launch_bounds__)
    if (per_sm < 1) DNB_FAIL(DNB_ECUDA, "first-layer kernel: %zu bytes of shared memory do not fit", smem);
    long long grid = (long long)sm_count() * per_sm;
    if (grid > a.tiles) grid = a.tiles;
    DNB_CUDA(launch_overlapped(kern, dim3((unsigned)grid), dim3(stem_threads(KS, S)), smem, s, a));
    DNB_LAUNCH_CHECK("conv_stem_tc");
    return DNB_OK;
}

template <int KS, int S, bool OBF>
static int launch_act(const StemTcArgs &a, cudaStream_t s)
{
    if constexpr (KS == 3 && S == 1)
        if (a.pool) return launch_stem<KS, S, DNB_LEAKY, OBF, true>(a, s);
    if (a.ep.activation == DNB_LEAKY) return launch_stem<KS, S, DNB_LEAKY, OBF>(a, s);
    if (a.ep.activation == DNB_LINEAR) return launch_stem<KS, S, DNB_LINEAR, OBF>(a, s);
    return launch_stem<KS, S, ST_ACT_GENERIC, OBF>(a, s);
}

template <int KS>
static int launch_size(const StemTcArgs &a, cudaStream_t s)
{
    const bool obf = a.y_dtype == DNB_BF16;
    if (a.g.stride == 1) return obf ? launch_act<KS, 1, true>(a, s) : launch_act<KS, 1, false>(a, s);
    return obf ? launch_act<KS, 2, true>(a, s) : launch_act<KS, 2, false>(a, s);
}

int launch_conv_stem_tc(StemTcArgs a, cudaStream_t s)
{
    const ConvGeom &g = a.g;
    if (!conv_stem_tc_covers(g) || a.y_cpitch != g.n) DNB_FAIL(DNB_EUNSUPPORTED, "first-layer kernel: geometry outside its coverage");
    if (a.xs_c >= (1LL << 31) / 4 || a.xs_h >= (1LL << 31) / 64) DNB_FAIL(DNB_EUNSUPPORTED, "first-layer kernel: image too large for 32-bit offsets");
    a.tiles_w = (g.out_w + ST_TW - 1) / ST_TW;
    a.tiles_h = (g.out_h + ST_TH - 1) / ST_TH;
    const long long tiles = (long long)a.tiles_w * a.tiles_h * g.batch;
    if (tiles >= (1LL << 31) - 4096) DNB_FAIL(DNB_EUNSUPPORTED, "first-layer kernel: %lld tiles", tiles);
    a.tiles = (int)tiles;
    a.n_pad = round_up(g.n, 16);
    a.tmem_cols = 32;
    while (a.tmem_cols < 2 * a.n_pad) a.tmem_cols *= 2;
    // a pixel's output row in segments of 32, 64 or 128 bytes, the swizzle spans; the last one may reach past the row (the store is clipped)
    const int es = a.y_dtype == DNB_BF16 ? 2 : 4, rb = g.n * es;
    a.seg_bytes = rb > 64 ? 128 : (rb > 32 ? 64 : 32);
    a.segs = (rb + a.seg_bytes - 1) / a.seg_bytes;
    if (a.pool && (!conv_stem_pool_covers(g, a.y_dtype, a.ep.activation) || a.segs != 1)) DNB_FAIL(DNB_EINVAL, "first-layer kernel: no pooled variant of this layer");
    const int half = a.pool ? 2 : 1, yw = g.out_w / half, yh = g.out_h / half;
    const uint64_t dims[4] = {(uint64_t)g.n, (uint64_t)yw, (uint64_t)yh, (uint64_t)g.batch};
    const uint64_t strides[3] = {(uint64_t)rb, (uint64_t)rb * yw, (uint64_t)rb * yw * yh};
    const uint32_t box[4] = {(uint32_t)(a.seg_bytes / es), (uint32_t)ST_TW / half, 4u / half, 1u};   // a warp's four pixel rows
    DNB_TRY(encode_tensor_map(&a.tmy, es == 2 ? 1 : 0, 4, a.y, dims, strides, box, a.seg_bytes));
    if (g.size == 7) return launch_size<7>(a, s);
    if (g.size == 5) return launch_size<5>(a, s);
    return launch_size<3>(a, s);
}

}  // namespace dnb
