// First-layer convolution of binarised networks, on the tensor cores with its products in the im2col order: 3x3 filters over at
// most 3 input channels, 5x5 and 7x7 filters over RGB.
//
// The layers after this one take the sign of its results, so one that lies at zero to the last bit of its sum decides a whole +1 or -1.
// conv_stem_tc.cu adds the products tap by tap, two taps to an MMA; here they are added in the order of the reference's
// matrix row, c*size*size + kh*size + kw (src/im2col.c:15-39), eight to an MMA, and the same way at every batch size.
// (Measured on Darknet-19 with xnor layers, 128 x 224 x 224: the other order changes 500 of an image's 1.6 million first-layer values in
// their last TF32 bit, one sign of the batch, and with it one image's answer.)  A network with xnor layers chooses this file
// (keep_k_order); it costs such a network nothing at 3x3, 207 us against 207 at that size.
//
// The 128 threads of a CTA build the im2col rows of 128 consecutive output pixels themselves: a thread gathers the values of its pixel
// (zero outside the image, which is the padding), rounds them to TF32 and writes its row in the 128-byte-swizzled K-major
// layout tcgen05.mma reads.  One thread issues the K=8 MMAs against the filter matrix, which stays in shared memory.
//  * 3x3: K <= 27 is one row of 32 values.  A thread requests the inputs of tile i+1 before it runs the epilogue of tile i.  The
//    finished rows are staged where the tile's im2col rows were and leave through one TMA store per warp (plain 16-byte stores
//    where a row is not 32, 64 or 128 bytes).
//  * 5x5, 7x7: blocks of 32 values in two alternating buffers.
// Several CTAs share an SM and fill each other's waits.  Every mbarrier wait is bounded; on expiry the CTA records a code in the
// status word and leaves.
#include "common.h"
#include "conv.h"
#include "device_utils.cuh"
#include "tc_ptx.cuh"

namespace dnb {

constexpr int SR_THREADS = 128;
constexpr int SR_A_BYTES = 128 * 128;   // one im2col tile: 128 rows of 32 TF32 values

struct StemRowsShared {
    uint64_t acc_full;
    uint32_t tmem_base;
    int abort_flag;
};

enum { SR_WAIT_ACC = 104, SR_BAD_SMEM_BASE = 106 };
enum { SR_ACT_GENERIC = -1 };

template <int ACT>
__device__ __forceinline__ float rows_act(float x, int runtime_act)
{
    if (ACT == DNB_LEAKY) return fmaxf(x, 0.1f * x);
    return activate_call(x, runtime_act);
}

// C: input channels (1..3); ACT: activation folded at compile time or SR_ACT_GENERIC; OUT_BF16: storage
// type of the channels-last output.
template <int C, int ACT, bool OUT_BF16>
__global__ void __launch_bounds__(SR_THREADS, 5)
conv_stem_rows_kernel(const __grid_constant__ StemTcArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    if (smem_u32(smem) & 1023u) {   // the swizzle pattern repeats every 1024 bytes
        if (threadIdx.x == 0) atomicCAS(a.status, 0, SR_BAD_SMEM_BASE);
        return;
    }
    constexpr int K = C * 9;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int n_pad = a.n_pad;
    uint8_t *sA = smem;                           // 2 x 128 rows x 128 bytes
    uint8_t *sB = smem + 2 * SR_A_BYTES;          // n_pad rows x 128 bytes
    float *s_scale = reinterpret_cast<float *>(sB + (size_t)n_pad * 128);
    float *s_shift = s_scale + n_pad;
    StemRowsShared *sh = reinterpret_cast<StemRowsShared *>(s_shift + n_pad);
    volatile int *abort_flag = &sh->abort_flag;
    const ConvGeom g = a.g;

    // filters: row f holds w[f][0..K) rounded to TF32, zero beyond K and beyond the layer's filters
    for (int i = tid; i < n_pad * 8; i += SR_THREADS) {
        const int f = i >> 3, q = i & 7;
        uint32_t v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int k = 4 * q + e;
            v[e] = (k < K && f < g.n) ? __float_as_uint(round_tf32(__ldg(a.w + (size_t)k * a.npg_pad + f))) : 0u;
        }
        *reinterpret_cast<uint4 *>(sB + f * 128 + ((q ^ (f & 7)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
    }
    for (int i = tid; i < n_pad; i += SR_THREADS) {
        s_scale[i] = i < g.n ? __ldg(a.ep.scale + i) : 0.f;
        s_shift[i] = i < g.n ? __ldg(a.ep.shift + i) : 0.f;
    }
    if (tid == 0) {
        mbar_init(smem_u32(&sh->acc_full), 1);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem_cols = (uint32_t)a.tmem_cols;
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
    const float *const x = a.x;
    const long long xs_b = a.xs_b;
    const int xs_c = (int)a.xs_c, xs_h = (int)a.xs_h, xs_w = (int)a.xs_w;
    const int npix = a.npix, tiles = a.tiles, plane = g.out_h * g.out_w;
    const int runtime_act = a.ep.activation, do_round = a.ep.round_tf32;
    uint8_t *const y = reinterpret_cast<uint8_t *>(a.y);
    const size_t y_row_bytes = (size_t)a.y_cpitch * (OUT_BF16 ? 2 : 4);
    int *const status = a.status;
    const long long wait_limit = a.wait_limit;
    const uint32_t idesc = mma_idesc<MMA_TF32>(128u, (uint32_t)n_pad);
    const uint64_t db = make_smem_desc(smem_u32(sB), 128);
    const uint64_t da0 = make_smem_desc(smem_u32(sA), 128);
    const uint32_t bar0 = smem_u32(&sh->acc_full);
    const uint32_t row_off = (uint32_t)tid * 128u, sw = (uint32_t)(tid & 7);

    // staged output rows for the TMA store: row m of the tile at m * row_bytes, 16-byte pieces swizzled as the map says
    const bool tma = a.tma_store != 0;
    const uint32_t out_row_bytes = (uint32_t)a.y_cpitch * (OUT_BF16 ? 2u : 4u);
    const uint32_t q_xor = out_row_bytes == 128 ? (uint32_t)(tid & 7) : (out_row_bytes == 64 ? (uint32_t)((tid >> 1) & 3) : (uint32_t)((tid >> 2) & 1));
    const CUtensorMap *ymap = &a.tmy;
    const int lane = tid & 31;

    bool failed = false;
    int prev_tile = 0;
    int it = 0;
    for (int tile = blockIdx.x;; tile += gridDim.x, ++it) {
        const bool have = tile < tiles;   // uniform over the CTA
        const int buf = it & 1;
        // ---- this thread's 27 input values of the next tile: requested first, used after the epilogue below
        float v[K];
        if (have) {
            const int p = tile * SR_THREADS + tid;
            const bool valid = p < npix;
            const int b = p / plane, rem = p - b * plane;
            const int oy = rem / g.out_w, ox = rem - oy * g.out_w;
            const int iy0 = oy * g.stride - g.pad, ix0 = ox * g.stride - g.pad;
            // three row and three column validity flags and one base pointer: a tap costs one predicated load
            const bool rv0 = valid && (unsigned)iy0 < (unsigned)g.h, rv1 = valid && (unsigned)(iy0 + 1) < (unsigned)g.h,
                       rv2 = valid && (unsigned)(iy0 + 2) < (unsigned)g.h;
            const bool cv0 = (unsigned)ix0 < (unsigned)g.w, cv1 = (unsigned)(ix0 + 1) < (unsigned)g.w, cv2 = (unsigned)(ix0 + 2) < (unsigned)g.w;
            const float *xp = x + (size_t)b * xs_b + (long long)iy0 * xs_h + (long long)ix0 * xs_w;   // dereferenced only where valid
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int kh = 0; kh < 3; ++kh) {
                    const bool rv = kh == 0 ? rv0 : (kh == 1 ? rv1 : rv2);
                    const float *rp = xp + c * xs_c + kh * xs_h;
                    v[c * 9 + kh * 3 + 0] = (rv && cv0) ? __ldg(rp) : 0.f;
                    v[c * 9 + kh * 3 + 1] = (rv && cv1) ? __ldg(rp + xs_w) : 0.f;
                    v[c * 9 + kh * 3 + 2] = (rv && cv2) ? __ldg(rp + 2 * xs_w) : 0.f;
                }
        }
        if (it > 0) {
            // ---- epilogue of the previous tile (its MMAs were issued at the end of the previous iteration)
            const int pb = (it - 1) & 1;
            if (!mbar_wait(bar0, (uint32_t)((it - 1) & 1), abort_flag, status, SR_WAIT_ACC, 0, wait_limit)) {
                failed = true;
            } else {
                tc_fence_after();
                const uint32_t t_row = tmem_base + ((uint32_t)(warp * 32) << 16);
                const int prev_p = prev_tile * SR_THREADS + tid;
                const bool store = prev_p < npix;
                uint8_t *dst = y + (size_t)prev_p * y_row_bytes;
                // the finished rows go where the tile's im2col rows were: its MMAs have retired
                uint8_t *srow = sA + pb * SR_A_BYTES + (uint32_t)tid * out_row_bytes;
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
                            float t = rows_act<ACT>(fmaf(__uint_as_float(r[j]), scv[e], sfv[e]), runtime_act);
                            if (do_round) t = round_tf32(t);
                            // beyond the layer's filters scale and shift are zero: only an activation with f(0) != 0 needs the mask
                            o[j] = (ACT == SR_ACT_GENERIC && c0 + j >= g.n) ? 0.f : t;
                        }
                    }
                    if (!OUT_BF16) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const uint4 pk = make_uint4(__float_as_uint(o[4 * q]), __float_as_uint(o[4 * q + 1]), __float_as_uint(o[4 * q + 2]), __float_as_uint(o[4 * q + 3]));
                            if (tma) *reinterpret_cast<uint4 *>(srow + ((((uint32_t)(c0 >> 2) + q) ^ q_xor) << 4)) = pk;
                            else if (store) reinterpret_cast<uint4 *>(dst + (size_t)c0 * 4)[q] = pk;
                        }
                    } else {
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            uint4 pk;
                            __nv_bfloat162 h0 = __floats2bfloat162_rn(o[8 * q], o[8 * q + 1]);
                            __nv_bfloat162 h1 = __floats2bfloat162_rn(o[8 * q + 2], o[8 * q + 3]);
                            __nv_bfloat162 h2 = __floats2bfloat162_rn(o[8 * q + 4], o[8 * q + 5]);
                            __nv_bfloat162 h3 = __floats2bfloat162_rn(o[8 * q + 6], o[8 * q + 7]);
                            pk.x = *reinterpret_cast<uint32_t *>(&h0); pk.y = *reinterpret_cast<uint32_t *>(&h1);
                            pk.z = *reinterpret_cast<uint32_t *>(&h2); pk.w = *reinterpret_cast<uint32_t *>(&h3);
                            if (tma) *reinterpret_cast<uint4 *>(srow + ((((uint32_t)(c0 >> 3) + q) ^ q_xor) << 4)) = pk;
                            else if (store) reinterpret_cast<uint4 *>(dst + (size_t)c0 * 2)[q] = pk;
                        }
                    }
                }
                if (tma) {
                    // each warp stores its own 32 rows: no CTA-wide barrier between the rows and the store
                    fence_async_smem();
                    __syncwarp();
                    const int row0 = prev_tile * SR_THREADS + warp * 32;
                    if (lane == 0 && row0 < npix) {   // the TMA unit clips the box at the last pixel
                        tma_store_2d(ymap, smem_u32(sA + pb * SR_A_BYTES) + (uint32_t)(warp * 32) * out_row_bytes, 0, row0);
                        tma_store_commit();
                    }
                }
            }
        }
        if (have) {
            // ---- im2col row into A[buf]; the buffer last held the staged rows of two tiles ago
            if (tma) {
                if (lane == 0) tma_store_wait_read1();   // all but the store just issued have read their rows
                __syncwarp();
                // Staged rows narrower than an im2col row (fewer than 128 bytes of output per pixel) put this thread's
                // im2col row over rows that OTHER warps staged two tiles ago: every warp's stores must have read them.
                if (out_row_bytes < 128) __syncthreads();
            }
            uint8_t *row = sA + buf * SR_A_BYTES + row_off;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                uint32_t w4[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) w4[e] = 4 * q + e < K ? __float_as_uint(round_tf32(v[4 * q + e < K ? 4 * q + e : 0])) : 0u;
                *reinterpret_cast<uint4 *>(row + ((q ^ sw) << 4)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
            }
            fence_async_smem();   // rows visible to the tensor cores
        }
        tc_fence_before();        // this thread's TMEM loads precede the barrier, the next MMAs follow it
        if (__syncthreads_or(failed)) break;
        if (!have) break;
        if (tid == 0) {
            tc_fence_after();
            const uint64_t da = da0 + (uint64_t)(buf * (SR_A_BYTES >> 4));
            umma<MMA_TF32>(tmem_base, da, db, idesc, 0u);
            umma<MMA_TF32>(tmem_base, da + 2, db + 2, idesc, 1u);
            umma<MMA_TF32>(tmem_base, da + 4, db + 4, idesc, 1u);
            umma<MMA_TF32>(tmem_base, da + 6, db + 6, idesc, 1u);
            umma_commit(bar0);
        }
        __syncwarp();
        prev_tile = tile;
    }
    if (tma && lane == 0) tma_store_wait_all();

    // ---- teardown (also the abort path)
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

// ------------------------------------------------------------------ with the 2x2 maxpool after it (3x3, stride 1, 32 filters, f32)
// The output is that of the maxpool with stride 2 after the layer, and optionally its signs, the next xnor layer's operand.  Same rows, same order of the
// products.  What bounded the form before (27 predicated loads and roundings a pixel, every value finished, staged and read back; 62 % of the issue slots) was
// instructions, so
//  * a tile is 16 x 8 windows of an image.  Its patch is loaded and rounded once, 18 values a thread, into shared memory, one tile ahead; a thread builds the
//    rows of its window's four pixels from pairs of values, two pixels at a time;
//  * the pixels of the same place in their windows are one MMA's 128 rows: a thread finds the four sums of its window in four accumulators, and what it
//    scales, activates and rounds is the largest, none of which changes which one that is.  Sums of filters with a negative scale change sign first.  A
//    warp that meets an infinity or NaN finishes all four, as the layer alone would, and then compares.
// 128 x 224 x 224: 250 -> 144 us.  Bytes: 51; the sixteen MMAs a tile, 77 clocks each: 55; shared memory (rows written and read by the MMAs, patch): some 80.
// (The upper pixels' sums compared while the lower ones are multiplied: the same time.)
constexpr int SRP_TW = 16, SRP_TH = 8, SRP_PITCH = 2 * SRP_TW + 2, SRP_ROWS = 2 * SRP_TH + 2;

struct StemRowsPoolShared {
    uint64_t done[2];       // the MMAs over the windows' upper, lower pixels have retired
    uint32_t tmem_base;
    int abort_flag;
};

// The largest of four sums, NaN if one is.
__device__ __forceinline__ float largest_or_nan(uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    float m;
    asm("{\n\t.reg .f32 t;\n\tmax.NaN.f32 t, %1, %2, %3;\n\tmax.NaN.f32 %0, t, %4;\n\t}"
        : "=f"(m) : "f"(__uint_as_float(a)), "f"(__uint_as_float(b)), "f"(__uint_as_float(c)), "f"(__uint_as_float(d)));
    return m;
}

template <int C>
__global__ void __launch_bounds__(SR_THREADS, 4)
conv_stem_rows_pool_kernel(const __grid_constant__ StemTcArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0) atomicCAS(a.status, 0, SR_BAD_SMEM_BASE);
        return;
    }
    constexpr int K = C * 9, PLANE = SRP_PITCH * SRP_ROWS, N = 32, PIECES = (K + 3) / 4;
    constexpr int LINES = SR_THREADS / SRP_PITCH, STEPS = SRP_ROWS / LINES;   // patch rows loaded at once, and how often, of a plane
    static_assert(SRP_ROWS % LINES == 0, "whole planes");
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint8_t *const sA = smem;                            // 2 x 128 rows x 128 bytes: a window's left pixel, its right one
    uint8_t *const sB = smem + 2 * SR_A_BYTES;           // 32 rows x 128 bytes
    float *const s_scale = reinterpret_cast<float *>(sB + N * 128), *const s_shift = s_scale + N;
    float *const patch = s_shift + N;                    // two patches of C planes of 18 x 34
    StemRowsPoolShared *const sh = reinterpret_cast<StemRowsPoolShared *>(patch + 2 * C * PLANE);
    volatile int *const abort_flag = &sh->abort_flag;
    const ConvGeom g = a.g;

    // filters as above; zeros where an im2col row has no value
    for (int i = tid; i < N * 8; i += SR_THREADS) {
        const int f = i >> 3, q = i & 7;
        uint32_t v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int k = 4 * q + e;
            v[e] = k < K ? __float_as_uint(round_tf32(__ldg(a.w + (size_t)k * a.npg_pad + f))) : 0u;
        }
        *reinterpret_cast<uint4 *>(sB + f * 128 + ((q ^ (f & 7)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
    }
    for (int i = tid; i < 2 * SR_A_BYTES / 16; i += SR_THREADS) reinterpret_cast<uint4 *>(sA)[i] = make_uint4(0u, 0u, 0u, 0u);
    bool below_zero = false, odd_scale = false;
    if (tid < N) {
        const float sc = __ldg(a.ep.scale + tid);
        s_scale[tid] = fabsf(sc);
        s_shift[tid] = __ldg(a.ep.shift + tid);
        below_zero = sc < 0.f;
        odd_scale = !(fabsf(sc) > 0.f && fabsf(sc) < INFINITY);
    }
    if (tid == 0) {
        mbar_init(smem_u32(&sh->done[0]), 1);
        mbar_init(smem_u32(&sh->done[1]), 1);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        const uint32_t bits = __ballot_sync(0xffffffffu, below_zero);
        if (tid == 0) *reinterpret_cast<uint32_t *>(patch) = bits;   // for the other warps, until the first patch
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"((uint32_t)a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    tc_fence_before();
    const bool plain = !__syncthreads_or(odd_scale);
    tc_fence_after();
    const uint32_t tmem_base = sh->tmem_base, negative = *reinterpret_cast<uint32_t *>(patch);
    __syncthreads();
    grid_dependency_wait();   // up to here only the layer's own parameters were read
    launch_dependents();

    const float *const x = a.x;
    float *const keep = a.keep;
    const long long xs_b = a.xs_b;
    const int xs_c = (int)a.xs_c, xs_h = (int)a.xs_h, xs_w = (int)a.xs_w;
    const int tiles = a.tiles, tiles_w = a.tiles_w, tiles_wh = a.tiles_w * a.tiles_h, do_round = a.ep.round_tf32;
    int8_t *const signs = a.signs;
    int *const status = a.status;
    const long long wait_limit = a.wait_limit;
    const uint32_t idesc = mma_idesc<MMA_TF32>(128u, (uint32_t)N);
    const uint64_t db = make_smem_desc(smem_u32(sB), 128), da0 = make_smem_desc(smem_u32(sA), 128);
    const uint32_t done0 = smem_u32(&sh->done[0]);

    const int wx = tid & (SRP_TW - 1), wy = tid / SRP_TW, sw = tid & 7;
    const float *const from = patch + 2 * wy * SRP_PITCH + 2 * wx;
    uint8_t *const row = sA + tid * 128;

    // A thread loads one column of every third row of the patch: value (c, k) is row line + LINES * k of plane c.
    const bool loads = tid < LINES * SRP_PITCH;
    const int line = tid / SRP_PITCH, column = tid - line * SRP_PITCH;
    const bool own_column = column >= 1 && column <= 2 * SRP_TW;
    const long long step_h = (long long)LINES * xs_h;
    float v[C][STEPS];
    const float *base = x;             // of the tile whose values are in v: may lie before the image, dereferenced only inside
    int next_b, next_y, next_x;        // its image and first window
    bool in_column;
    auto fetch = [&](int tile) {
        const int b = tile / tiles_wh, r = tile - b * tiles_wh, ty = r / tiles_w;
        next_b = b; next_y = ty * SRP_TH; next_x = (r - ty * tiles_w) * SRP_TW;
        const int yy = 2 * next_y - 1 + line, xx = 2 * next_x - 1 + column;
        base = x + b * xs_b + (long long)yy * xs_h + (long long)xx * xs_w;
        in_column = loads && (unsigned)xx < (unsigned)g.w;
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int k = 0; k < STEPS; ++k) v[c][k] = in_column && (unsigned)(yy + LINES * k) < (unsigned)g.h ? __ldg(base + c * xs_c + k * step_h) : 0.f;
    };
    // rows of the window's two pixels at `from`
    auto build = [&](const float *src) {
        float w[2][PIECES * 4];
#pragma unroll
        for (int k = K; k < PIECES * 4; ++k) w[0][k] = w[1][k] = 0.f;
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int kh = 0; kh < 3; ++kh) {
                const float2 p0 = *reinterpret_cast<const float2 *>(src + c * PLANE + kh * SRP_PITCH), p1 = *reinterpret_cast<const float2 *>(src + c * PLANE + kh * SRP_PITCH + 2);
                const int k = c * 9 + kh * 3;
                w[0][k] = p0.x; w[0][k + 1] = p0.y; w[0][k + 2] = p1.x;
                w[1][k] = p0.y; w[1][k + 1] = p1.x; w[1][k + 2] = p1.y;
            }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < PIECES; ++q)
                *reinterpret_cast<float4 *>(row + h * SR_A_BYTES + ((q ^ sw) << 4)) = make_float4(w[h][4 * q], w[h][4 * q + 1], w[h][4 * q + 2], w[h][4 * q + 3]);
        fence_async_smem();
    };
    auto multiply = [&](int lower) {   // one thread
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint64_t da = da0 + (uint64_t)(h * (SR_A_BYTES >> 4));
            const uint32_t d = tmem_base + (uint32_t)(2 * lower + h) * N;
            umma<MMA_TF32>(d, da, db, idesc, 0u);
            umma<MMA_TF32>(d, da + 2, db + 2, idesc, 1u);
            umma<MMA_TF32>(d, da + 4, db + 4, idesc, 1u);
            umma<MMA_TF32>(d, da + 6, db + 6, idesc, 1u);
        }
        umma_commit(done0 + 8 * lower);
    };
    auto finish = [&](float sum, float sc, float sf) {
        float t = fmaf(sum, sc, sf);
        t = fmaxf(t, 0.1f * t);
        return do_round ? round_tf32(t) : t;
    };

    // what was fetched, into the patch of its tile
    auto put = [&](float *to_patch) {
        if (loads) {
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int k = 0; k < STEPS; ++k) to_patch[c * PLANE + k * (LINES * SRP_PITCH) + tid] = round_tf32(v[c][k]);
        }
        if (keep && in_column && own_column) {   // a copy of the images: every value by the tile whose pixel it is
            float *const to = keep + (base - x);
            const int left = g.h - (2 * next_y - 1 + line);   // image rows from this thread's first on
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int k = 0; k < STEPS; ++k) {
                    const bool own = (k > 0 || line > 0) && (k < STEPS - 1 || line < LINES - 1);   // not the rows above and below
                    if (own && LINES * k < left) to[c * xs_c + k * step_h] = v[c][k];
                }
        }
    };

    bool failed = false;
    if ((int)blockIdx.x < tiles) { fetch(blockIdx.x); put(patch); }
    __syncthreads();
    int it = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {   // uniform over the CTA
        const int b = next_b, tile_y = next_y, tile_x = next_x, py = next_y + wy, px = next_x + wx;
        const bool more = tile + (int)gridDim.x < tiles;
        if (more) fetch(tile + gridDim.x);
        if (lane == 0) tma_store_wait_read0();   // the last tile's store has read this warp's rows
        __syncwarp();
#pragma unroll
        for (int q = PIECES; q < 8; ++q)         // ... whose values, where an im2col row has none, an infinity among them would multiply the filters' zeros
            *reinterpret_cast<uint4 *>(row + ((q ^ sw) << 4)) = make_uint4(0u, 0u, 0u, 0u);
        build(from + (it & 1) * (C * PLANE));
        __syncthreads();
        if (tid == 0) multiply(0);
        __syncwarp();
        if (more) put(patch + ((it + 1) & 1) * (C * PLANE));   // while the upper pixels are multiplied (after the second build: 145.5 us, this 141.8)
        if (!mbar_wait(done0, (uint32_t)(it & 1), abort_flag, status, SR_WAIT_ACC, 0, wait_limit)) failed = true;
        if (!failed) build(from + (it & 1) * (C * PLANE) + SRP_PITCH);
        if (__syncthreads_or(failed)) break;
        if (tid == 0) multiply(1);
        __syncwarp();
        if (!mbar_wait(done0 + 8, (uint32_t)(it & 1), abort_flag, status, SR_WAIT_ACC, 0, wait_limit)) { failed = true; continue; }   // all leave together, at the next tile's vote
        // ---- the window's largest sums
        tc_fence_after();
        const uint32_t t_row = tmem_base + ((uint32_t)(warp * 32) << 16);
        const bool stores = 2 * py < g.out_h && 2 * px < g.out_w;
        const size_t window = ((size_t)b * (g.out_h >> 1) + py) * (g.out_w >> 1) + px;
        uint32_t sg[8];
#pragma unroll
        for (int c0 = 0; c0 < N; c0 += 16) {
            uint32_t r[4][16], o[16];
#pragma unroll
            for (int p = 0; p < 4; ++p) tmem_ld16(t_row + p * N + c0, r[p]);
            tmem_ld_wait();
            if (negative) {
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int j = 0; j < 16; ++j) r[p][j] ^= (negative << (31 - c0 - j)) & 0x80000000u;
            }
            bool odd_value = !plain;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float m = largest_or_nan(r[0][j], r[1][j], r[2][j], r[3][j]);
                odd_value |= !(fabsf(m) < INFINITY);
                o[j] = __float_as_uint(m);
            }
            if (__any_sync(0xffffffffu, odd_value)) {   // (a block by itself: as a condition at every value it cost its instructions every time)
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float sc = s_scale[c0 + j], sf = s_shift[c0 + j];
                    float t = finish(__uint_as_float(r[0][j]), sc, sf);
#pragma unroll
                    for (int p = 1; p < 4; ++p) t = fmaxf(t, finish(__uint_as_float(r[p][j]), sc, sf));
                    o[j] = __float_as_uint(fmaxf(-FLT_MAX, t));
                }
            } else {
                const float4 *const sc4 = reinterpret_cast<const float4 *>(s_scale + c0), *const sf4 = reinterpret_cast<const float4 *>(s_shift + c0);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 sc = sc4[q], sf = sf4[q];
                    const float scv[4] = {sc.x, sc.y, sc.z, sc.w}, sfv[4] = {sf.x, sf.y, sf.z, sf.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[4 * q + e] = __float_as_uint(fmaxf(-FLT_MAX, finish(__uint_as_float(o[4 * q + e]), scv[e], sfv[e])));
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) sg[c0 / 4 + q] = four_signs_no_nan(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
            // staged where the tile's rows were, which its MMAs have read
#pragma unroll
            for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4 *>(row + (((c0 / 4 + q) ^ sw) << 4)) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {   // a warp's 16 x 2 windows; the TMA unit clips them
            tma_store_4d(&a.tmy, smem_u32(sA + warp * 4096), 0, tile_x, tile_y + 2 * warp, b);
            tma_store_commit();
        }
        if (signs && stores) st_global_32(signs + window * 32, sg);
        tc_fence_before();        // this thread's TMEM loads precede the barriers before the next MMAs
    }
    if (lane == 0) tma_store_wait_all();

    // ---- teardown (also the abort path)
    if (*abort_flag) {   // give MMAs that may still read shared memory time to retire
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000LL) { }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)a.tmem_cols) : "memory");
    }
}

// ------------------------------------------------------------------ wider first layers (5x5, 7x7 over RGB)
// K = c*size*size no longer fits one 128-byte row (147 for ResNet's 7x7 layer): the tile's im2col rows are built
// and multiplied in blocks of 32 values.  Two 16 KB row buffers alternate; the MMAs of block kb read one while
// the threads gather block kb+1 into the other; the filter matrix (all blocks) stays in shared memory.  The
// epilogue follows the last block's MMAs, staged over both row buffers and stored by TMA, one or two boxes of
// 32 rows x 128 bytes per warp.
struct StemRowsWideShared {
    uint64_t mma_done[2];   // the MMAs that read row buffer i have retired
    uint64_t acc_full;
    uint32_t tmem_base;
    int abort_flag;
};

template <int C, int KS, int ACT, bool OUT_BF16>
__global__ void __launch_bounds__(SR_THREADS, 3)
conv_stem_rows_wide_kernel(const __grid_constant__ StemTcArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0) atomicCAS(a.status, 0, SR_BAD_SMEM_BASE);
        return;
    }
    constexpr int K = C * KS * KS, KB = (K + 31) / 32;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_pad = a.n_pad;
    uint8_t *sA = smem;                              // 2 x 128 rows x 128 bytes; also the staging rows of the epilogue
    uint8_t *sB = smem + 2 * SR_A_BYTES;             // KB blocks of n_pad rows x 128 bytes
    float *s_scale = reinterpret_cast<float *>(sB + (size_t)KB * n_pad * 128);
    float *s_shift = s_scale + n_pad;
    StemRowsWideShared *sh = reinterpret_cast<StemRowsWideShared *>(s_shift + n_pad);
    volatile int *abort_flag = &sh->abort_flag;
    const ConvGeom g = a.g;

    for (int i = tid; i < KB * n_pad * 8; i += SR_THREADS) {
        const int kb = i / (n_pad * 8), r = i - kb * n_pad * 8, f = r >> 3, q = r & 7;
        uint32_t v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int k = kb * 32 + 4 * q + e;
            v[e] = (k < K && f < g.n) ? __float_as_uint(round_tf32(__ldg(a.w + (size_t)k * a.npg_pad + f))) : 0u;
        }
        *reinterpret_cast<uint4 *>(sB + (size_t)kb * n_pad * 128 + f * 128 + ((q ^ (f & 7)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
    }
    for (int i = tid; i < n_pad; i += SR_THREADS) {
        s_scale[i] = i < g.n ? __ldg(a.ep.scale + i) : 0.f;
        s_shift[i] = i < g.n ? __ldg(a.ep.shift + i) : 0.f;
    }
    if (tid == 0) {
        mbar_init(smem_u32(&sh->mma_done[0]), 1);
        mbar_init(smem_u32(&sh->mma_done[1]), 1);
        mbar_init(smem_u32(&sh->acc_full), 1);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem_cols = (uint32_t)a.tmem_cols;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = sh->tmem_base;
    grid_dependency_wait();   // up to here only the layer's own parameters were read
    launch_dependents();

    const float *const x = a.x;
    const long long xs_b = a.xs_b;
    const long long xs_c = a.xs_c, xs_h = a.xs_h;
    const int xs_w = (int)a.xs_w;
    const int npix = a.npix, tiles = a.tiles, plane = g.out_h * g.out_w;
    const int runtime_act = a.ep.activation, do_round = a.ep.round_tf32;
    int *const status = a.status;
    const long long wait_limit = a.wait_limit;
    const uint32_t idesc = mma_idesc<MMA_TF32>(128u, (uint32_t)n_pad);
    const uint64_t db0 = make_smem_desc(smem_u32(sB), 128);
    const uint64_t da0 = make_smem_desc(smem_u32(sA), 128);
    const uint64_t b_step = (uint64_t)((n_pad * 128) >> 4);
    const uint32_t done0 = smem_u32(&sh->mma_done[0]), acc_bar = smem_u32(&sh->acc_full);
    const uint32_t row_off = (uint32_t)tid * 128u, sw = (uint32_t)(tid & 7);
    const uint32_t out_row_bytes = (uint32_t)a.y_cpitch * (OUT_BF16 ? 2u : 4u);   // 32, 64, 128 or 256
    const uint32_t half_bytes = out_row_bytes > 128 ? 128u : out_row_bytes;       // bytes of a row per staging half
    const uint32_t q_mask = half_bytes / 16 - 1;
    const uint32_t q_xor = (half_bytes == 128 ? (uint32_t)tid : (half_bytes == 64 ? (uint32_t)(tid >> 1) : (uint32_t)(tid >> 2))) & q_mask;
    const CUtensorMap *ymap = &a.tmy;

    bool failed = false, stop = false;
    uint32_t kcount = 0;        // blocks of 32 K values processed so far (buffer = kcount & 1)
    int it = 0;
    for (int tile = blockIdx.x; tile < tiles && !stop; tile += gridDim.x, ++it) {
        const int p = tile * SR_THREADS + tid;
        const bool valid = p < npix;
        const int b = p / plane, rem = p - b * plane;
        const int oy = rem / g.out_w, ox = rem - oy * g.out_w;
        const int iy0 = oy * g.stride - g.pad, ix0 = ox * g.stride - g.pad;
        uint32_t rmask = 0, cmask = 0;   // bit k: row iy0+k / column ix0+k is inside the image
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            rmask |= (valid && (unsigned)(iy0 + k) < (unsigned)g.h) ? (1u << k) : 0u;
            cmask |= ((unsigned)(ix0 + k) < (unsigned)g.w) ? (1u << k) : 0u;
        }
        const float *xp = x + (size_t)b * xs_b + (long long)iy0 * xs_h + (long long)ix0 * xs_w;   // dereferenced only where valid
        // the previous tile's stores read the row buffers this tile overwrites
        if (lane == 0) tma_store_wait_read0();
        __syncwarp();
#pragma unroll
        for (int kb = 0; kb < KB; ++kb) {
            const uint32_t buf = kcount & 1u, use = kcount >> 1;
            if (use > 0 && !mbar_wait(done0 + 8 * buf, (use - 1) & 1u, abort_flag, status, SR_WAIT_ACC, 0, wait_limit)) failed = true;
            float v[32];
#pragma unroll
            for (int t = 0; t < 32; ++t) {
                const int k = kb * 32 + t;
                if (k < K) {
                    const int c = k / (KS * KS), r = k - c * KS * KS, kh = r / KS, kw = r - kh * KS;
                    const bool in = ((rmask >> kh) & (cmask >> kw) & 1u) != 0;
                    v[t] = in ? __ldg(xp + c * xs_c + kh * xs_h + kw * xs_w) : 0.f;
                } else {
                    v[t] = 0.f;
                }
            }
            uint8_t *row = sA + buf * SR_A_BYTES + row_off;
#pragma unroll
            for (int q = 0; q < 8; ++q)
                *reinterpret_cast<uint4 *>(row + ((q ^ sw) << 4)) =
                    make_uint4(__float_as_uint(round_tf32(v[4 * q])), __float_as_uint(round_tf32(v[4 * q + 1])),
                               __float_as_uint(round_tf32(v[4 * q + 2])), __float_as_uint(round_tf32(v[4 * q + 3])));
            fence_async_smem();
            tc_fence_before();
            if (__syncthreads_or(failed)) { stop = true; break; }
            if (tid == 0) {
                tc_fence_after();
                const uint64_t da = da0 + (uint64_t)(buf * (SR_A_BYTES >> 4)), db = db0 + kb * b_step;
                umma<MMA_TF32>(tmem_base, da, db, idesc, kb > 0 ? 1u : 0u);
                umma<MMA_TF32>(tmem_base, da + 2, db + 2, idesc, 1u);
                umma<MMA_TF32>(tmem_base, da + 4, db + 4, idesc, 1u);
                umma<MMA_TF32>(tmem_base, da + 6, db + 6, idesc, 1u);
                umma_commit(done0 + 8 * buf);
                if (kb == KB - 1) umma_commit(acc_bar);
            }
            __syncwarp();
            ++kcount;
        }
        if (stop) break;
        // ---- epilogue: all of the tile's MMAs have retired, the row buffers are free for the staged output
        if (!mbar_wait(acc_bar, (uint32_t)(it & 1), abort_flag, status, SR_WAIT_ACC, 0, wait_limit)) failed = true;
        if (!failed) {
            tc_fence_after();
            const uint32_t t_row = tmem_base + ((uint32_t)(warp * 32) << 16);
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
                        float t = rows_act<ACT>(fmaf(__uint_as_float(r[j]), scv[e], sfv[e]), runtime_act);
                        if (do_round) t = round_tf32(t);
                        o[j] = (ACT == SR_ACT_GENERIC && c0 + j >= g.n) ? 0.f : t;
                    }
                }
                // byte offset of these 16 columns inside the pixel's row, split into 128-byte halves
                const uint32_t byte0 = (uint32_t)c0 * (OUT_BF16 ? 2u : 4u);
                uint8_t *half = sA + (byte0 >> 7) * SR_A_BYTES + (uint32_t)tid * half_bytes;
                const uint32_t q0 = (byte0 & 127u) >> 4;
                if (!OUT_BF16) {
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        *reinterpret_cast<uint4 *>(half + (((q0 + q) ^ q_xor) << 4)) =
                            make_uint4(__float_as_uint(o[4 * q]), __float_as_uint(o[4 * q + 1]), __float_as_uint(o[4 * q + 2]), __float_as_uint(o[4 * q + 3]));
                } else {
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        uint4 pk;
                        __nv_bfloat162 h0 = __floats2bfloat162_rn(o[8 * q], o[8 * q + 1]);
                        __nv_bfloat162 h1 = __floats2bfloat162_rn(o[8 * q + 2], o[8 * q + 3]);
                        __nv_bfloat162 h2 = __floats2bfloat162_rn(o[8 * q + 4], o[8 * q + 5]);
                        __nv_bfloat162 h3 = __floats2bfloat162_rn(o[8 * q + 6], o[8 * q + 7]);
                        pk.x = *reinterpret_cast<uint32_t *>(&h0); pk.y = *reinterpret_cast<uint32_t *>(&h1);
                        pk.z = *reinterpret_cast<uint32_t *>(&h2); pk.w = *reinterpret_cast<uint32_t *>(&h3);
                        *reinterpret_cast<uint4 *>(half + (((q0 + q) ^ q_xor) << 4)) = pk;
                    }
                }
            }
            fence_async_smem();
            __syncwarp();
            const int row0 = tile * SR_THREADS + warp * 32;
            if (lane == 0 && row0 < npix) {
                for (uint32_t hb = 0; hb * 128u < out_row_bytes; ++hb)
                    tma_store_2d(ymap, smem_u32(sA + hb * SR_A_BYTES) + (uint32_t)(warp * 32) * half_bytes,
                                 (int)(hb * 128u / (OUT_BF16 ? 2u : 4u)), row0);
                tma_store_commit();
            }
        }
        tc_fence_before();   // this tile's TMEM loads precede the next tile's first barrier and MMA
    }
    if (lane == 0) tma_store_wait_all();

    if (*abort_flag) {
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
// What conv_stem_tc.cu covers, but for 5x5 and 7x7 layers whose output rows are not whole swizzle spans.
bool conv_stem_rows_covers(const ConvGeom &g, int y_dtype)
{
    const int rb = g.n * (y_dtype == DNB_BF16 ? 2 : 4);
    return conv_stem_tc_covers(g) && (g.size == 3 || rb == 32 || rb == 64 || rb == 128 || rb == 256) &&
           (long long)g.batch * g.out_h * g.out_w + SR_THREADS < (1LL << 31);
}

bool conv_stem_rows_pool_covers(const ConvGeom &g, int y_dtype) { return conv_stem_rows_covers(g, y_dtype) && y_dtype == DNB_F32 && g.n == 32; }

template <typename K>
static int launch_rows(K kern, size_t smem, int most, const StemTcArgs &a, cudaStream_t s)
{
    smem = tmem_smem(smem, a.tmem_cols);
    const size_t sm_bytes = 228 * 1024, reserved = 1024;   // per SM, and per resident CTA
    DNB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // all of the SM's configurable memory as shared memory, so that several CTAs are resident
    DNB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    int per_sm = (int)(sm_bytes / (smem + reserved));
    if (per_sm > most) per_sm = most;   // the kernel's register budget (__launch_bounds__)
    if (per_sm < 1) DNB_FAIL(DNB_ECUDA, "first-layer kernel: %zu bytes of shared memory do not fit", smem);
    long long grid = (long long)sm_count() * per_sm;
    if (grid > a.tiles) grid = a.tiles;
    DNB_CUDA(launch_overlapped(kern, dim3((unsigned)grid), dim3(SR_THREADS), smem, s, a));
    DNB_LAUNCH_CHECK("conv_stem_rows");
    return DNB_OK;
}

template <int C, bool OBF>
static int launch_narrow(const StemTcArgs &a, cudaStream_t s)
{
    const size_t smem = 2 * SR_A_BYTES + (size_t)a.n_pad * 128 + 2 * sizeof(float) * a.n_pad + sizeof(StemRowsShared) + 16;
    if constexpr (!OBF)
        if (a.pool) {
            const size_t pooled = 2 * SR_A_BYTES + 32 * 128 + 2 * sizeof(float) * 32 + 2 * sizeof(float) * C * SRP_PITCH * SRP_ROWS + sizeof(StemRowsPoolShared) + 16;
            return launch_rows(conv_stem_rows_pool_kernel<C>, pooled, 4, a, s);
        }
    if (a.ep.activation == DNB_LEAKY) return launch_rows(conv_stem_rows_kernel<C, DNB_LEAKY, OBF>, smem, 5, a, s);
    return launch_rows(conv_stem_rows_kernel<C, SR_ACT_GENERIC, OBF>, smem, 5, a, s);
}

template <int KS, bool OBF>
static int launch_wide(const StemTcArgs &a, cudaStream_t s)
{
    constexpr int KB = (3 * KS * KS + 31) / 32;
    const size_t smem = 2 * SR_A_BYTES + (size_t)KB * a.n_pad * 128 + 2 * sizeof(float) * a.n_pad + sizeof(StemRowsWideShared) + 16;
    if (a.ep.activation == DNB_LEAKY) return launch_rows(conv_stem_rows_wide_kernel<3, KS, DNB_LEAKY, OBF>, smem, 3, a, s);
    return launch_rows(conv_stem_rows_wide_kernel<3, KS, SR_ACT_GENERIC, OBF>, smem, 3, a, s);
}

template <bool OBF>
static int launch_geometry(const StemTcArgs &a, cudaStream_t s)
{
    if (a.g.size == 7) return launch_wide<7, OBF>(a, s);
    if (a.g.size == 5) return launch_wide<5, OBF>(a, s);
    return a.g.c == 1 ? launch_narrow<1, OBF>(a, s) : a.g.c == 2 ? launch_narrow<2, OBF>(a, s) : launch_narrow<3, OBF>(a, s);
}

int launch_conv_stem_rows(StemTcArgs a, cudaStream_t s)
{
    const ConvGeom &g = a.g;
    if (!conv_stem_rows_covers(g, a.y_dtype) || a.y_cpitch != g.n) DNB_FAIL(DNB_EUNSUPPORTED, "first-layer kernel: geometry outside its coverage");
    if (a.xs_c >= (1LL << 31) / 4 || a.xs_h >= (1LL << 31) / 4) DNB_FAIL(DNB_EUNSUPPORTED, "first-layer kernel: image too large for 32-bit offsets");
    if (a.pool && !(conv_stem_pool_covers(g, a.y_dtype, a.ep.activation) && conv_stem_rows_pool_covers(g, a.y_dtype))) DNB_FAIL(DNB_EINVAL, "first-layer kernel: no pooled variant of this layer");
    a.n_pad = round_up(g.n, 16);
    a.tmem_cols = 32;
    while (a.tmem_cols < a.n_pad) a.tmem_cols *= 2;
    if (a.pool) {
        a.tiles_w = (g.out_w / 2 + SRP_TW - 1) / SRP_TW;
        a.tiles_h = (g.out_h / 2 + SRP_TH - 1) / SRP_TH;
        a.tiles = g.batch * a.tiles_w * a.tiles_h;
        a.tmem_cols = 128;   // four accumulators of 32 columns
        const uint64_t pw = (uint64_t)g.out_w / 2, ph = (uint64_t)g.out_h / 2;
        const uint64_t dims[4] = {32u, pw, ph, (uint64_t)g.batch}, strides[3] = {128u, 128u * pw, 128u * pw * ph};
        const uint32_t box[4] = {32u, (uint32_t)SRP_TW, 32u / SRP_TW, 1u};
        DNB_TRY(encode_tensor_map(&a.tmy, 0, 4, a.y, dims, strides, box, 128));
        return launch_geometry<false>(a, s);
    }
    const long long npix = (long long)g.batch * g.out_h * g.out_w;   // output pixels
    a.npix = (int)npix;
    a.tiles = (int)((npix + SR_THREADS - 1) / SR_THREADS);
    // rows of 32, 64 or 128 bytes leave through TMA stores from swizzled staging rows, the wide kernel's 256-byte rows in two halves;
    // other ones by plain stores
    const int es = a.y_dtype == DNB_BF16 ? 2 : 4, rb = g.n * es, half = rb > 128 ? 128 : rb;
    a.tma_store = rb == 32 || rb == 64 || rb == 128 || g.size != 3;
    if (a.tma_store) {
        const uint64_t dims[2] = {(uint64_t)g.n, (uint64_t)npix};
        const uint64_t strides[1] = {(uint64_t)rb};
        const uint32_t box[2] = {(uint32_t)(half / es), 32u};
        DNB_TRY(encode_tensor_map(&a.tmy, es == 2 ? 1 : 0, 2, a.y, dims, strides, box, half));
    }
    return es == 2 ? launch_geometry<true>(a, s) : launch_geometry<false>(a, s);
}

}  // namespace dnb
