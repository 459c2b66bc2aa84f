// Full-precision convolution on the sm_100a tensor cores: implicit GEMM as in conv_tc.cu, every fp32 operand as the sum of
// three bf16 numbers (the splitting of Henry, Tang and Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For
// Higher-Precision Computations", 2019), sums in fp32 registers.
//
//   x = x0 + x1 + x2, w = w0 + w1 + w2    (x0: x rounded to bf16; x1: the rest, rounded to bf16; x2: what is left, exactly: 8 + 8 + 8 bits)
//   x*w = x0*w0 + (x1*w2 + x2*w1 + x1*w1 + x2*w0 + x0*w2 + x1*w0 + x0*w1)       (x2*w2, at most 2^-34 of the product, is left out)
//
// What bounds the fp32 GEMM of conv_direct.cu is operand pairing and FMA issue on the CUDA cores, 37 TFLOP/s.  What has to hold is its
// precision.  The products of bf16 numbers are exact in the tensor core; its running sums, which it cuts off instead of rounding them, are not.  So
// there are two: the large products' (x0*w0, 16 bits each) leaves TMEM after the 32 channels of a tap and is added to a register, rounded to
// nearest; the small ones', whose cut-off digits count 2^-8 of that, goes on for up to 64 such steps, and is added at the end.  A sum of one product is
// that product rounded, 2^-24 as in fp32, of a few mostly just as well, and a factor of 1 is exact.  (Two TF32 halves with one sum for all, 22 bits
// and cut off, were 2.4 times as far from 64 bits as fp32 for sums of one to a few products; the small sums added step by step, a rounding
// more for each, 1.2 times.)  Error of dense sums: see fp32_tc_covers in conv_plan.cu, where it is set beside the CUDA-core kernel's.
//
// * Tile: 128 output pixels (a wt x ht x bt box) by BN filters; a step of K is one tap and 32 channels, sixteen MMAs.
// * Warp 0 loads a step by TMA: BN x 32 of each part of w, and of a channels-last input 16 KB as it is.  The input goes through
//   registers anyway to be split, so its parts are written to TMEM, where the MMA takes its A operand from: no shared memory for
//   them, and half of what the MMAs would read there.
// * A Darknet tensor needs no channels-last copy: its channels are planes, so the threads that split fetch their pixel's 32 values
//   themselves, along the plane's rows, the next step's while this one's are multiplied.  The ring then holds filters only, and what
//   is left of an SM's 256 KB caches the rows, which the nine taps of a block of channels read one after the other.  No scratch, no
//   allocation, no state but the plan's weights: a plan may run on several streams and threads at once, and under capture as without.
// * Warps 4-11 split, one half of them the even steps, the other the odd ones: a thread takes its pixel's row, writes 16 columns of
//   each part.  (Four warps for all steps: 110 us where eight took 80, 8 x 64 x 104 x 104 -> 128, 3x3; a step's way through a
//   warp is all latency.)
// * Warp 1 issues a step's MMAs, the large products' first, into one of two accumulators that is added up while the small ones' MMAs run, then those.
// * Warps 12-19 add the finished accumulators to registers, half the filters each, and after the tile's last step scale, shift,
//   activate and store.  They take the registers that the other warps give up.
// * A ring of four slots of shared memory for what TMA brings, and one of 48 columns of TMEM each for the split rows: two beside three
//   accumulators of 128 columns, four beside narrower ones.
// * Parts and products must be numbers that bf16 and the tensor core's fp32 hold in full.  The threads that split look at what they split: a pixel that has
//   read a value other than zero below a.smallest (2^-90 over the layer's smallest weight, at least 2^-100: every product is then 2^-90 or more, and
//   what counts of it, 2^-26, a normal number) is added up again in fp32, product by product in the CUDA-core kernel's order, and so is one with a sum that
//   is infinite or NaN, which operands beyond bf16's largest number make too.  Layers with weights below 2^-45 run on the CUDA cores.
// * Every wait is bounded as in conv_tc.cu.
#include <cuda.h>

#include "common.h"
#include "conv.h"
#include "device_utils.cuh"
#include "tc_ptx.cuh"

namespace dnb {

namespace {

constexpr int FT_THREADS = 640;
// registers a thread: 96 at launch; 128 * (40 + 2 * 96 + 2 * 120) of the launch's 128 * 5 * 96 after the shift
constexpr int FT_REGS_ISSUE = 40, FT_REGS_SPLIT = 96, FT_REGS_SUM = 120;
static_assert(FT_REGS_ISSUE + 2 * FT_REGS_SPLIT + 2 * FT_REGS_SUM <= 5 * 96, "no more registers than the launch has");
constexpr int FT_STAGES = 4;
constexpr int FT_A_BYTES = 128 * 128;
constexpr int FT_TMEM = 512;
constexpr int FT_SLOT = 48;                // columns of a split row: 16 of each part
constexpr int FT_RUN = 64;                 // steps after which the small products' sum is added up
template <int BN> constexpr int FT_SLOTS = BN == 128 ? 2 : 4;
static_assert(FT_SLOTS<128> * FT_SLOT + 3 * 128 <= FT_TMEM && FT_SLOTS<64> * FT_SLOT + 3 * 64 <= FT_TMEM, "columns");

struct FtShared {
    uint64_t full[FT_STAGES];      // a step's tiles are in shared memory
    uint64_t empty[FT_STAGES];     // its MMAs have retired
    uint64_t split[4];             // a step's input rows are in TMEM
    uint64_t split_empty[4];       // ... and the MMAs that read them have retired
    uint64_t acc_full[3], acc_empty[3];   // the large products' two, the small ones'
    uint32_t tiny[2][2][4];        // of a tile (even and odd ones in turn): pixels that have read a tiny value, by half of the splitting warps and quarter
    uint32_t tmem_base;
    int abort_flag;
};

enum { FT_WAIT_EMPTY = 101, FT_WAIT_FULL = 102, FT_WAIT_ACC_EMPTY = 103, FT_WAIT_ACC_FULL = 104, FT_WAIT_SPLIT = 105, FT_BAD_BASE = 106 };

// A from TMEM: row i of the operand in lane i, a column per two bf16 values.
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}

// x1*w2 + x2*w1 + x1*w1 + x2*w0 + x0*w2 + x1*w0 + x0*w1 over K slices of 16 channels; the parts of w lie PART bytes apart
template <uint32_t PART, int K>
__device__ __forceinline__ void small_products(uint32_t d, uint32_t x, uint64_t w, uint32_t idesc, uint32_t accumulate)
{
    constexpr int xi[7] = {1, 2, 1, 2, 0, 1, 0}, wi[7] = {2, 1, 1, 0, 2, 0, 1};
#pragma unroll
    for (int i = 0; i < 7; ++i)
#pragma unroll
        for (int k = 0; k < K; ++k) umma_bf16_ts(d, x + 16 * xi[i] + 8 * k, w + wi[i] * (PART >> 4) + 2 * k, idesc, i + k ? 1u : accumulate);
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ const float ft_zero = 0.f;   // what a tap outside the image reads: 32 predicates a step cost more than 32 loads of it (32 x 64 x 104 x 104 -> 64: 373 us, 289 without)

// Two values' nearest bf16 as one word (first in the low half), and what is left of them.  An infinity leaves a NaN.
__device__ __forceinline__ uint32_t take_bf16(float &a, float &b)
{
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    a -= __uint_as_float(r << 16);
    b -= __uint_as_float(r & 0xffff0000u);
    return r;
}

// The 128 threads of one of the two halves that sum meet, and agree on whether to go on.
__device__ __forceinline__ bool meet(int half, bool fine)
{
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %2, 0;\n\t"
        "bar.red.and.pred q, %1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all) : "r"(1 + half), "r"((uint32_t)fine) : "memory");
    return all != 0;
}

template <int ACT>
__device__ __forceinline__ float apply(float x, int act)
{
    if (ACT == DNB_LEAKY) return fmaxf(x, 0.1f * x);
    return ACT == DNB_LINEAR ? x : activate_fast(x, act);
}

// Where the sums of pixel m (of 128) and of one half's filters of a tile belong.
struct FtTile {
    int n0, ow0, oh0, b0, ow, oh, b;
    bool inside;
    __device__ __forceinline__ FtTile(const Fp32TcArgs &a, int tile, int bn, int col0, int m)
    {
        const int pt = tile / a.n_tiles;
        n0 = tile % a.n_tiles * bn + col0;
        ow0 = pt % a.tiles_w * a.wt; oh0 = pt / a.tiles_w % a.tiles_h * a.ht; b0 = pt / (a.tiles_w * a.tiles_h) * a.bt;
        ow = ow0 + m % a.wt; oh = oh0 + m / a.wt % a.ht; b = b0 + m / (a.wt * a.ht);
        inside = ow < a.g.out_w && oh < a.g.out_h && b < a.g.batch;
    }
};

// Scale, shift, activation and stores of a finished tile's half.
template <int BN, int ACT>
__device__ __forceinline__ void finish_tile(const Fp32TcArgs &a, const FtTile &at, const float (&sum)[BN / 2], uint8_t *staged, int half, int m, bool stored)
{
    constexpr int COLS = BN / 2, LD = COLS < 32 ? COLS : 32, ROW = LD * 4;
    const ConvGeom &g = a.g;
    const int act = a.ep.activation, n0 = at.n0, real = g.n - n0;
    const bool stores = m == 0;
    uint8_t *const my_row = staged + m * ROW;
    const int q_xor = (m >> (ROW == 128 ? 0 : 1)) & (ROW / 16 - 1);   // the store map's swizzle
    const size_t plane = (size_t)g.out_h * g.out_w, pix = (size_t)at.oh * g.out_w + at.ow;
    float *const nchw = a.y_nchw && at.inside ? a.y_nchw + ((size_t)at.b * g.n + n0) * plane + pix : nullptr;
#pragma unroll
    for (int c = 0; c < COLS; c += LD) {
        if (a.y_nhwc && (c > 0 || stored)) {            // the row's last store has been read
            if (stores) tma_store_wait_read0();
            meet(half, true);
        }
#pragma unroll
        for (int q = c / 4; q < (c + LD) / 4; ++q) {
            float v[4];
            const bool in = n0 + 4 * q < a.n_pad;       // whole quads: n_pad is a multiple of 16
            const float4 sc = in ? __ldg(reinterpret_cast<const float4 *>(a.ep.scale + n0) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 sf = in ? __ldg(reinterpret_cast<const float4 *>(a.ep.shift + n0) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float scv[4] = {sc.x, sc.y, sc.z, sc.w}, sfv[4] = {sf.x, sf.y, sf.z, sf.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = 4 * q + e < real ? apply<ACT>(sum[4 * q + e] * scv[e] + sfv[e], act) : 0.f;
            if (a.y_nhwc) *reinterpret_cast<float4 *>(my_row + (((q - c / 4) ^ q_xor) << 4)) = make_float4(v[0], v[1], v[2], v[3]);
            if (nchw) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (4 * q + e < real) nchw[(size_t)(4 * q + e) * plane] = v[e];
            }
        }
        if (a.y_nhwc) {
            fence_async_smem();
            meet(half, true);
            // the TMA unit clips the box at the tensor's extents: ragged tiles need no predicates
            if (stores && c < real) { tma_store_4d(&a.tmy, smem_u32(staged), n0 + c, at.ow0, at.oh0, at.b0); tma_store_commit(); }
        }
    }
}

// Rarely: the sums of an odd pixel in the order c, kh, kw, the CUDA-core kernel's over a Darknet tensor, each weight from shared memory, where the half's
// threads put 32 products' at a time; the other pixels' threads add 0 * w.  (A sum at a time in its own thread, 8 x 64 x 104 x 104 -> 128 full of
// NaN took 53 ms.  So it takes five times as long as the CUDA-core kernel, which reads a weight for eight pixels.)
template <int COLS>   // at most 32
__device__ __noinline__ void add_again(const Fp32TcArgs &a, float *sums, uint8_t *staged, bool odd, int half, int n0, int b, int oh, int ow)
{
    const ConvGeom &g = a.g;
    float sum[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) sum[j] = sums[j];
    float4 *const wk = reinterpret_cast<float4 *>(staged);
    const int products = g.c * g.size * g.size, ih0 = oh * g.stride - g.pad, iw0 = ow * g.stride - g.pad;
    const float *const image = a.x + (long long)b * a.xs_b;
    int k = 0, c = 0, kh = 0, kw = 0;               // of the next input value
    auto next_x = [&]() {
        const int ih = ih0 + kh, iw = iw0 + kw;
        const bool in = odd && k < products && (unsigned)ih < (unsigned)g.h && (unsigned)iw < (unsigned)g.w;
        const float v = in ? __ldg(image + c * a.xs_c + ih * a.xs_h + iw * a.xs_w) : 0.f;
        ++k;
        if (++kw == g.size) { kw = 0; if (++kh == g.size) { kh = 0; ++c; } }
        return v;
    };
    float x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = next_x();
    for (int k0 = 0; k0 < products; k0 += 32) {
        meet(half, true);
        for (int i = threadIdx.x & 127; i < 32 * COLS / 4; i += 128) {
            const int kk = k0 + i / (COLS / 4), f = n0 + 4 * (i % (COLS / 4));
            wk[i] = kk < products && f < a.npg_pad ? __ldg(reinterpret_cast<const float4 *>(a.w + (size_t)kk * a.npg_pad + f)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        meet(half, true);
#pragma unroll 1
        for (int kk = 0; kk < 32; kk += 4) {
            float later[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) later[u] = next_x();
#pragma unroll
            for (int u = 0; u < 4; ++u) {
#pragma unroll
                for (int q = 0; q < COLS / 4; ++q) {
                    const float4 w = wk[(kk + u) * (COLS / 4) + q];
                    sum[4 * q] = fmaf(x[u], w.x, sum[4 * q]);
                    sum[4 * q + 1] = fmaf(x[u], w.y, sum[4 * q + 1]);
                    sum[4 * q + 2] = fmaf(x[u], w.z, sum[4 * q + 2]);
                    sum[4 * q + 3] = fmaf(x[u], w.w, sum[4 * q + 3]);
                }
                x[u] = later[u];
            }
        }
    }
    meet(half, true);
#pragma unroll
    for (int j = 0; j < COLS; ++j) sums[j] = sum[j];
}

// ... and a tile that has such pixels.  A function of its own: its registers are not the kernel's loop's.
template <int BN, int ACT>
__device__ __noinline__ void odd_tile(const Fp32TcArgs &a, float *sums, uint8_t *staged, bool odd, int half, int tile, int m, bool stored)
{
    constexpr int COLS = BN / 2, LD = COLS < 32 ? COLS : 32;
    const FtTile at(a, tile, BN, half * COLS, m);
    if (a.y_nhwc && stored && m == 0) tma_store_wait_read0();
#pragma unroll 1
    for (int c = 0; c < COLS; c += LD) add_again<LD>(a, sums + c, staged, odd, half, at.n0 + c, at.b, at.oh, at.ow);
    float sum[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) sum[j] = sums[j];
    finish_tile<BN, ACT>(a, at, sum, staged, half, m, stored);
}

// BN: filters per tile; PLANES: the input is a Darknet tensor.
template <int BN, int ACT, bool PLANES>
__global__ void __launch_bounds__(FT_THREADS, 1)
conv_fp32_tc_kernel(const __grid_constant__ Fp32TcArgs a)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    constexpr uint32_t B_BYTES = BN * 64, A_BYTES = PLANES ? 0 : FT_A_BYTES, STAGE = A_BYTES + 3 * B_BYTES;   // 32 channels of one part of w; a stage
    constexpr int SLOTS = FT_SLOTS<BN>;
    constexpr int COLS = BN / 2, LD = COLS < 32 ? COLS : 32;   // filters of one half of the summing warps, columns of a TMEM read and of a staged row
    constexpr int ROW = LD * 4;
    const uint32_t ring = smem_u32(smem_raw);
    if (ring & 1023u) {
        if (threadIdx.x == 0) atomicCAS(a.status, 0, FT_BAD_BASE);
        return;
    }
    FtShared *sh = reinterpret_cast<FtShared *>(smem_raw + FT_STAGES * STAGE + 2 * 128 * ROW);
    volatile int *abort_flag = &sh->abort_flag;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < FT_STAGES; ++s) {
            mbar_init(smem_u32(&sh->full[s]), 1);
            mbar_init(smem_u32(&sh->empty[s]), 1);
        }
        for (int s = 0; s < SLOTS; ++s) {
            mbar_init(smem_u32(&sh->split[s]), 4);
            mbar_init(smem_u32(&sh->split_empty[s]), 1);
        }
        for (int i = 0; i < 3; ++i) {
            mbar_init(smem_u32(&sh->acc_full[i]), 1);
            mbar_init(smem_u32(&sh->acc_empty[i]), 8);
        }
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"((uint32_t)FT_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    launch_dependents();
    grid_dependency_wait();
    const uint32_t tmem_base = sh->tmem_base, acc0 = tmem_base + SLOTS * FT_SLOT;

    const int taps = a.taps, c_blocks = a.c_blocks, steps = taps * c_blocks, last_slices = a.last_slices;
    const int n_tiles = a.n_tiles, total_tiles = a.total_tiles;
    const int wt = a.wt, ht = a.ht, bt = a.bt, tiles_w = a.tiles_w, tiles_h = a.tiles_h;
    const long long limit = a.wait_limit;
    int *status = a.status;
    const uint32_t full0 = smem_u32(&sh->full[0]), empty0 = smem_u32(&sh->empty[0]), split0 = smem_u32(&sh->split[0]), split_empty0 = smem_u32(&sh->split_empty[0]);
    const uint32_t acc_full0 = smem_u32(&sh->acc_full[0]), acc_empty0 = smem_u32(&sh->acc_empty[0]);

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FT_REGS_ISSUE));
    if (warp == 0) {
        // ---------------- loads
        const int ksize = a.g.size, stride = a.g.stride, pad = a.g.pad;
        const bool withhold = (a.debug & 32) != 0;
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
            const int n0 = tile % n_tiles * BN, pt = tile / n_tiles;
            const int ow0 = pt % tiles_w * wt, oh0 = pt / tiles_w % tiles_h * ht, b0 = pt / (tiles_w * tiles_h) * bt;
            for (int cb = 0; cb < c_blocks && ok; ++cb)          // the taps of a block of channels: their rows are neighbours
                for (int tap = 0, kh = 0, kw = 0; tap < taps; ++tap) {
                    const int dh = kh - pad, dw = kw - pad;
                    int ph = 0, qh = dh, pw = 0, qw = dw;
                    if (stride == 2) { ph = dh & 1; qh = (dh - ph) >> 1; pw = dw & 1; qw = (dw - pw) >> 1; }
                    const CUtensorMap *mx = a.tmx + (ph * stride + pw);
                    ok = mbar_wait_warp(empty0 + 8 * stage, phase ^ 1, abort_flag, status, FT_WAIT_EMPTY, limit);
                    if (!ok) break;
                    if (withhold && tile == (int)blockIdx.x && tap == taps - 1 && cb == c_blocks - 1) { ok = false; break; }
                    if (elect_one()) {
                        const uint32_t bar = full0 + 8 * stage, slot = ring + stage * STAGE;
                        mbar_expect_tx(bar, PLANES ? 3 * B_BYTES : STAGE);
                        if (!PLANES) tma_load_4d(slot, mx, bar, cb * 32, ow0 + qw, oh0 + qh, b0);
                        tma_load_4d(slot + A_BYTES, &a.tmw, bar, 0, n0, 0, cb * taps + tap);   // three tiles of BN rows, one of each part
                    }
                    if (++stage == FT_STAGES) { stage = 0; phase ^= 1; }
                    if (++kw == ksize) { kw = 0; ++kh; }
                }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMAs
        const uint32_t idesc = mma_idesc<MMA_BF16>(128u, (uint32_t)BN);
        const uint64_t b_desc0 = make_smem_desc(ring + A_BYTES, 64);
        int stage = 0, slot = 0, acc = 0, run = 0;
        uint32_t phase = 0, slot_phase = 0, acc_phase = 0, small_phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x)
            for (int step = 0, tap = 0, cb = 0; step < steps; ++step) {
                const bool whole = cb != c_blocks - 1 || last_slices == 2;   // all 32 channels; else the first 16
                const uint32_t x0 = tmem_base + slot * FT_SLOT;
                const uint64_t w0 = b_desc0 + (uint64_t)(stage * (STAGE >> 4));
                ok = mbar_wait_warp(acc_empty0 + 8 * acc, acc_phase ^ 1, abort_flag, status, FT_WAIT_ACC_EMPTY, limit) &&
                     mbar_wait_warp(full0 + 8 * stage, phase, abort_flag, status, FT_WAIT_FULL, limit) &&
                     mbar_wait_warp(split0 + 8 * slot, slot_phase, abort_flag, status, FT_WAIT_SPLIT, limit);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t d = acc0 + acc * BN;
                    umma_bf16_ts(d, x0, w0, idesc, 0u);
                    if (whole) umma_bf16_ts(d, x0 + 8, w0 + 2, idesc, 1u);
                    umma_commit(acc_full0 + 8 * acc);
                }
                acc ^= 1;
                if (!acc) acc_phase ^= 1;
                if (run == 0) {
                    ok = mbar_wait_warp(acc_empty0 + 16, small_phase ^ 1, abort_flag, status, FT_WAIT_ACC_EMPTY, limit);
                    if (!ok) break;
                    tc_fence_after();
                }
                const bool last = run == FT_RUN - 1 || step == steps - 1;
                if (elect_one()) {   // the smallest first: they then meet the larger ones in a sum that still has room for them
                    const uint32_t d = acc0 + 2 * BN;
                    if (whole) small_products<B_BYTES, 2>(d, x0, w0, idesc, run != 0);
                    else small_products<B_BYTES, 1>(d, x0, w0, idesc, run != 0);
                    umma_commit(empty0 + 8 * stage);
                    umma_commit(split_empty0 + 8 * slot);
                    if (last) umma_commit(acc_full0 + 16);
                }
                ++run;
                if (last) { run = 0; small_phase ^= 1; }
                if (++tap == taps) { tap = 0; ++cb; }
                if (++stage == FT_STAGES) { stage = 0; phase ^= 1; }
                if (++slot == SLOTS) { slot = 0; slot_phase ^= 1; }
            }
        __syncwarp();
    }
    } else if (warp < 12) {
        // ---------------- split: thread m's row of the input tile (128-byte swizzle) to TMEM lane m
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(FT_REGS_SPLIT));
        const int m = (warp & 3) * 32 + lane, q_xor = m & 7;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        const int mine = (int)blockIdx.x < total_tiles ? (total_tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
        const long long count = (long long)mine * steps;
        // The smallest value but zero this thread's pixel has read of the tile, as twice its bits less one (zero is then the largest).  A tile has four steps or
        // more, two of them this half's; its word is written before the last of them is handed on and read with the tile's last sums.  Before it is
        // written again, two tiles on, a step of the tile between has been added up, by threads that had read the word.
        const uint32_t bound = 2u * a.smallest - 1u;
        uint32_t least = ~0u;
        int left = warp < 8 ? steps : steps - 1, parity = 0;   // steps of the tile from this half's next one on
        // PLANES: this thread's 32 values of a step, zero beyond the image and the channels; steps are asked for in order
        const int channels = a.g.c, ksize = a.g.size, img_h = a.g.h, img_w = a.g.w;
        const long long xs_c = a.xs_c;
        float x[32];
        int tile = blockIdx.x, cb = 0, kh = 0, kw = 0, ih0 = 0, iw0 = 0;
        const float *image = nullptr;     // null outside the output
        auto at_tile = [&]() {
            const int pt = tile / n_tiles;
            const int ow = pt % tiles_w * wt + m % wt, oh = pt / tiles_w % tiles_h * ht + m / wt % ht, b = pt / (tiles_w * tiles_h) * bt + m / (wt * ht);
            ih0 = oh * a.g.stride - a.g.pad; iw0 = ow * a.g.stride - a.g.pad;
            image = ow < a.g.out_w && oh < a.g.out_h && b < a.g.batch ? a.x + (long long)b * a.xs_b : nullptr;
        };
        auto advance = [&]() {            // one step
            if (++kw < ksize) return;
            kw = 0;
            if (++kh < ksize) return;
            kh = 0;
            if (++cb < c_blocks) return;
            cb = 0;
            tile += gridDim.x;
            at_tile();
        };
        auto fetch = [&]() {
            const int ih = ih0 + kh, iw = iw0 + kw;
            const bool in = image != nullptr && (unsigned)ih < (unsigned)img_h && (unsigned)iw < (unsigned)img_w;
            const float *p = in ? image + (cb * 32 * xs_c + ih * a.xs_h + iw) : &ft_zero;
            const long long next = in ? xs_c : 0;
            if (cb * 32 + 32 <= channels) {
#pragma unroll
                for (int j = 0; j < 32; ++j, p += next) x[j] = __ldg(p);
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j, p += next) x[j] = cb * 32 + j < channels ? __ldg(p) : 0.f;
            }
            advance(); advance();
        };
        if (PLANES) {
            at_tile();
            if (warp >= 8) advance();
        }
        if (PLANES && (warp < 8 ? 0 : 1) < count) fetch();
        for (long long it = warp < 8 ? 0 : 1; it < count; it += 2) {
            const int stage = (int)it & (FT_STAGES - 1), slot = (int)it & (SLOTS - 1);
            if (!mbar_wait(full0 + 8 * stage, (uint32_t)(it / FT_STAGES) & 1, abort_flag, status, FT_WAIT_FULL, 0, limit)) break;
            const uint8_t *row = smem_raw + stage * STAGE + m * 128;
            const uint32_t dst = tmem_base + lane_base + slot * FT_SLOT;
            if (!PLANES) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float4 f = *reinterpret_cast<const float4 *>(row + ((q ^ q_xor) << 4));
                    x[4 * q] = f.x; x[4 * q + 1] = f.y; x[4 * q + 2] = f.z; x[4 * q + 3] = f.w;
                }
            }
            uint32_t part[3][16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                least = __vimin3_u32(least, 2u * __float_as_uint(x[2 * j]) - 1u, 2u * __float_as_uint(x[2 * j + 1]) - 1u);
                part[0][j] = take_bf16(x[2 * j], x[2 * j + 1]);
                part[1][j] = take_bf16(x[2 * j], x[2 * j + 1]);
            }
            if (!mbar_wait(split_empty0 + 8 * slot, ((uint32_t)(it / SLOTS) & 1) ^ 1, abort_flag, status, FT_WAIT_SPLIT, 0, limit)) break;
            tc_fence_after();
            tmem_st16(dst, part[0]);
            tmem_st16(dst + 16, part[1]);
#pragma unroll
            for (int j = 0; j < 16; ++j) part[2][j] = take_bf16(x[2 * j], x[2 * j + 1]);   // here for the registers
            tmem_st16(dst + 32, part[2]);
            if ((left -= 2) <= 0) {
                const uint32_t rows = __ballot_sync(0xffffffffu, least < bound);
                if (lane == 0) *(volatile uint32_t *)&sh->tiny[parity][warp < 8 ? 0 : 1][warp & 3] = rows;
                least = ~0u;
                left += steps;
                parity ^= 1;
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(split0 + 8 * slot);
            if (PLANES && it + 2 < count) fetch();
        }
    } else {
        // ---------------- sums and epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(FT_REGS_SUM));
        const int half = warp < 16 ? 0 : 1, col0 = half * COLS;
        const int quarter = warp & 3, m = quarter * 32 + lane;
        uint8_t *const staged = smem_raw + FT_STAGES * STAGE + half * 128 * ROW;
        int acc = 0;
        uint32_t acc_phase = 0, small_phase = 0, parity = 0;
        bool ok = true, stored = false;
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
            float sum[COLS];
#pragma unroll
            for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
            auto add_up = [&](int which, uint32_t parity) {
                if (!mbar_wait(acc_full0 + 8 * which, parity, abort_flag, status, FT_WAIT_ACC_FULL, 0, limit)) return false;
                tc_fence_after();
                const uint32_t src = acc0 + which * BN + col0 + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
                for (int c = 0; c < COLS; c += LD) {
                    uint32_t r[LD];
#pragma unroll
                    for (int u = 0; u < LD; u += 16) tmem_ld16(src + c + u, *reinterpret_cast<uint32_t(*)[16]>(&r[u]));
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < LD; ++j) sum[c + j] += __uint_as_float(r[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty0 + 8 * which);
                return true;
            };
            for (int step = 0; step < steps && ok; ) {
                const int end = min(steps, step + FT_RUN);
                for (; step < end && ok; ++step) {
                    ok = add_up(acc, acc_phase);
                    acc ^= 1;
                    if (!acc) acc_phase ^= 1;
                }
                if (ok) ok = add_up(2, small_phase);
                small_phase ^= 1;
            }
            if (!meet(half, ok && !*abort_flag)) break;
            float all = 0.f;                                    // NaN where a sum is infinite or NaN
#pragma unroll
            for (int j = 0; j < COLS; ++j) all = fmaf(sum[j], 0.f, all);
            const uint32_t rows = *(volatile uint32_t *)&sh->tiny[parity][0][quarter] | *(volatile uint32_t *)&sh->tiny[parity][1][quarter];
            parity ^= 1;
            const FtTile at(a, tile, BN, col0, m);
            const bool odd = at.inside && (all != 0.f || (rows >> lane & 1u));
            if (meet(half, !odd)) finish_tile<BN, ACT>(a, at, sum, staged, half, m, stored);
            else {
                float again[COLS];
#pragma unroll
                for (int j = 0; j < COLS; ++j) again[j] = odd ? 0.f : sum[j];
                odd_tile<BN, ACT>(a, again, staged, odd, half, tile, m, stored);
            }
            stored = true;
        }
        if (quarter == 0 && lane == 0) tma_store_wait_all();
    }

    // ---------------- teardown (also the abort path)
    if (*abort_flag) {   // give loads that are still in flight time to land before shared memory is released
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000LL) { }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)FT_TMEM) : "memory");
    }
}

template <int BN, int ACT, bool PLANES>
int launch_one(const Fp32TcArgs &a, cudaStream_t s)
{
    // The launch asks for no more shared memory than it uses, unlike the other kernels with TMEM (tmem_smem): its 61440 registers already
    // keep every kernel that allocates columns off its SM.
    static_assert(FT_THREADS * 96 + 128 * 40 > 65536, "no other CTA of four warps beside it");
    const size_t smem = FT_STAGES * (size_t)((PLANES ? 0 : FT_A_BYTES) + 3 * BN * 64) + 2 * 128 * (BN < 64 ? 64 : 128) + sizeof(FtShared);
    DNB_CUDA(cudaFuncSetAttribute(conv_fp32_tc_kernel<BN, ACT, PLANES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    DNB_CUDA(cudaFuncSetAttribute(conv_fp32_tc_kernel<BN, ACT, PLANES>, cudaFuncAttributePreferredSharedMemoryCarveout, (int)((smem + 1024) * 100 / (228 * 1024) + 1)));
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(a.total_tiles < sm_count() ? a.total_tiles : sm_count()));
    cfg.blockDim = dim3(FT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    DNB_CUDA(cudaLaunchKernelEx(&cfg, conv_fp32_tc_kernel<BN, ACT, PLANES>, a));
    DNB_LAUNCH_CHECK("conv_fp32_tc");
    return DNB_OK;
}

template <int BN, bool PLANES>
int launch_act(const Fp32TcArgs &a, cudaStream_t s)
{
    switch (a.ep.activation) {
    case DNB_LINEAR: return launch_one<BN, DNB_LINEAR, PLANES>(a, s);
    case DNB_LEAKY: return launch_one<BN, DNB_LEAKY, PLANES>(a, s);
    default: return launch_one<BN, -1, PLANES>(a, s);
    }
}

template <int BN>
int launch_bn(const Fp32TcArgs &a, cudaStream_t s)
{
    return a.planes ? launch_act<BN, true>(a, s) : launch_act<BN, false>(a, s);
}

}  // namespace

int launch_conv_fp32_tc(const Fp32TcArgs &a, cudaStream_t s)
{
    switch (a.bn) {
    case 32: return launch_bn<32>(a, s);
    case 64: return launch_bn<64>(a, s);
    default: return launch_bn<128>(a, s);
    }
}

}  // namespace dnb
