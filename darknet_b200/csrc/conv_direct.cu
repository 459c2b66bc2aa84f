// Direct convolution on the CUDA cores (fp32 FMA, fp32 accumulate): a general kernel (any filter size, narrow groups), a
// tiled GEMM for 1x1 and 3x3 filters with more than 16 filters per group, and a first-layer specialisation.
//
// Used where the tensor-core kernel does not apply: very narrow inputs (the
// 3-channel first layer, which it reads straight from Darknet's NCHW input),
// grouped convolutions, and DNB_MODE_FP32 networks.
//
// General kernel: a block owns 128 consecutive output pixels and a slab of FB filters; a
// thread owns one pixel and all filters of the slab.  The slab's weights are
// staged through shared memory in K chunks together with a (c,kh,kw) table, so
// the inner loop is one predicated, warp-coalesced load of x and 32 FMAs fed by
// broadcast 16-byte shared loads.  Accumulation runs over
// k = c*size*size + kh*size + kw in increasing order, the reference's own order
// (src/im2col.c:25-28, src/gemm.c:81-87).  Results go through a shared tile so
// that the global stores are 16-byte and contiguous across the warp in either
// output layout (a pixel's channel run for NHWC, a filter's pixel run for NCHW).
#include "common.h"
#include "conv.h"
#include "device_utils.cuh"
#include "tc_ptx.cuh"

namespace dnb {

constexpr int FB = 32;         // filters per thread / per block slab (the general kernel also has narrower slabs)
constexpr int KCHUNK = 192;    // taps staged per pass: 192 * (32*4 + 4) B = 25 KB
constexpr int DTHREADS = 128;  // pixels per block

// FB: filters per slab, 4 to 32: a grouped layer with few filters per group would spend most of a wide slab's FMAs on
// filters that do not exist.
template <typename TX, typename TY, int FB>
__global__ void __launch_bounds__(DTHREADS)
conv_direct_kernel(const __grid_constant__ DirectArgs a)
{
    grid_dependency_wait();
    launch_dependents_if_small();
    __shared__ __align__(16) float w_s[KCHUNK][FB];
    __shared__ int tap_s[KCHUNK];
    __shared__ __align__(16) float out_s[DTHREADS][FB + 4];   // +4 floats: rows stay 16-byte aligned, banks spread

    const ConvGeom &g = a.g;
    const int cpg = g.c / g.groups;           // input channels per group
    const int npg = g.n / g.groups;           // filters per group
    const int fblocks_per_group = (npg + FB - 1) / FB;
    const int grp = blockIdx.y / fblocks_per_group;
    const int f0 = (blockIdx.y % fblocks_per_group) * FB;   // first filter within the group
    const int K = cpg * g.size * g.size;
    const int ksq = g.size * g.size;

    const long long npix = (long long)g.batch * g.out_h * g.out_w;
    const long long pix0 = (long long)blockIdx.x * DTHREADS;
    const long long pix = pix0 + threadIdx.x;
    const bool live = pix < npix;
    int b = 0, oh = 0, ow = 0;
    if (live) {
        ow = (int)(pix % g.out_w);
        long long t = pix / g.out_w;
        oh = (int)(t % g.out_h);
        b = (int)(t / g.out_h);
    }
    const int ih0 = oh * g.stride - g.pad, iw0 = ow * g.stride - g.pad;
    const TX *xb = reinterpret_cast<const TX *>(a.x) + b * a.xs_b + (long long)grp * cpg * a.xs_c;

    float acc[FB];
#pragma unroll
    for (int j = 0; j < FB; ++j) acc[j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += KCHUNK) {
        const int kn = min(KCHUNK, K - k0);
        __syncthreads();
        // weights of this slab: packed [group][k][npg_pad], npg_pad a multiple of FB
        for (int i = threadIdx.x; i < kn * FB; i += DTHREADS) {
            int kk = i / FB, j = i % FB;
            w_s[kk][j] = __ldg(a.wpk + ((size_t)grp * K + k0 + kk) * a.npg_pad + f0 + j);
        }
        for (int kk = threadIdx.x; kk < kn; kk += DTHREADS) {
            int k = k0 + kk, c = k / ksq, r = k - c * ksq, kh = r / g.size, kw = r - kh * g.size;
            tap_s[kk] = (c << 8) | (kh << 4) | kw;
        }
        __syncthreads();
        if (live) {
#pragma unroll 4
            for (int kk = 0; kk < kn; ++kk) {   // four taps' loads in flight
                const int t = tap_s[kk];
                const int c = t >> 8, ih = ih0 + ((t >> 4) & 15), iw = iw0 + (t & 15);
                float xv = 0.f;
                if (ih >= 0 && ih < g.h && iw >= 0 && iw < g.w)
                    xv = to_float<TX>(xb[c * a.xs_c + ih * a.xs_h + iw * a.xs_w]);
                const float4 *wr = reinterpret_cast<const float4 *>(w_s[kk]);
#pragma unroll
                for (int q = 0; q < FB / 4; ++q) {
                    float4 w4 = wr[q];
                    acc[4 * q + 0] = fmaf(xv, w4.x, acc[4 * q + 0]);
                    acc[4 * q + 1] = fmaf(xv, w4.y, acc[4 * q + 1]);
                    acc[4 * q + 2] = fmaf(xv, w4.z, acc[4 * q + 2]);
                    acc[4 * q + 3] = fmaf(xv, w4.w, acc[4 * q + 3]);
                }
            }
        }
    }

    // Epilogue: folded batchnorm / bias, activation, into the shared tile.
    const int n0 = grp * npg + f0;  // first global filter of this slab
#pragma unroll
    for (int j = 0; j < FB; ++j) {
        float v = 0.f;
        if (f0 + j < npg) {
            v = acc[j] * __ldg(a.ep.scale + n0 + j) + __ldg(a.ep.shift + n0 + j);
            v = activate_fast(v, a.ep.activation);
            if (a.ep.round_tf32) v = round_tf32(v);
        }
        out_s[threadIdx.x][j] = v;
    }
    __syncthreads();
    const int live_pix = (int)min((long long)DTHREADS, npix - pix0);
    const int nvalid = min(FB, npg - f0);                  // filters of this slab that exist

    if (a.y_nhwc) {
        // Channels [n0, n0 + cols) of every pixel; the last slab of the last group also writes the zero
        // padding up to cpitch.  16-byte pieces, consecutive threads -> consecutive pieces of a pixel.
        const bool last = grp == g.groups - 1 && f0 + FB >= npg;
        const int cols = last ? min(FB, a.y_cpitch - n0) : nvalid;
        constexpr int EPV = 16 / sizeof(TY);               // elements per 16-byte piece
        if (cols % EPV == 0 && n0 % EPV == 0) {
            const int pieces = cols / EPV;
            TY *base = reinterpret_cast<TY *>(a.y_nhwc) + (size_t)pix0 * a.y_cpitch + n0;
            for (int i = threadIdx.x; i < live_pix * pieces; i += DTHREADS) {
                const int p = i / pieces, q = i - p * pieces;
                const float *src = &out_s[p][q * EPV];
                if (sizeof(TY) == 4) {
                    *reinterpret_cast<float4 *>(base + (size_t)p * a.y_cpitch + q * EPV) = *reinterpret_cast<const float4 *>(src);
                } else {
                    __align__(16) __nv_bfloat16 h[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) h[e] = __float2bfloat16_rn(src[e]);
                    *reinterpret_cast<uint4 *>(base + (size_t)p * a.y_cpitch + q * EPV) = *reinterpret_cast<uint4 *>(h);
                }
            }
        } else {
            TY *base = reinterpret_cast<TY *>(a.y_nhwc) + (size_t)pix0 * a.y_cpitch + n0;
            for (int i = threadIdx.x; i < live_pix * cols; i += DTHREADS) {
                const int p = i / cols, j = i - p * cols;
                base[(size_t)p * a.y_cpitch + j] = from_float<TY>(out_s[p][j]);
            }
        }
        // padding channels that the last slab does not reach
        if (last)
            for (int ch = n0 + cols; ch < min(a.y_cpitch, (g.n + 7) & ~7); ++ch)
                if (live) reinterpret_cast<TY *>(a.y_nhwc)[(size_t)pix * a.y_cpitch + ch] = from_float<TY>(0.f);
    }
    if (a.y_nchw && live) {
        const size_t plane = (size_t)g.out_h * g.out_w;
        float *dst = a.y_nchw + ((size_t)b * g.n + n0) * plane + (size_t)oh * g.out_w + ow;
        for (int j = 0; j < nvalid; ++j) dst[j * plane] = out_s[threadIdx.x][j];
    }
}

// ------------------------------------------------------------------ tiled fp32 GEMM (1x1 and 3x3 filters)
// What bounds it is FMA issue and the 128 bytes per clock that shared memory returns to registers.  The
// one-pixel-per-thread kernel above issues a load, its bounds tests and eight shared loads for every 32 FMAs and shares no
// input value between threads.  Here a block multiplies BM pixels by BN filters from shared memory and a thread keeps
// TM pixels x TN filters, two pixels to a packed fma.rn.f32x2 (the halves are independent IEEE fp32 FMAs): with 16 x 8 a
// thread reads 96 bytes for 128 FMAs, under the one byte per FMA at which the two limits meet (8 x 8 with the weights
// stored twice, as an operand pair, read 96 bytes for 64 and ran at 0.6 of this rate: LSU wavefronts 69 % under ncu).
// A chunk of K is CPC channels x the taps of one filter row (VEC) or of all rows: every load's tap is a compile-time
// constant, its bounds test one bit of a mask built once per thread.
//   VEC false (NCHW, or channels-last tensors whose groups start off a 4-channel boundary): values go from global to
//     shared memory with 4-byte cp.async, coalesced along the pixels of an NCHW row, three chunks in rotation.
//   VEC true (channels-last): 4 channels of a pixel per load, through registers (the tile is channel-major in shared
//     memory), two chunks in rotation.
__device__ __forceinline__ void ffma2(unsigned long long &d, unsigned long long a, unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long twice(float v)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src, bool in)   // zero where !in: the source is then not read
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 4 : 0) : "memory");
}

// KS: 1 or 3.  (BM / TM) * (BN / TN) threads.
template <typename TX, typename TY, int KS, int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), TM == 16 ? 4 : 7)
conv_fp32_gemm_kernel(const __grid_constant__ DirectArgs a)
{
    grid_dependency_wait();
    launch_dependents_if_small();
    constexpr int THREADS = (BM / TM) * (BN / TN);
    static_assert(THREADS == 64 && (BM / TM == 8 || BM / TM == 16), "two warps, 8 x 4 threads each");
    static_assert(VEC || sizeof(TX) == 4, "cp.async copies f32 values");
    constexpr int NPX = BM > THREADS ? BM / THREADS : 1;        // pixels whose values a thread fetches
    constexpr int TPP = THREADS > BM ? THREADS / BM : 1;        // threads that share a pixel's values, by channel
    constexpr int ROWS = VEC ? KS : 1;                          // chunks per channel block: one per filter row, or one
    constexpr int TAPS = VEC ? KS : KS * KS;                    // taps per chunk
    constexpr int CPC = KS == 1 ? (VEC ? 8 : 16) : (VEC ? 4 * TPP : 2);   // channels per chunk
    constexpr int CPT = CPC / TPP;                              // ... that one thread fetches per pixel
    constexpr int KC = CPC * TAPS;
    constexpr int NST = VEC ? 2 : 3;
    constexpr int BV = (KC * BN / 4 + THREADS - 1) / THREADS;
    __shared__ __align__(16) float a_s[NST][KC][BM];
    __shared__ __align__(16) float b_s[NST][KC][BN];

    const ConvGeom &g = a.g;
    const int cpg = g.c / g.groups, npg = g.n / g.groups;
    const int fblocks = (npg + BN - 1) / BN;
    const int grp = blockIdx.y / fblocks, f0 = (blockIdx.y - grp * fblocks) * BN;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long npix = (long long)g.batch * g.out_h * g.out_w;
    const long long pix0 = (long long)blockIdx.x * BM;
    const int csub = TPP > 1 ? (tid / BM) * CPT : 0;            // this thread's first channel of a chunk

    const TX *xp[NPX];
    uint32_t in_mask[NPX];
#pragma unroll
    for (int u = 0; u < NPX; ++u) {
        const long long pix = pix0 + tid % BM + u * THREADS;
        int b = 0, oh = 0, ow = 0;
        if (pix < npix) {
            ow = (int)(pix % g.out_w);
            const long long t = pix / g.out_w;
            oh = (int)(t % g.out_h);
            b = (int)(t / g.out_h);
        }
        const int ih0 = oh * g.stride - g.pad, iw0 = ow * g.stride - g.pad;
        xp[u] = reinterpret_cast<const TX *>(a.x) + b * a.xs_b + (long long)(grp * cpg + csub) * a.xs_c + (long long)ih0 * a.xs_h + (long long)iw0 * a.xs_w;
        uint32_t m = 0;
#pragma unroll
        for (int t = 0; t < KS * KS; ++t)
            if (pix < npix && (unsigned)(ih0 + t / KS) < (unsigned)g.h && (unsigned)(iw0 + t % KS) < (unsigned)g.w) m |= 1u << t;
        in_mask[u] = m;
    }
    int off[TAPS];
#pragma unroll
    for (int t = 0; t < TAPS; ++t) off[t] = (int)((t / KS) * a.xs_h + (t % KS) * a.xs_w);
    const float *wp = a.wpk + (size_t)grp * cpg * (KS * KS) * a.npg_pad + f0;
    const int n_chunks = (cpg + CPC - 1) / CPC * ROWS;

    // weights of chunk ch: row kk of the chunk is (channel c0 + kk / TAPS, tap kk % TAPS of the chunk's taps)
    auto fetch_b = [&](int ch, int st) {
        const int c0 = ch / ROWS * CPC, kh = ROWS > 1 ? ch % ROWS : 0;
#pragma unroll
        for (int v = 0; v < BV; ++v) {
            const int i = tid + v * THREADS, kk = i / (BN / 4), q = i - kk * (BN / 4), c = c0 + kk / TAPS;
            if (KC * BN / 4 % THREADS == 0 || i < KC * BN / 4) {
                // npg_pad is a multiple of 32: four filters lie inside the packed row or beyond it together
                const bool in = c < cpg && f0 + 4 * q < a.npg_pad;
                cp_async16(smem_u32(&b_s[st][kk][4 * q]), in ? wp + ((size_t)c * (KS * KS) + kh * KS + kk % TAPS) * a.npg_pad + 4 * q : a.wpk, in);
            }
        }
    };
    auto fetch_a = [&](int ch, int st) {      // VEC false
        const int c0 = ch * CPC;
#pragma unroll
        for (int u = 0; u < NPX; ++u)
#pragma unroll
            for (int c = 0; c < CPT; ++c) {
                const TX *p = xp[u] + (long long)(c0 + c) * a.xs_c;
                const uint32_t m = c0 + csub + c < cpg ? in_mask[u] : 0u;
#pragma unroll
                for (int t = 0; t < TAPS; ++t) {
                    const bool in = (m >> t) & 1u;
                    cp_async4(&a_s[st][(csub + c) * TAPS + t][tid % BM + u * THREADS], in ? p + off[t] : reinterpret_cast<const TX *>(a.x), in);
                }
            }
    };
    uint4 av[VEC ? NPX : 1][VEC ? TAPS * CPT / 4 : 1];          // VEC true: 4 channels of a pixel each (bf16: in the first two words)
    auto load_a = [&](int ch) {
        const int c0 = ch / ROWS * CPC, kh = ROWS > 1 ? ch % ROWS : 0;
#pragma unroll
        for (int u = 0; u < NPX; ++u) {
            const TX *p = xp[u] + c0 + (long long)kh * a.xs_h;
            const uint32_t m = in_mask[u] >> (kh * KS);
#pragma unroll
            for (int v = 0; v < CPT / 4; ++v)
#pragma unroll
                for (int t = 0; t < TAPS; ++t) {
                    // channels beyond the group's meet zero weights; 4-channel pieces never leave the pixel's pitch (a multiple of 8)
                    const bool in = ((m >> t) & 1u) && c0 + csub + 4 * v < cpg;
                    uint4 r = make_uint4(0u, 0u, 0u, 0u);
                    if (in) {
                        if (sizeof(TX) == 4) r = __ldg(reinterpret_cast<const uint4 *>(p + off[t] + 4 * v));
                        else { const uint2 h = __ldg(reinterpret_cast<const uint2 *>(p + off[t] + 4 * v)); r.x = h.x; r.y = h.y; }
                    }
                    av[u][v * TAPS + t] = r;
                }
        }
    };
    auto put_a = [&](int st) {
#pragma unroll
        for (int u = 0; u < NPX; ++u)
#pragma unroll
            for (int v = 0; v < CPT / 4; ++v)
#pragma unroll
                for (int t = 0; t < TAPS; ++t) {
                    const uint4 r = av[u][v * TAPS + t];
                    float f[4];
                    if (sizeof(TX) == 4) { f[0] = __uint_as_float(r.x); f[1] = __uint_as_float(r.y); f[2] = __uint_as_float(r.z); f[3] = __uint_as_float(r.w); }
                    else { f[0] = __uint_as_float(r.x << 16); f[1] = __uint_as_float(r.x & 0xffff0000u); f[2] = __uint_as_float(r.y << 16); f[3] = __uint_as_float(r.y & 0xffff0000u); }
#pragma unroll
                    for (int e = 0; e < 4; ++e) a_s[st][(csub + 4 * v + e) * TAPS + t][tid % BM + u * THREADS] = f[e];
                }
    };

    // what this thread multiplies: pixel quads q * PSTEP + 4*tx, filter quads h * FSTEP + 4*ty
    constexpr int PQ = TM / 4, FQ = TN / 4, PSTEP = BM / PQ, FSTEP = BN / FQ;
    const int tx = BM / TM == 8 ? (lane & 7) : warp * 8 + (lane & 7), ty = BM / TM == 8 ? warp * 4 + (lane >> 3) : lane >> 3;
    unsigned long long acc[TN][TM / 2];
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int i = 0; i < TM / 2; ++i) acc[j][i] = 0ull;
    auto multiply = [&](int st) {
#pragma unroll
        for (int k = 0; k < KC; ++k) {
            unsigned long long aa[TM / 2];
            float bb[TN];
#pragma unroll
            for (int q = 0; q < PQ; ++q) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(&a_s[st][k][q * PSTEP + 4 * tx]);
                aa[2 * q] = v.x; aa[2 * q + 1] = v.y;
            }
#pragma unroll
            for (int h = 0; h < FQ; ++h) {
                const float4 v = *reinterpret_cast<const float4 *>(&b_s[st][k][h * FSTEP + 4 * ty]);
                bb[4 * h] = v.x; bb[4 * h + 1] = v.y; bb[4 * h + 2] = v.z; bb[4 * h + 3] = v.w;
            }
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const unsigned long long b2 = twice(bb[j]);
#pragma unroll
                for (int i = 0; i < TM / 2; ++i) ffma2(acc[j][i], aa[i], b2);
            }
        }
    };
    if (VEC) {
        load_a(0);
        fetch_b(0, 0);
        cp_async_commit();
        put_a(0);
        cp_async_wait<0>();
        __syncthreads();
        for (int ch = 0; ch < n_chunks; ++ch) {
            const bool more = ch + 1 < n_chunks;
            if (more) { load_a(ch + 1); fetch_b(ch + 1, (ch + 1) & 1); }
            cp_async_commit();
            multiply(ch & 1);
            if (more) put_a((ch + 1) & 1);
            cp_async_wait<0>();
            __syncthreads();
        }
    } else {
        fetch_a(0, 0); fetch_b(0, 0); cp_async_commit();
        if (n_chunks > 1) { fetch_a(1, 1); fetch_b(1, 1); }
        cp_async_commit();
        int st = 0, st2 = 2;
        for (int ch = 0; ch < n_chunks; ++ch) {
            cp_async_wait<1>();
            __syncthreads();              // chunk ch has landed for everybody, and everybody is done with the buffer of chunk ch - 1
            if (ch + 2 < n_chunks) { fetch_a(ch + 2, st2); fetch_b(ch + 2, st2); }
            cp_async_commit();
            multiply(st);
            st = st == 2 ? 0 : st + 1;
            st2 = st2 == 2 ? 0 : st2 + 1;
        }
        cp_async_wait<0>();
    }

    // folded batchnorm / bias, activation, stores straight from the registers, one filter quad at a time
    const int n0 = grp * npg + f0;
    const int nvalid = npg - f0;                            // filters of this block that exist, at least one
    const int pad_end = min(a.y_cpitch, (g.n + 7) & ~7);
    const bool last = grp == g.groups - 1 && f0 + BN >= npg;
    const int cols = last ? min(BN, a.y_cpitch - n0) : min(BN, nvalid);   // the last block of the last group also writes the zero padding channels
    if (a.y_nhwc && last && n0 + cols < pad_end)            // those that its columns do not reach
        for (int i = tid; i < BM; i += THREADS)
            for (int ch = n0 + cols; ch < pad_end; ++ch)
                if (pix0 + i < npix) reinterpret_cast<TY *>(a.y_nhwc)[(size_t)(pix0 + i) * a.y_cpitch + ch] = from_float<TY>(0.f);
    const bool whole_c = n0 % 4 == 0;                       // 4-channel pieces start aligned (the pitch is a multiple of 8)
    const int plane = g.out_h * g.out_w;
    const bool whole_p = plane % 4 == 0;                    // a pixel quad then lies in one plane, 16-byte aligned
#pragma unroll
    for (int h = 0; h < FQ; ++h) {
        const int f = h * FSTEP + 4 * ty;
        float sc[4], sh[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const bool real = f + e < nvalid;
            sc[e] = real ? __ldg(a.ep.scale + n0 + f + e) : 0.f;
            sh[e] = real ? __ldg(a.ep.shift + n0 + f + e) : 0.f;
        }
#pragma unroll
        for (int q = 0; q < PQ; ++q) {
            float v[4][4];   // [pixel][filter]
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const unsigned long long pair = acc[4 * h + e][2 * q + p / 2];
                    float t = __uint_as_float((uint32_t)(p & 1 ? pair >> 32 : pair));
                    t = activate_fast(t * sc[e] + sh[e], a.ep.activation);
                    if (a.ep.round_tf32) t = round_tf32(t);
                    v[p][e] = f + e < nvalid ? t : 0.f;
                }
            const long long pix = pix0 + q * PSTEP + 4 * tx;
            if (a.y_nhwc) {
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    if (pix + p >= npix) continue;
                    TY *row = reinterpret_cast<TY *>(a.y_nhwc) + (size_t)(pix + p) * a.y_cpitch + n0;
                    if (whole_c && f + 4 <= cols) {
                        if (sizeof(TY) == 4) {
                            *reinterpret_cast<float4 *>(row + f) = make_float4(v[p][0], v[p][1], v[p][2], v[p][3]);
                        } else {
                            __nv_bfloat162 lo = __floats2bfloat162_rn(v[p][0], v[p][1]), hi = __floats2bfloat162_rn(v[p][2], v[p][3]);
                            *reinterpret_cast<uint2 *>(row + f) = make_uint2(*reinterpret_cast<uint32_t *>(&lo), *reinterpret_cast<uint32_t *>(&hi));
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (f + e < cols) row[f + e] = from_float<TY>(v[p][e]);
                    }
                }
            }
            if (a.y_nchw) {
                if (whole_p) {
                    if (pix < npix) {
                        const int b = (int)(pix / plane), r = (int)(pix - (long long)b * plane);
                        float *dst = a.y_nchw + ((size_t)b * g.n + n0 + f) * plane + r;
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (f + e < nvalid) *reinterpret_cast<float4 *>(dst + (size_t)e * plane) = make_float4(v[0][e], v[1][e], v[2][e], v[3][e]);
                    }
                } else {
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        if (pix + p >= npix) continue;
                        const int b = (int)((pix + p) / plane), r = (int)(pix + p - (long long)b * plane);
                        float *dst = a.y_nchw + ((size_t)b * g.n + n0 + f) * plane + r;
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (f + e < nvalid) dst[(size_t)e * plane] = v[p][e];
                    }
                }
            }
        }
    }
}

// First-layer specialisation: 3 input channels, 3x3, stride 1, pad 1 (the RGB stems of YOLOv3,
// YOLOv3-tiny and Darknet-19).  Everything is compile-time, so the 36 input values of a thread's two
// neighbouring output pixels are loaded up front (independent loads in flight instead of one
// load-use chain per tap) and every broadcast weight load feeds two FMAs.  256 pixels per block, results
// stored straight from registers.
constexpr int SPIX = 2;                       // output pixels per thread, adjacent in x
constexpr int STHREADS = 128;

template <typename TX, typename TY>
__global__ void __launch_bounds__(STHREADS)
conv_stem3x3_kernel(DirectArgs a)
{
    grid_dependency_wait();
    launch_dependents_if_small();
    __shared__ __align__(16) float w_s[27][FB];

    const ConvGeom g = a.g;
    const int f0 = blockIdx.y * FB;
    for (int i = threadIdx.x; i < 27 * FB; i += STHREADS) w_s[i / FB][i % FB] = __ldg(a.wpk + (size_t)(i / FB) * a.npg_pad + f0 + (i % FB));

    // pixel pairs never straddle a row: out_w is padded to even per row by the launcher's grid math
    const int pairs_per_row = (g.out_w + 1) / 2;
    const unsigned npairs = (unsigned)g.batch * g.out_h * pairs_per_row;   // < 2^31, checked by the launcher
    const unsigned pair = blockIdx.x * STHREADS + threadIdx.x;
    const bool live = pair < npairs;
    int b = 0, oh = 0, ow = 0;
    if (live) {
        ow = (int)(pair % pairs_per_row) * 2;
        const unsigned t = pair / pairs_per_row;
        oh = (int)(t % g.out_h);
        b = (int)(t / g.out_h);
    }
    const TX *xb = reinterpret_cast<const TX *>(a.x) + b * a.xs_b;
    float xv[3][3][4];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int ih = oh + r - 1, iw = ow + q - 1;
                const bool in = live && ih >= 0 && ih < g.h && iw >= 0 && iw < g.w;
                xv[c][r][q] = in ? to_float<TX>(xb[c * a.xs_c + ih * a.xs_h + iw * a.xs_w]) : 0.f;
            }
    __syncthreads();

    float acc0[FB], acc1[FB];
#pragma unroll
    for (int j = 0; j < FB; ++j) { acc0[j] = 0.f; acc1[j] = 0.f; }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const float4 *wr = reinterpret_cast<const float4 *>(w_s[(c * 3 + r) * 3 + q]);
                const float x0 = xv[c][r][q], x1 = xv[c][r][q + 1];
#pragma unroll
                for (int v = 0; v < FB / 4; ++v) {
                    const float4 w4 = wr[v];
                    acc0[4 * v + 0] = fmaf(x0, w4.x, acc0[4 * v + 0]); acc1[4 * v + 0] = fmaf(x1, w4.x, acc1[4 * v + 0]);
                    acc0[4 * v + 1] = fmaf(x0, w4.y, acc0[4 * v + 1]); acc1[4 * v + 1] = fmaf(x1, w4.y, acc1[4 * v + 1]);
                    acc0[4 * v + 2] = fmaf(x0, w4.z, acc0[4 * v + 2]); acc1[4 * v + 2] = fmaf(x1, w4.z, acc1[4 * v + 2]);
                    acc0[4 * v + 3] = fmaf(x0, w4.w, acc0[4 * v + 3]); acc1[4 * v + 3] = fmaf(x1, w4.w, acc1[4 * v + 3]);
                }
            }
    // Epilogue straight from registers: every thread owns whole pixels, so a pixel's 32 channels leave as
    // eight 16-byte stores into one 128-byte line (no shared-memory staging, no index arithmetic).
    const int nvalid = min(FB, g.n - f0);
    const int act = a.ep.activation, rnd = a.ep.round_tf32;
#pragma unroll
    for (int j = 0; j < FB; ++j) {
        float v0 = 0.f, v1 = 0.f;
        if (j < nvalid) {
            const float sc = __ldg(a.ep.scale + f0 + j), sh = __ldg(a.ep.shift + f0 + j);
            v0 = activate_fast(acc0[j] * sc + sh, act);
            v1 = activate_fast(acc1[j] * sc + sh, act);
            if (rnd) { v0 = round_tf32(v0); v1 = round_tf32(v1); }
        }
        acc0[j] = v0;
        acc1[j] = v1;
    }
    if (!live) return;
    const bool second = ow + 1 < g.out_w;
    const size_t pix = ((size_t)b * g.out_h + oh) * g.out_w + ow;
    if (a.y_nhwc) {
        // channels [f0, f0 + cols): the last slab also writes the zero padding up to cpitch
        const int cols = (f0 + FB >= g.n) ? min(FB, a.y_cpitch - f0) : nvalid;
        TY *d0 = reinterpret_cast<TY *>(a.y_nhwc) + pix * a.y_cpitch + f0;
        TY *d1 = d0 + a.y_cpitch;
        if (sizeof(TY) == 4) {
#pragma unroll
            for (int q = 0; q < FB / 4; ++q)
                if (4 * q < cols) {      // cpitch is a multiple of 8: whole pieces
                    reinterpret_cast<float4 *>(d0)[q] = make_float4(acc0[4 * q], acc0[4 * q + 1], acc0[4 * q + 2], acc0[4 * q + 3]);
                    if (second) reinterpret_cast<float4 *>(d1)[q] = make_float4(acc1[4 * q], acc1[4 * q + 1], acc1[4 * q + 2], acc1[4 * q + 3]);
                }
        } else {
#pragma unroll
            for (int q = 0; q < FB / 8; ++q)
                if (8 * q < cols) {
                    uint4 p0, p1;
                    __nv_bfloat162 h;
                    h = __floats2bfloat162_rn(acc0[8 * q], acc0[8 * q + 1]); p0.x = *reinterpret_cast<uint32_t *>(&h);
                    h = __floats2bfloat162_rn(acc0[8 * q + 2], acc0[8 * q + 3]); p0.y = *reinterpret_cast<uint32_t *>(&h);
                    h = __floats2bfloat162_rn(acc0[8 * q + 4], acc0[8 * q + 5]); p0.z = *reinterpret_cast<uint32_t *>(&h);
                    h = __floats2bfloat162_rn(acc0[8 * q + 6], acc0[8 * q + 7]); p0.w = *reinterpret_cast<uint32_t *>(&h);
                    h = __floats2bfloat162_rn(acc1[8 * q], acc1[8 * q + 1]); p1.x = *reinterpret_cast<uint32_t *>(&h);
                    h = __floats2bfloat162_rn(acc1[8 * q + 2], acc1[8 * q + 3]); p1.y = *reinterpret_cast<uint32_t *>(&h);
                    h = __floats2bfloat162_rn(acc1[8 * q + 4], acc1[8 * q + 5]); p1.z = *reinterpret_cast<uint32_t *>(&h);
                    h = __floats2bfloat162_rn(acc1[8 * q + 6], acc1[8 * q + 7]); p1.w = *reinterpret_cast<uint32_t *>(&h);
                    reinterpret_cast<uint4 *>(d0)[q] = p0;
                    if (second) reinterpret_cast<uint4 *>(d1)[q] = p1;
                }
        }
    }
    if (a.y_nchw) {
        const size_t plane = (size_t)g.out_h * g.out_w;
        float *dst = a.y_nchw + ((size_t)b * g.n + f0) * plane + (size_t)oh * g.out_w + ow;
#pragma unroll
        for (int j = 0; j < FB; ++j)
            if (j < nvalid) {
                dst[j * plane] = acc0[j];
                if (second) dst[j * plane + 1] = acc1[j];
            }
    }
}

// Tile of the fp32 GEMM: 16 x 8 per thread where the filters fill 64 columns, 8 x 8 below that, and 32 x 32 tiles of
// 4 x 4 threads where the larger ones would leave SMs empty (fewer than two blocks each): more, shorter blocks then.
template <typename TX, typename TY, int KS, bool VEC>
static int launch_gemm_tile(const DirectArgs &a, cudaStream_t s)
{
    const ConvGeom &g = a.g;
    const long long npix = (long long)g.batch * g.out_h * g.out_w;
    const int npg = g.n / g.groups;
    int bm = 128, bn = npg > 32 ? 64 : 32;
    auto blocks = [&](int m, int n) { return (npix + m - 1) / m * g.groups * ((npg + n - 1) / n); };
    if (blocks(bm, bn) < 2LL * sm_count()) { bm = 32; bn = 32; }
    dim3 grid((unsigned)((npix + bm - 1) / bm), (unsigned)(g.groups * ((npg + bn - 1) / bn)));
    if (grid.y > 65535) DNB_FAIL(DNB_EUNSUPPORTED, "direct conv: too many filter blocks (%u)", grid.y);
    if (bm == 32) DNB_CUDA((launch_overlapped(conv_fp32_gemm_kernel<TX, TY, KS, 32, 32, 4, 4, VEC>, grid, 64, 0, s, a)));
    else if (bn == 64) DNB_CUDA((launch_overlapped(conv_fp32_gemm_kernel<TX, TY, KS, 128, 64, 16, 8, VEC>, grid, 64, 0, s, a)));
    else DNB_CUDA((launch_overlapped(conv_fp32_gemm_kernel<TX, TY, KS, 128, 32, 8, 8, VEC>, grid, 64, 0, s, a)));
    DNB_LAUNCH_CHECK("conv_fp32_gemm");
    return DNB_OK;
}

template <typename TX, typename TY, bool VEC>
static int launch_gemm(const DirectArgs &a, cudaStream_t s)
{
    return a.g.size == 3 ? launch_gemm_tile<TX, TY, 3, VEC>(a, s) : launch_gemm_tile<TX, TY, 1, VEC>(a, s);
}

int launch_conv_direct(const DirectArgs &a, cudaStream_t s)
{
    const ConvGeom &g = a.g;
    if (g.size > 15) DNB_FAIL(DNB_EUNSUPPORTED, "direct conv: kernel size %d > 15", g.size);
    const long long npix = (long long)g.batch * g.out_h * g.out_w;
    const int npg = g.n / g.groups;
    const bool xb = a.x_dtype == DNB_BF16, yb = a.y_dtype == DNB_BF16;
    if (g.c == 3 && g.size == 3 && g.stride == 1 && g.pad == 1 && g.groups == 1 && !xb &&
        (!a.y_nhwc || (a.y_cpitch % 8 == 0))) {
        const long long npairs = (long long)g.batch * g.out_h * ((g.out_w + 1) / 2);
        if (npairs >= (1LL << 31)) DNB_FAIL(DNB_EUNSUPPORTED, "first-layer kernel: %lld pixel pairs", npairs);
        dim3 sgrid((unsigned)((npairs + STHREADS - 1) / STHREADS), (unsigned)((g.n + FB - 1) / FB));
        if (yb) DNB_CUDA((launch_overlapped(conv_stem3x3_kernel<float, __nv_bfloat16>, sgrid, STHREADS, 0, s, a)));
        else DNB_CUDA((launch_overlapped(conv_stem3x3_kernel<float, float>, sgrid, STHREADS, 0, s, a)));
        DNB_LAUNCH_CHECK("conv_stem3x3");
        return DNB_OK;
    }
    // One input and one output type per plan mode: bf16 tensors belong to BF16 plans, which may also read or write f32.
#define DIRECT_TYPES(GO)                                        \
    do {                                                        \
        if (!xb && !yb) GO(float, float);                       \
        else if (!xb && yb) GO(float, __nv_bfloat16);           \
        else if (xb && !yb) GO(__nv_bfloat16, float);           \
        else GO(__nv_bfloat16, __nv_bfloat16);                  \
    } while (0)
    // The tiled kernel wants filters to fill its tile: below 17 per group a slab of the general kernel does less padded work.
    // A 3x3 chunk of its channels-last form holds a few channels of one filter row, so it adds row by row, in steps that depend
    // on the tile; every other form adds in the order c, kh, kw, which is what a layer with signs behind it has to do.
    if (npg > 16 && (g.size == 1 || g.size == 3) && a.xs_h < (1LL << 28) && a.xs_w < (1LL << 28)) {
        const bool vec = a.xs_c == 1 && a.xs_w % 4 == 0 && (g.groups == 1 || (g.c / g.groups) % 4 == 0) && !(a.in_order && g.size == 3);
        if (xb && vec) return yb ? launch_gemm<__nv_bfloat16, __nv_bfloat16, true>(a, s) : launch_gemm<__nv_bfloat16, float, true>(a, s);
        if (!xb && vec) return yb ? launch_gemm<float, __nv_bfloat16, true>(a, s) : launch_gemm<float, float, true>(a, s);
        if (!xb) return yb ? launch_gemm<float, __nv_bfloat16, false>(a, s) : launch_gemm<float, float, false>(a, s);
    }
    const int fb = npg <= 4 ? 4 : npg <= 8 ? 8 : npg <= 16 ? 16 : 32;
    dim3 grid((unsigned)((npix + DTHREADS - 1) / DTHREADS), (unsigned)(g.groups * ((npg + fb - 1) / fb)));
    if (grid.y > 65535) DNB_FAIL(DNB_EUNSUPPORTED, "direct conv: too many filter blocks (%u)", grid.y);
#define SLAB_GO(TX, TY)                                                                       \
    do {                                                                                      \
        if (fb == 4) DNB_CUDA((launch_overlapped(conv_direct_kernel<TX, TY, 4>, grid, DTHREADS, 0, s, a)));              \
        else if (fb == 8) DNB_CUDA((launch_overlapped(conv_direct_kernel<TX, TY, 8>, grid, DTHREADS, 0, s, a)));         \
        else if (fb == 16) DNB_CUDA((launch_overlapped(conv_direct_kernel<TX, TY, 16>, grid, DTHREADS, 0, s, a)));       \
        else DNB_CUDA((launch_overlapped(conv_direct_kernel<TX, TY, 32>, grid, DTHREADS, 0, s, a)));                     \
    } while (0)
    DIRECT_TYPES(SLAB_GO);
#undef SLAB_GO
#undef DIRECT_TYPES
    DNB_LAUNCH_CHECK("conv_direct");
    return DNB_OK;
}

}  // namespace dnb
