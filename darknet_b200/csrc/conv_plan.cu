// Convolution plans: geometry checks, kernel choice, derived parameter tensors
// (folded batchnorm, repacked / rounded / bit-packed weights) and the forward
// dispatch behind dnb_conv_*.
#include <math.h>
#include <stdlib.h>
#include <string.h>
#include <unistd.h>

#include <vector>

#include <cuda_bf16.h>

#include "common.h"
#include "conv.h"

using namespace dnb;

enum { K_TC_TF32 = 0, K_TC_BF16 = 1, K_DIRECT = 2, K_XNOR = 3 };
static const char *const kKernelNames[] = {"tc_tf32", "tc_bf16", "direct_fp32", "xnor_popc"};
static const char kXnorTcName[] = "xnor_tc";

// Layers of full-precision plans that may run as products of three bf16 parts on the tensor cores (conv_fp32_tc.cu): sums of 128 products and
// more, which are less far from 64-bit sums than the CUDA-core kernel's, which rounds at every product.
// Measured as the root mean square of the error over that of the layer, CUDA cores / tensor cores, for K products, in units of 1e-7:
//   K = 128  2.0 / 0.70     K = 144  2.1 / 0.73     K = 576  4.3 / 0.99     K = 2304  8.5 / 1.7     K = 4608  11.4 / 2.2
static bool fp32_tc_covers(const ConvGeom &g)
{
    return g.groups == 1 && g.stride <= 2 && g.c >= 8 && g.c * g.size * g.size >= 128 && (long long)g.batch * g.h * g.w < (1LL << 31);
}

// Bits of the smallest input, but zero, whose products with weights of these sizes (bits) are 2^-90 or more, at least 2^-100; 0 where that would be
// more than 2^-45, or where a weight is infinite, NaN or beyond bf16's largest number: such a layer stays on the CUDA cores.
static uint32_t fp32_tc_smallest_input(uint32_t least, uint32_t most)
{
    if (most >= 0x7f7f8000u) return 0;
    const int e = most ? (int)(least >> 23) - 127 : 0;   // the smallest weight is 2^e or more (no weight but zeros: any input does)
    if (e < -45) return 0;
    const int x = -90 - e < -100 ? -100 : -90 - e;
    return (uint32_t)(x + 127) << 23;
}

// Whether a launch of this plan runs on the tensor cores (after set_params; before it, whether the layer is one for them).
static bool on_fp32_tc(const dnb_conv_plan *p) { return p->fp32_tc && !p->keep_k_order && (!p->params_set || p->fp32_smallest); }

static int fp32_tc_filters(int n) { return n <= 32 ? 32 : n <= 64 ? 64 : 128; }   // of a tile

// Whether they should: for either layout, so that a plan's sums are the same in both.  Microseconds of either kernel, measured on B200: a step of
// 32 channels of a tap takes a tile of 128 filters 1.04 on the tensor cores, of 64 0.75, of 32 0.59; a block of the CUDA-core kernel's large tiles of 64
// filters 64 ns a product where four share an SM, of 32 filters 34 and 50 more, one of its small ones 17.5 and 11.5 more for every other block
// there, its slabs of up to 16 filters 6 a product and filter.  Of 208 launches between 10 us and 1 ms 199 take the faster kernel, or one within 5 %
// of it; the worst choice was 1.2 times the other's time.  8 x 64 x 104 x 104 -> 128, 3x3: 316 -> 104 us, from Darknet's layout 352 -> 113; 32 x 64 x 104 x 104
// -> 64 676 -> 298; 8 x 100 x 38 x 38 -> 70, stride 2, would be 27 -> 42.  DNB_FP32_TC: 0 never, 1 whenever it can.
static bool fp32_tc_pays(const ConvGeom &g)
{
    if (const char *e = getenv("DNB_FP32_TC")) return atoi(e) != 0;
    const double npix = (double)g.batch * g.out_h * g.out_w, K = (double)g.c * g.size * g.size, sms = sm_count();
    const int bn = fp32_tc_filters(g.n);
    const double tiles = ceil(npix / 128) * ceil((double)g.n / bn);
    const double tc = 6 + ceil(tiles / sms) * ((bn == 32 ? 0.59 : bn == 64 ? 0.75 : 1.04) * g.size * g.size * ((g.c + 31) / 32) + 0.012 * bn);
    double direct;
    if (g.n <= 16 || (g.size != 1 && g.size != 3)) {
        const int slab = g.n < 4 ? 4 : g.n > 16 ? 16 : g.n;
        direct = 5 + K * 0.006 * slab * ceil(ceil(npix / 128) * ((g.n + 15) / 16) / sms);
    } else if (ceil(npix / 128) * ceil(g.n / (g.n > 32 ? 64.0 : 32.0)) >= 2 * sms) {
        const double b = ceil(npix / 128) * ceil(g.n / (g.n > 32 ? 64.0 : 32.0)) / sms;
        direct = 6 + K * (g.n <= 32 ? 0.05 + 0.034 * b : b < 4 ? 0.04 + 0.05 * ceil(b) : 0.064 * b);
    }
    else direct = 5 + K * (0.006 + 0.0115 * ceil(ceil(npix / 32) * ceil(g.n / 32.0) / sms));
    return tc < direct;
}

extern "C" int dnb_conv_plan_create(const dnb_conv_desc *d, int mode, dnb_conv_plan **out)
{
    if (!d || !out) DNB_FAIL(DNB_EINVAL, "conv plan: null argument");
    *out = nullptr;
    if (mode != DNB_MODE_TF32 && mode != DNB_MODE_BF16 && mode != DNB_MODE_FP32) DNB_FAIL(DNB_EINVAL, "conv plan: mode %d", mode);
    if (d->batch < 1 || d->h < 1 || d->w < 1 || d->c < 1 || d->n < 1 || d->size < 1 || d->stride < 1 || d->pad < 0 || d->groups < 1)
        DNB_FAIL(DNB_EINVAL, "conv plan: non-positive geometry (batch %d, %dx%dx%d, n %d, size %d, stride %d, pad %d, groups %d)",
                 d->batch, d->c, d->h, d->w, d->n, d->size, d->stride, d->pad, d->groups);
    if (d->c % d->groups || d->n % d->groups) DNB_FAIL(DNB_EINVAL, "conv plan: groups %d does not divide c %d and n %d", d->groups, d->c, d->n);
    if (d->activation < 0 || d->activation > DNB_SELU) DNB_FAIL(DNB_EINVAL, "conv plan: activation %d", d->activation);
    if (d->size > 15) DNB_FAIL(DNB_EUNSUPPORTED, "conv plan: kernel size %d > 15", d->size);
    const int out_h = (d->h + 2 * d->pad - d->size) / d->stride + 1;
    const int out_w = (d->w + 2 * d->pad - d->size) / d->stride + 1;
    if (out_h < 1 || out_w < 1) DNB_FAIL(DNB_EINVAL, "conv plan: empty output (%dx%d)", out_w, out_h);
    if (d->size == 1 && (d->stride != 1 || d->pad != 0))
        DNB_FAIL(DNB_EUNSUPPORTED, "conv plan: 1x1 kernel with stride %d / pad %d: the reference's CPU path skips im2col for size 1 and "
                 "multiplies the unstrided image (src/convolutional_layer.c:468-470), so its result is not a convolution; not reproduced", d->stride, d->pad);
    if (d->xnor && d->groups != 1) DNB_FAIL(DNB_EUNSUPPORTED, "conv plan: xnor with groups %d", d->groups);

    dnb_conv_plan *p = new dnb_conv_plan();
    memset(p, 0, sizeof(*p));
    p->d = *d;
    p->mode = mode;
    p->g = ConvGeom{d->batch, d->h, d->w, d->c, d->n, d->groups, d->size, d->stride, d->pad, out_h, out_w};
    p->n_pad = round_up(d->n, 16);
    p->c_pad = round_up(d->c, 8);
    p->npg_pad = round_up(d->n / d->groups, 32);
    p->cwords = (d->c + 31) / 32;
    p->c_pad_i8 = round_up(d->c, 32);
    if (d->xnor) p->kernel = K_XNOR;
    else if (mode == DNB_MODE_FP32 || d->groups != 1 || d->c < 8) p->kernel = K_DIRECT;
    else p->kernel = mode == DNB_MODE_BF16 ? K_TC_BF16 : K_TC_TF32;
    // the tensor-core kernel reads strided inputs through stride*stride lattices and carries maps for strides 1
    // and 2 only; wider strides (none in the benchmark networks) run on the CUDA-core kernel
    if ((p->kernel == K_TC_TF32 || p->kernel == K_TC_BF16) && d->stride > 2) p->kernel = K_DIRECT;
    // RGB first layers of the TF32 / BF16 modes: tensor cores, rows read from the patch in shared memory (DNB_STEM_TC=0 keeps the FP32 kernel)
    const char *stem_env = getenv("DNB_STEM_TC");
    p->stem_tc = p->kernel == K_DIRECT && mode != DNB_MODE_FP32 && !d->xnor && conv_stem_tc_covers(p->g) && !(stem_env && atoi(stem_env) == 0);
    p->fp32_tc = p->kernel == K_DIRECT && mode == DNB_MODE_FP32 && fp32_tc_covers(p->g) && fp32_tc_pays(p->g);
    // xnor layers: int8 sign tensors through the tensor cores (kind::i8, exact int32 sums) unless DNB_XNOR_TC=0 asks
    // for the bit-packed popcount kernel; strides above 2 have no lattice maps and stay with the popcount kernel
    {
        const char *e = getenv("DNB_XNOR_TC");
        p->xnor_tc = p->kernel == K_XNOR && d->stride <= 2 && !(e && atoi(e) == 0);
    }
    cudaGetDevice(&p->device);
    *out = p;
    return DNB_OK;
}

// The same layer over another batch, with launch blocks and scratch of its own; its parameters are p's, which outlives it and
// is given no new ones meanwhile.
dnb_conv_plan *conv_plan_for_batch(const dnb_conv_plan *p, int batch)
{
    dnb_conv_plan *q = new dnb_conv_plan(*p);
    q->d.batch = q->g.batch = batch;
    q->borrowed = true;
    q->whole_batch = p->g.batch;
    q->x_nhwc_scratch = nullptr; q->x_bits = nullptr; q->x_i8 = nullptr;
    q->x_nhwc_bytes = q->x_bits_bytes = q->x_i8_bytes = 0;
    q->tc_x_ptr = q->tc_y_ptr = q->tc_res_ptr = nullptr;
    q->sign_consumer = nullptr; q->signs_given = false; q->signs_of = nullptr;
    return q;
}

extern "C" void dnb_conv_plan_destroy(dnb_conv_plan *p)
{
    if (!p) return;
    if (p->borrowed) {
        cudaFree(p->x_nhwc_scratch); cudaFree(p->x_bits); cudaFree(p->x_i8);
        delete p;
        return;
    }
    cudaFree(p->scale); cudaFree(p->shift); cudaFree(p->w_tc); cudaFree(p->w_direct); cudaFree(p->w_bits);
    cudaFree(p->w_mean); cudaFree(p->x_nhwc_scratch); cudaFree(p->x_bits); cudaFree(p->w_i8); cudaFree(p->scale_i8); cudaFree(p->x_i8);
    if (!p->status_shared && !p->status_in_block) cudaFree(p->status);
    delete p;
}

extern "C" const char *dnb_conv_plan_kernel(const dnb_conv_plan *p)
{
    if (!p) return "";
    if (p->kernel == K_XNOR && p->xnor_tc) return kXnorTcName;
    return p->stem_tc ? "stem_tc_tf32" : kKernelNames[p->kernel];
}

extern "C" int dnb_conv_plan_describe(const dnb_conv_plan *p, char *buf, int len)
{
    if (!p || !buf || len < 1) DNB_FAIL(DNB_EINVAL, "conv describe: bad argument");
    const TcArgs &a = p->tc;
    const bool tc = p->kernel == K_TC_TF32 || p->kernel == K_TC_BF16 || (p->kernel == K_XNOR && p->xnor_tc);
    if (tc && p->tc_x_ptr && p->tc_split)
        snprintf(buf, len, "%s pair=%d halo=0 bn=%d tile=%dx%dx%d tiles=%d stages=%d splits=%d signs_in=%d signs_out=%d one_tile_per_cluster", kKernelNames[p->kernel], p->sp.pair,
                 p->sp.bn, p->sp.wt, p->sp.ht, p->sp.bt, p->sp.tiles, p->sp.stages, p->sp.splits, p->signs_given ? 1 : 0, p->sp.sign_out ? 1 : 0);
    else if (tc && p->tc_x_ptr && p->tc_taps)
        snprintf(buf, len, "%s pair=1 halo=0 bn=%d tiles=%d stages=%d+%d epi=2 splits=1 one_load_for_%s%s", kKernelNames[p->kernel], p->tp.bn, p->tp.total_tiles,
                 p->tp.x_stages, p->tp.w_stages, p->tp.taps == 9 ? "nine_taps" : "a_block", p->tp.boxes ? (p->tp.resident ? " boxes resident" : " boxes") : p->tp.resident ? " resident" : "");
    else if ((p->kernel == K_TC_TF32 || p->kernel == K_TC_BF16 || (p->kernel == K_XNOR && p->xnor_tc)) && p->tc_x_ptr)
        snprintf(buf, len, "%s pair=%d halo=%d bn=%d tile=%dx%dx%d tiles=%d stages=%d ctas_per_sm=%d srb=%d epi=%d splits=1 signs_in=%d signs_out=%d", kKernelNames[p->kernel], a.pair, a.halo,
                 a.bn, a.wt, a.ht, a.bt, a.total_tiles, a.stages, a.ctas_per_sm, a.store_row_bytes, a.epi_groups, p->signs_given ? 1 : 0, a.sign_out ? 1 : 0);
    else if (on_fp32_tc(p))
        snprintf(buf, len, "%s three_bf16_parts bn=%d", dnb_conv_plan_kernel(p), fp32_tc_filters(p->d.n));
    else
        snprintf(buf, len, "%s", dnb_conv_plan_kernel(p));
    return DNB_OK;
}

static int ensure_status(dnb_conv_plan *p)
{
    if (p->status) return DNB_OK;
    DNB_CUDA(cudaMalloc((void **)&p->status, sizeof(int)));
    DNB_CUDA(cudaMemset(p->status, 0, sizeof(int)));
    return DNB_OK;
}

template <typename T>
static int upload(T **dst, const std::vector<T> &src)
{
    if (*dst) { cudaFree(*dst); *dst = nullptr; }
    DNB_CUDA(cudaMalloc((void **)dst, src.size() * sizeof(T)));
    DNB_CUDA(cudaMemcpy(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice));
    return DNB_OK;
}

// ------------------------------------------------------------------ derived parameter tensors, built on the device
// One host-to-device copy of the layer's weights as Darknet holds them ([n][c/groups][size][size]) and one kernel per
// derived tensor: transposition into the kernels' layouts, rounding to the storage type, sign extraction.
namespace {

// tensor-core layout [tap][n_pad][c_pad], zero where padded; T = float (rounded to TF32-nearest) or bf16
template <typename T>
__global__ void repack_tc_kernel(const float *__restrict__ w, T *__restrict__ out, int n, int c, int taps, int n_pad, int c_pad)
{
    const size_t total = (size_t)taps * n_pad * c_pad;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int cc = (int)(i % c_pad);
        const size_t r = i / c_pad;
        const int f = (int)(r % n_pad), t = (int)(r / n_pad);
        float v = 0.f;
        if (f < n && cc < c) v = __ldg(w + ((size_t)f * c + cc) * taps + t);
        if (sizeof(T) == 4) {
            // nearest TF32, ties away from zero (what cvt.rna.tf32.f32 computes); infinities and NaNs pass through
            uint32_t u = __float_as_uint(v);
            if ((u & 0x7f800000u) != 0x7f800000u) u = (u + 0x1000u) & ~0x1fffu;
            reinterpret_cast<float *>(out)[i] = __uint_as_float(u);
        } else {
            reinterpret_cast<__nv_bfloat16 *>(out)[i] = __float2bfloat16_rn(v);
        }
    }
}

// [c_blocks][taps][3][n_pad][32]: the weights as sums of three bf16 numbers, each the nearest to what the ones before it leave (the last
// one exactly that).  range: the bits of the smallest |weight| but zero, of the largest.  A status word behind them starts at 0.
__global__ void split_weights_kernel(const float *__restrict__ w, __nv_bfloat16 *__restrict__ out, int n, int c, int taps, int n_pad, int c_blocks, uint32_t *range, int *status)
{
    if (status && blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
    uint32_t least = ~0u, most = 0u;
    const size_t part = (size_t)n_pad * 32, total = part * taps * c_blocks;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t step = i / part, r = i - step * part;
        const int cc = (int)(step / taps) * 32 + (int)(r & 31), t = (int)(step % taps), f = (int)(r >> 5);
        float v = f < n && cc < c ? __ldg(w + ((size_t)f * c + cc) * taps + t) : 0.f;
        const uint32_t size = __float_as_uint(v) & 0x7fffffffu;
        if (size && size < least) least = size;
        if (size > most) most = size;
        for (int k = 0; k < 3; ++k) {
            const __nv_bfloat16 h = __float2bfloat16_rn(v);
            out[(3 * step + k) * part + r] = h;
            v -= __bfloat162float(h);
        }
    }
    least = __reduce_min_sync(0xffffffffu, least);
    most = __reduce_max_sync(0xffffffffu, most);
    if ((threadIdx.x & 31) == 0) { atomicMin(range, least); atomicMax(range + 1, most); }
}

// CUDA-core layout [groups][K][npg_pad], K = c/groups * size * size, filters innermost
__global__ void repack_direct_kernel(const float *__restrict__ w, float *__restrict__ out, int groups, int npg, size_t K, int npg_pad)
{
    const size_t total = (size_t)groups * K * npg_pad;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int f = (int)(i % npg_pad);
        const size_t r = i / npg_pad;
        const size_t k = r % K;
        const int g = (int)(r / K);
        out[i] = f < npg ? __ldg(w + ((size_t)(g * npg + f)) * K + k) : 0.f;
    }
}

// xnor: per filter the mean |w|, summed in a float in index order as binarize_weights does (src/convolutional_layer.c:28-41):
// one thread per filter, so the order of the additions is the reference's
__global__ void xnor_mean_kernel(const float *__restrict__ w, float *__restrict__ mean, int n, size_t K)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n) return;
    float acc = 0.f;
    for (size_t k = 0; k < K; ++k) acc += fabsf(__ldg(w + (size_t)f * K + k));
    mean[f] = acc / (float)K;
}

// xnor: sign bits [n][taps][cwords] (bit c % 32 of word c / 32 set where w > 0), one thread per word
__global__ void xnor_bits_kernel(const float *__restrict__ w, uint32_t *__restrict__ bits, int n, int c, int taps, int cwords)
{
    const size_t total = (size_t)n * taps * cwords;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int wd = (int)(i % cwords);
        const size_t r = i / cwords;
        const int t = (int)(r % taps), f = (int)(r / taps);
        uint32_t word = 0;
        for (int k = 0; k < 32; ++k) {
            const int cc = wd * 32 + k;
            if (cc < c && __ldg(w + ((size_t)f * c + cc) * taps + t) > 0.f) word |= 1u << k;
        }
        bits[i] = word;
    }
}

// xnor on the tensor cores: signs as int8 in the tensor-core weight layout [tap][n_pad][c_pad], zero where padded
__global__ void xnor_i8_kernel(const float *__restrict__ w, int8_t *__restrict__ out, int n, int c, int taps, int n_pad, int c_pad)
{
    const size_t total = (size_t)taps * n_pad * c_pad;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int cc = (int)(i % c_pad);
        const size_t r = i / c_pad;
        const int f = (int)(r % n_pad), t = (int)(r / n_pad);
        int8_t v = 0;
        if (f < n && cc < c) v = __ldg(w + ((size_t)f * c + cc) * taps + t) > 0.f ? 1 : -1;
        out[i] = v;
    }
}

// mean|w| folded into the batchnorm scale of the tensor-core xnor kernel
__global__ void scale_times_mean_kernel(const float *__restrict__ scale, const float *__restrict__ mean, float *__restrict__ out, int n, int n_pad)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f < n_pad) out[f] = f < n ? mean[f] * scale[f] : 0.f;
}

int grid_of(size_t total)
{
    const size_t blocks = (total + 255) / 256, cap = (size_t)sm_count() * 16;
    return (int)(blocks < cap ? (blocks ? blocks : 1) : cap);
}

template <typename T>
int device_alloc(T **dst, size_t count)
{
    if (*dst) { cudaFree(*dst); *dst = nullptr; }
    DNB_CUDA(cudaMalloc((void **)dst, count * sizeof(T)));
    return DNB_OK;
}

}  // namespace

extern "C" int dnb_conv_plan_set_params(dnb_conv_plan *p, const float *weights, const float *biases, const float *scales,
                                        const float *mean, const float *var)
{
    if (!p || !weights || !biases) DNB_FAIL(DNB_EINVAL, "conv params: null argument");
    const dnb_conv_desc &d = p->d;
    if (d.batch_normalize && (!scales || !mean || !var)) DNB_FAIL(DNB_EINVAL, "conv params: batch_normalize layer needs scales, rolling_mean, rolling_variance");
    DNB_TRY(check_current_device(p->device, "conv params"));
    const int cpg = d.c / d.groups, npg = d.n / d.groups, taps = d.size * d.size;
    const size_t K = (size_t)cpg * taps, nw = (size_t)d.n * K;

    // Folded inference batchnorm.  The CPU reference computes
    // ((x - mean) / (sqrt(var) + 1e-6f)) * scale + bias (src/blas.c:147-158,
    // src/batchnorm_layer.c:151-154); folded: x*s + (bias - mean*s).
    std::vector<float> s(p->n_pad, 0.f), b(p->n_pad, 0.f);
    for (int n = 0; n < d.n; ++n) {
        if (d.batch_normalize) {
            const double sc = (double)scales[n] / (sqrt((double)var[n]) + (double).000001f);
            s[n] = (float)sc;
            b[n] = (float)((double)biases[n] - (double)mean[n] * sc);
        } else {
            s[n] = 1.f;
            b[n] = biases[n];
        }
    }
    p->params_set = false;   // until all of the tensors are the new ones
    DNB_TRY(upload(&p->scale, s));
    DNB_TRY(upload(&p->shift, b));

    // the weights as Darknet holds them, once; every derived tensor is built from this copy on the device
    float *raw = nullptr;
    DNB_CUDA(cudaMalloc((void **)&raw, nw * sizeof(float)));
    struct Raw { float *p; ~Raw() { cudaFree(p); } } raw_guard{raw};
    DNB_CUDA(cudaMemcpy(raw, weights, nw * sizeof(float), cudaMemcpyHostToDevice));

    if (p->kernel == K_TC_TF32) {
        const size_t total = (size_t)taps * p->n_pad * p->c_pad;
        float *dev = (float *)p->w_tc;
        DNB_TRY(device_alloc(&dev, total));
        p->w_tc = dev;
        repack_tc_kernel<float><<<grid_of(total), 256>>>(raw, dev, d.n, d.c, taps, p->n_pad, p->c_pad);
    } else if (p->kernel == K_TC_BF16) {
        const size_t total = (size_t)taps * p->n_pad * p->c_pad;
        __nv_bfloat16 *dev = (__nv_bfloat16 *)p->w_tc;
        DNB_TRY(device_alloc(&dev, total));
        p->w_tc = dev;
        repack_tc_kernel<__nv_bfloat16><<<grid_of(total), 256>>>(raw, dev, d.n, d.c, taps, p->n_pad, p->c_pad);
    } else if (p->kernel == K_DIRECT) {
        const size_t total = (size_t)d.groups * K * p->npg_pad;
        // one allocation: the CUDA-core kernel's weights, and for the tensor cores their three parts and the status word
        const int c_blocks = (d.c + 31) / 32;
        const size_t first = (total + 63) / 64 * 64, parts = p->fp32_tc && !p->keep_k_order ? (size_t)c_blocks * taps * 3 * p->n_pad * 32 : 0;   // bf16 values
        if (p->status_in_block) { p->status = nullptr; p->status_in_block = false; }
        p->fp32_smallest = 0;
        DNB_TRY(device_alloc(&p->w_direct, parts ? first + parts / 2 + 3 : total));
        repack_direct_kernel<<<grid_of(total), 256>>>(raw, p->w_direct, d.groups, npg, K, p->npg_pad);
        if (parts) {
            p->w_parts = reinterpret_cast<__nv_bfloat16 *>(p->w_direct + first);
            uint32_t *const range = reinterpret_cast<uint32_t *>(p->w_parts + parts);
            int *word = nullptr;
            if (!p->status) { word = p->status = reinterpret_cast<int *>(range + 2); p->status_in_block = true; }
            DNB_CUDA(cudaMemsetAsync(range, 0xff, sizeof(uint32_t)));
            DNB_CUDA(cudaMemsetAsync(range + 1, 0, sizeof(uint32_t)));
            split_weights_kernel<<<grid_of(parts / 3), 256>>>(raw, p->w_parts, d.n, d.c, taps, p->n_pad, c_blocks, range, word);
            uint32_t bits[2];
            DNB_CUDA(cudaMemcpy(bits, range, sizeof(bits), cudaMemcpyDeviceToHost));
            p->fp32_smallest = fp32_tc_smallest_input(bits[0], bits[1]);
        }
    } else {
        DNB_TRY(device_alloc(&p->w_bits, (size_t)d.n * taps * p->cwords));
        DNB_TRY(device_alloc(&p->w_mean, (size_t)d.n));
        xnor_bits_kernel<<<grid_of((size_t)d.n * taps * p->cwords), 256>>>(raw, p->w_bits, d.n, d.c, taps, p->cwords);
        xnor_mean_kernel<<<(d.n + 127) / 128, 128>>>(raw, p->w_mean, d.n, K);
        if (p->xnor_tc) {
            const size_t total = (size_t)taps * p->n_pad * p->c_pad_i8;
            DNB_TRY(device_alloc(&p->w_i8, total));
            DNB_TRY(device_alloc(&p->scale_i8, (size_t)p->n_pad));
            xnor_i8_kernel<<<grid_of(total), 256>>>(raw, p->w_i8, d.n, d.c, taps, p->n_pad, p->c_pad_i8);
            scale_times_mean_kernel<<<(p->n_pad + 127) / 128, 128>>>(p->scale, p->w_mean, p->scale_i8, d.n, p->n_pad);
        }
    }
    DNB_LAUNCH_CHECK("weight repack");
    DNB_CUDA(cudaDeviceSynchronize());   // the staging copy is released on return
    p->params_set = true;
    // The launch block caches a tensor map over the weights just replaced: have the next forward rebuild it.
    p->tc_x_ptr = p->tc_y_ptr = p->tc_res_ptr = nullptr;
    return DNB_OK;
}

// Shortens the bound of the plan's device-side waits (cycles; 0 restores the default of about one second) and
// sets diagnostic bits of the tensor-core kernel.  Bit 32 makes every CTA withhold one operand load, so that a
// wait runs out: the way the time-out path is exercised without faulting the device.
extern "C" int dnb_conv_plan_set_diagnostics(dnb_conv_plan *p, long long wait_limit_cycles, int debug_bits)
{
    if (!p || wait_limit_cycles < 0) DNB_FAIL(DNB_EINVAL, "conv diagnostics: bad argument");
    p->wait_limit = wait_limit_cycles;
    p->debug_bits = debug_bits;
    p->tc_x_ptr = p->tc_y_ptr = p->tc_res_ptr = nullptr;
    return DNB_OK;
}

// ------------------------------------------------------------------ tensor-core launch block
// The tuning knobs of a launch block (DNB_TC_..., null where unset), from one pass over the environment.  A block asks for some of them several times, some 25
// lookups of the whole environment: without them a block of a 1x1 layer takes 4.9 us, 5.5 before (90 variables).
struct Knobs {
    const char *bn = nullptr, *pair = nullptr, *epi = nullptr, *halo = nullptr, *warp_stores = nullptr, *splitk = nullptr, *flat = nullptr, *debug = nullptr, *srb = nullptr,
               *min_stages = nullptr, *ctas = nullptr, *max2 = nullptr, *shortk = nullptr, *stages = nullptr, *taps = nullptr, *taps_bn = nullptr, *taps_box = nullptr;
    Knobs()
    {
        const struct { const char *name, **value; } all[] = {
            {"BN", &bn}, {"PAIR", &pair}, {"EPI", &epi}, {"HALO", &halo}, {"WARP_STORES", &warp_stores}, {"SPLITK", &splitk}, {"FLAT", &flat}, {"DEBUG", &debug}, {"SRB", &srb},
            {"MIN_STAGES", &min_stages}, {"CTAS", &ctas}, {"MAX2", &max2}, {"SHORTK", &shortk}, {"STAGES", &stages}, {"TAPS", &taps}, {"TAPS_BN", &taps_bn}, {"TAPS_BOX", &taps_box}};
        for (char **e = environ; e && *e; ++e) {
            if (strncmp(*e, "DNB_TC_", 7) != 0) continue;
            const char *const name = *e + 7, *const eq = strchr(name, '=');
            if (!eq) continue;
            for (const auto &k : all)
                if (strlen(k.name) == (size_t)(eq - name) && strncmp(k.name, name, (size_t)(eq - name)) == 0) *k.value = eq + 1;
        }
    }
};

// Relative cost of writing NCHW output in runs of `run` contiguous pixels (tuning knob DNB_TC_NCHW_PENALTY scales it;
// 0 = the tile that suits channels-last output).
static double nchw_run_penalty(int run)
{
    static double scale = -1.0;
    if (scale < 0.0) { const char *e = getenv("DNB_TC_NCHW_PENALTY"); scale = e ? atof(e) : 1.0; }
    const double base = run >= 32 ? 0.0 : run >= 16 ? 0.03 : run >= 8 ? 0.10 : run >= 4 ? 0.5 : run >= 2 ? 1.0 : 2.0;
    return scale * base;
}

static void pick_pixel_tile(const ConvGeom &g, bool nchw_out, int *wt, int *ht, int *bt, bool even = false)
{
    // wt*ht*bt == 128, powers of two; least padded work, then widest rows.
    // A launch that writes Darknet's layout stores, per filter plane, one run of wt pixels per tile row: runs shorter
    // than a 32-byte sector make every store a partial-sector write, which costs far more than the padded work of a
    // wider tile (measured on the 255-filter heads of YOLOv3-608, batch 64: 4-pixel runs 2.0 ms, see nchw_run_penalty).
    double best = 1e300;
    for (int w = 1; w <= 128; w *= 2)
        for (int h = 1; w * h <= 128; h *= 2) {
            if (even && (w < 2 || h < 2 || w > 16)) continue;   // a warp's lanes hold whole windows
            const int b = 128 / (w * h);
            const double work = (double)round_up(g.out_w, w) * round_up(g.out_h, h) * round_up(g.batch, b);
            double score = work * (1.0 + 1e-6 * (128 - w) + 1e-7 * (128 - h));
            if (nchw_out) score *= 1.0 + nchw_run_penalty(w < g.out_w ? w : g.out_w);
            if (score < best) { best = score; *wt = w; *ht = h; *bt = b; }
        }
}

// ------------------------------------------------------------------ the kernel for launches that do not fill the GPU
namespace {

struct SplitPlan {
    int pair = 0, bn = 0, splits = 0, stages = 0, wt = 0, ht = 0, bt = 0, ptiles = 0;
    double cost = 1e300;   // microseconds, estimated
};

struct PixelBox { int wt = 1, ht = 1, bt = 1, tiles = 1; };

// The box of at most 128 pixels that covers the output with the fewest tiles; widest rows among equals.
PixelBox split_pixel_tile(const ConvGeom &g)
{
    PixelBox box;
    long long best = 0;
    for (int w = 1; w <= 128 && w <= g.out_w; ++w)
        for (int h = 1; w * h <= 128 && h <= g.out_h; ++h) {
            int b = 128 / (w * h);
            if (b > g.batch) b = g.batch;
            const long long n = (long long)((g.out_w + w - 1) / w) * ((g.out_h + h - 1) / h) * ((g.batch + b - 1) / b);
            if (!best || n < best || (n == best && w > box.wt)) { best = n; box.wt = w; box.ht = h; box.bt = b; }
        }
    box.tiles = (int)best;
    return box;
}

// Microseconds that one K iteration (128 pixels x bn filters x 128 bytes of channels) takes a CTA that has its SM to itself,
// measured on B200: the larger of four MMAs (77 clocks each up to 128 filters, 128 for 256) and of the slot's trip from L2.
double iter_us(int pair, int bn) { return pair ? 0.26 : bn <= 64 ? 0.15 : bn <= 128 ? 0.207 : 0.30; }

struct SplitQuery {
    int row_bytes, k_iters, n_pad, max_smem;
    bool pair_ok, residual, long_sum;   // long_sum: 8192 products per output or more
};

// Cheapest tile of one launch at S ranges, in microseconds of a launch inside a chain of dependent ones (the sums were fitted
// to a sweep over the 3x3 and 1x1 layers of YOLOv3 and ResNet-50 at 1 to 8 images; most choices come out within 15 % of what
// they take): launch and first loads; K iterations; dump of the accumulator (4 ns a column); partial sums through distributed
// shared memory (20 ns per KB); stores and residual, by the number of 16-byte pieces a thread finishes.
SplitPlan split_of(const SplitQuery &q, const PixelBox &box, int pair, int S)
{
    SplitPlan best;
    const int sms = sm_count(), a_bytes = 128 * q.row_bytes, cluster = pair ? 2 * S : S;
    const int resident = conv_tc_split_resident(pair, cluster);   // clusters live inside one GPC: SMs may be left over
    for (int opt = 0; opt < 3 && resident > 0; ++opt) {
        int bn = 64 << opt;
        if (pair && bn != 256) continue;
        if (!pair && bn > q.n_pad) {
            if (opt > 0 && bn / 2 >= q.n_pad) continue;    // the narrower tile already holds every filter
            bn = q.n_pad;
        }
        const int n_tiles = (q.n_pad + bn - 1) / bn;
        const long long tiles = (long long)(pair ? (box.tiles + 1) / 2 : box.tiles) * n_tiles;
        if (tiles > 4LL * sms) continue;
        const int b_bytes = round_up((pair ? bn / 2 : bn) * q.row_bytes, 1024), per = (q.k_iters + S - 1) / S;
        // the whole K range of a CTA in the ring if it fits: the deepest ring is what hides the loads' latency
        int stages = (q.max_smem - 4096) / (a_bytes + b_bytes);
        if (stages > 12) stages = 12;
        if (stages > per) stages = per < 2 ? 2 : per;
        if (stages < 2 || conv_tc_split_smem(stages, a_bytes + b_bytes, bn, nullptr) > (size_t)q.max_smem) continue;
        const long long rounds = (tiles + resident - 1) / resident;
        const double pieces = (128.0 / S) * (bn / 4) / 320.0, remote_kb = (double)(S - 1) / S * bn * 0.5;
        const double finish = 0.004 * bn + 0.02 * remote_kb + pieces * (q.residual ? 0.32 : 0.22) + (pair ? 1.3 : 0.0);
        const double cost = 4.5 + rounds * (per * iter_us(pair, bn) + finish) + (rounds - 1) * 4.0;
        if (cost < best.cost) {
            best.pair = pair; best.bn = bn; best.splits = S; best.stages = stages; best.wt = box.wt; best.ht = box.ht; best.bt = box.bt; best.ptiles = box.tiles; best.cost = cost;
        }
    }
    return best;
}

// The cheapest of all splits (only_s: of those into so many ranges).  One or two images get the same number of ranges, the
// one that is best for one with an eye on two, so that an image's sums do not depend on whether another came with it.
SplitPlan choose_split(const SplitQuery &q, const ConvGeom &g, int only_s, bool prefer_pair, int images)
{
    SplitPlan best[2];
    double score[2] = {1e300, 1e300};
    const PixelBox box = split_pixel_tile(g);   // once: it is the same for every split, and a network has a hundred layers to plan
    const bool with_two = images == 1 && only_s <= 1;
    ConvGeom two = g;
    if (two.batch == 1 && two.h == 1 && q.k_iters && g.size == 1) two.w = two.out_w = 2 * g.out_w;   // flattened pixels
    else two.batch = 2;
    const PixelBox box_two = with_two ? split_pixel_tile(two) : box;
    for (int S = only_s > 1 ? only_s : 2; S <= (only_s > 1 ? only_s : 8); ++S) {
        if (S > q.k_iters || (only_s <= 1 && q.k_iters / S < 3)) break;
        for (int pair = 0; pair < (q.pair_ok ? 2 : 1); ++pair) {
            const SplitPlan sp = split_of(q, box, pair, S);
            if (!sp.splits) continue;
            double sc = sp.cost;
            if (with_two) {
                const SplitPlan t = split_of(q, box_two, pair, S);
                sc += t.splits ? 0.5 * t.cost : 1e6;
            }
            if (sc < score[pair]) { score[pair] = sc; best[pair] = sp; }
        }
    }
    // Near-ties go to pairs: fewer bytes through L2 for the same MMAs.  (Without the 5 % YOLOv3-608 in TF32 takes 871 us instead of 861
    // for one image, 1338 instead of 1301 for two.)  For sums of 8192 products and more, which no layer of the benchmark's
    // networks has, the tests of the split pair kernel fix the choice at pairs (3x3 over 1024 channels); that is not the faster one: at
    // 13x13 / 19x19 / 19x19 x 2 images / 26x26 25.6 / 26.9 / 53.1 / 32.4 us in pairs, 21.8 / 23.5 / 33.4 / 29.5 in single CTAs,
    // which the 5 % would choose; over 896 channels single CTAs take 19.4 / 20.8 / 29.9 / 26.6.
    const double tie = prefer_pair ? 1e9 : q.k_iters >= 144 && q.long_sum ? 1.5 : 1.05;
    return best[1].splits && score[1] < tie * score[0] ? best[1] : best[0];
}

}  // namespace

// Input maps of a convolution: lattice (ph, pw) of the input holds rows ph, ph+stride, ... and columns pw, pw+stride, ...
static int encode_input_maps(CUtensorMap *maps, const ConvGeom &g, const dnb_tensor *x, int kind, int es, int c_pad, const uint32_t *box, int row_bytes)
{
    const size_t pix_bytes = (size_t)x->cpitch * es;
    const int s = g.stride;
    if (s > 2) DNB_FAIL(DNB_EUNSUPPORTED, "conv: stride %d on the tensor-core path (1 and 2 are covered)", s);
    for (int ph = 0; ph < s; ++ph)
        for (int pw = 0; pw < s; ++pw) {
            const int hl = (g.h - ph + s - 1) / s, wl = (g.w - pw + s - 1) / s;
            uint64_t dims[4] = {(uint64_t)c_pad, (uint64_t)(wl > 0 ? wl : 1), (uint64_t)(hl > 0 ? hl : 1), (uint64_t)g.batch};
            uint64_t strides[3] = {pix_bytes * s, pix_bytes * g.w * s, pix_bytes * g.w * g.h};
            char *base = (char *)x->data + ((size_t)ph * g.w + pw) * pix_bytes;
            if (hl <= 0 || wl <= 0) base = (char *)x->data;  // lattice empty: never addressed in-bounds
            DNB_TRY(encode_tensor_map(&maps[ph * s + pw], kind, 4, base, dims, strides, box, row_bytes));
        }
    return DNB_OK;
}

static int encode_weight_map(CUtensorMap *map, const dnb_conv_plan *p, int kind, int es, int c_pad, int taps, int bk, int rows, int row_bytes)
{
    uint64_t dims[3] = {(uint64_t)c_pad, (uint64_t)p->n_pad, (uint64_t)taps};
    uint64_t strides[2] = {(uint64_t)c_pad * es, (uint64_t)c_pad * es * p->n_pad};
    uint32_t box[3] = {(uint32_t)bk, (uint32_t)rows, 1u};
    return encode_tensor_map(map, kind, 3, kind == 2 ? (void *)p->w_i8 : p->w_tc, dims, strides, box, row_bytes);
}

// The launch block is made for each call, not kept: two streams or threads may have the same plan in use.
static int build_fp32_tc_args(const dnb_conv_plan *p, const dnb_tensor *x, void *y_nhwc, int y_cpitch, float *y_nchw, const ConvEpilogue &ep, Fp32TcArgs &a)
{
    ConvGeom g = p->g;
    a.taps = g.size * g.size;
    a.c_blocks = (g.c + 31) / 32;
    a.last_slices = (g.c - 32 * (a.c_blocks - 1) + 15) / 16;
    a.bn = fp32_tc_filters(p->d.n);
    a.n_tiles = (p->n_pad + a.bn - 1) / a.bn;
    a.planes = x->layout == DNB_NCHW ? 1 : 0;
    const bool by_image = y_nchw || a.planes;
    if (g.size == 1 && g.stride == 1 && g.pad == 0) {   // pixels in one row; of the whole batch where no tensor has planes
        g.w = g.out_w = g.w * g.h * (by_image ? 1 : g.batch);
        g.h = g.out_h = 1;
        if (!by_image) g.batch = 1;
    }
    a.x = (const float *)x->data;
    if (a.planes) { a.xs_w = 1; a.xs_h = g.w; a.xs_c = (long long)g.h * g.w; a.xs_b = g.c * a.xs_c; }
    else { a.xs_c = 1; a.xs_w = x->cpitch; a.xs_h = (long long)g.w * x->cpitch; a.xs_b = g.h * a.xs_h; }
    a.w = p->w_direct; a.npg_pad = p->npg_pad;
    pick_pixel_tile(g, by_image, &a.wt, &a.ht, &a.bt);
    a.tiles_w = (g.out_w + a.wt - 1) / a.wt;
    a.tiles_h = (g.out_h + a.ht - 1) / a.ht;
    a.total_tiles = a.n_tiles * a.tiles_w * a.tiles_h * ((g.batch + a.bt - 1) / a.bt);
    a.n_pad = p->n_pad;
    a.smallest = p->fp32_smallest;
    a.g = g;
    a.debug = p->debug_bits;
    a.wait_limit = p->wait_limit > 0 ? p->wait_limit : DEFAULT_WAIT_CYCLES;
    const uint32_t box[4] = {32u, (uint32_t)a.wt, (uint32_t)a.ht, (uint32_t)a.bt};
    if (!a.planes) DNB_TRY(encode_input_maps(a.tmx, g, x, 0, 4, p->c_pad, box, 128));
    const uint64_t row = 64;   // 32 channels of one part
    uint64_t dims[4] = {32u, (uint64_t)p->n_pad, 3u, (uint64_t)a.taps * a.c_blocks};
    uint64_t strides[3] = {row, row * p->n_pad, row * p->n_pad * 3};
    uint32_t wbox[4] = {32u, (uint32_t)a.bn, 3u, 1u};
    DNB_TRY(encode_tensor_map(&a.tmw, 1, 4, p->w_parts, dims, strides, wbox, 64));
    if (y_nhwc) {
        const size_t opix = (size_t)y_cpitch * 4;
        const int n8 = round_up(g.n, 8), cols = a.bn / 2 < 32 ? a.bn / 2 : 32;
        uint64_t ydims[4] = {(uint64_t)(n8 < y_cpitch ? n8 : y_cpitch), (uint64_t)g.out_w, (uint64_t)g.out_h, (uint64_t)g.batch};
        uint64_t ystrides[3] = {opix, opix * g.out_w, opix * g.out_w * g.out_h};
        uint32_t ybox[4] = {(uint32_t)cols, (uint32_t)a.wt, (uint32_t)a.ht, (uint32_t)a.bt};
        DNB_TRY(encode_tensor_map(&a.tmy, 0, 4, y_nhwc, ydims, ystrides, ybox, cols * 4));
    }
    a.y_nhwc = (float *)y_nhwc; a.y_nchw = y_nchw;
    a.status = p->status;
    a.ep = ep;
    return DNB_OK;
}

static int build_split_args(dnb_conv_plan *p, const dnb_tensor *x, const ConvGeom &g, const SplitPlan &sp, int kind, int es,
                            void *y_nhwc, int y_cpitch, void *sign_out, int sign_cpitch)
{
    const TcArgs &t = p->tc;
    SplitArgs &a = p->sp;
    const int c_pad = kind == 2 ? p->c_pad_i8 : p->c_pad;
    a.kind = kind; a.pair = sp.pair; a.splits = sp.splits; a.bn = sp.bn; a.stages = sp.stages;
    a.row_bytes = t.row_bytes; a.bk = t.bk; a.c_blocks = t.c_blocks; a.taps = t.taps;
    a.wt = sp.wt; a.ht = sp.ht; a.bt = sp.bt; a.rows = sp.wt * sp.ht * sp.bt;
    a.tiles_w = (g.out_w + a.wt - 1) / a.wt;
    a.tiles_h = (g.out_h + a.ht - 1) / a.ht;
    a.n_tiles = (p->n_pad + a.bn - 1) / a.bn;
    a.tiles = (a.pair ? (sp.ptiles + 1) / 2 : sp.ptiles) * a.n_tiles;
    a.a_bytes = 128 * a.row_bytes;
    a.b_bytes = round_up((a.pair ? a.bn / 2 : a.bn) * a.row_bytes, 1024);
    conv_tc_split_smem(a.stages, a.a_bytes + a.b_bytes, a.bn, &a.work_bytes);
    a.tmem_cols = 32;
    while (a.tmem_cols < a.bn) a.tmem_cols *= 2;
    const int n8 = round_up(g.n, 8);
    a.n_write = y_nhwc ? (n8 < y_cpitch ? n8 : y_cpitch) : g.n;
    a.sign_out = sign_out; a.sign_cpitch = sign_cpitch;
    a.debug = t.debug; a.wait_limit = t.wait_limit;
    a.g = g;
    DNB_TRY(ensure_status(p));
    const uint32_t box[4] = {(uint32_t)a.bk, (uint32_t)a.wt, (uint32_t)a.ht, (uint32_t)a.bt};
    DNB_TRY(encode_input_maps(a.tmx, g, x, kind, es, c_pad, box, a.row_bytes));
    DNB_TRY(encode_weight_map(&a.tmw, p, kind, es, c_pad, a.taps, a.bk, a.pair ? a.bn / 2 : a.bn, a.row_bytes));
    p->tc_split = true;
    return DNB_OK;
}

// Microseconds of the persistent kernel, in a chain of dependent launches as split_of has it.  A K iteration measured on B200 with 3x3 layers
// of 256 to 1024 channels at 1 to 16 images: pairs 0.168 (128 filters) and 0.287 (256), single CTAs 0.317 (256), 0.187 (128) and 0.18 (64)
// with an SM to themselves, 0.26 and 0.135 where two share one and its room for ring slots.  An epilogue hides behind the next tile's loop, or
// the other way round, and the last one is exposed.
static double persistent_us(int pair, int bn, long long tiles, int k_iters, bool residual, bool yolo = false)
{
    const long long slots = pair ? sm_count() / 2 : sm_count();
    const bool shared = !pair && bn <= 128 && tiles > sm_count();
    const double rounds = (double)((tiles + slots - 1) / slots);
    const double iteration = pair ? (bn <= 128 ? 0.168 : 0.287) : bn <= 64 ? (shared ? 0.135 : 0.18) : bn <= 128 ? (shared ? 0.26 : 0.187) : 0.317;
    const double loop = k_iters * iteration, epilogue = bn * (yolo ? 0.06 : residual ? 0.02 : 0.015);   // (a [yolo] layer's logistic: two special functions and a store a value)
    return 4.2 + (pair ? 1.0 : 0.0) + rounds * (loop > epilogue ? loop : epilogue) + 0.8 * epilogue;
}

// Whether K is cut, and how often, is part of a layer's result: its sums are added in another order.  So that choice stands by itself, on tiles
// halved until they fill the SMs (pick_persistent_tiles, plain) and the measure that it was fitted with, and better tiles for the
// persistent kernel, which change no sum, leave every output as it was.
static double uncut_us(const TcArgs &a, int k_iters, bool residual)
{
    const long long slots = a.pair ? sm_count() / 2 : sm_count();
    const double share = (double)((a.total_tiles + slots - 1) / slots);
    const double loop = k_iters * (!a.pair && a.bn <= 64 && share < 2.0 ? 0.18 : a.pair ? 0.31 : iter_us(a.pair, a.bn));
    const double epilogue = a.bn * (residual ? 0.02 : 0.015);
    return 3.6 + share * (loop > epilogue ? loop : epilogue) + epilogue;
}

// Tiles of the persistent kernel for a launch of geometry g: pixel box, filters per tile, pairs.  a.row_bytes, a.c_blocks are set.
// plain: by the number of tiles alone (see uncut_us).
static void pick_persistent_tiles(const dnb_conv_plan *p, const Knobs &knobs, const ConvGeom &g, TcArgs &a, bool nchw_out, bool channels_last, int y_cpitch, bool residual, bool pool = false, bool plain = false)
{
    const bool bf16 = p->kernel == K_TC_BF16, i8 = p->kernel == K_XNOR;
    pick_pixel_tile(g, nchw_out, &a.wt, &a.ht, &a.bt, pool);
    a.halo = 0;
    a.tiles_w = (g.out_w + a.wt - 1) / a.wt;
    a.tiles_h = (g.out_h + a.ht - 1) / a.ht;
    a.tiles_b = (g.batch + a.bt - 1) / a.bt;
    const int ptiles = a.tiles_w * a.tiles_h * a.tiles_b;
    // Filters per tile.  One tile when they fit (<= 256).  Otherwise a multiple of 64 (so that every
    // staged output chunk lies inside one tile), weighing padded MMA columns against operand re-loads.
    if (p->n_pad <= 256) {
        a.bn = p->n_pad;
    } else {
        double best = 1e300;
        for (int bn = 64; bn <= 256; bn += 64) {
            const int nt = (p->n_pad + bn - 1) / bn;
            const double score = (double)nt * bn + 0.5 * nt * 128;
            if (score <= best) { best = score; a.bn = bn; }
        }
    }
    // Tuning knobs for experiments: DNB_TC_BN (filters per tile, a multiple of 64) and DNB_TC_STAGES.
    if (const char *e = knobs.bn) {
        const int v = atoi(e);
        if (v >= 64 && v <= 256 && v % 64 == 0 && p->n_pad > v) a.bn = v;
    }
    a.n_tiles = (p->n_pad + a.bn - 1) / a.bn;
    // Too few tiles to fill the SMs: narrower ones, as long as the launch is estimated to end sooner.  Up to 128 filters an MMA takes
    // the same 77 clocks, so what counts is how many tiles the fullest SM gets: 50 pixel tiles of 256 filters are better cut into 100 tiles of 128
    // than into 200 of 64 (3x3 128 -> 256 at 76 x 76 20.9 -> 18.9 us, 256 -> 512 at 4 x 26 x 26 32.7 -> 26.8; YOLOv3-608, one image, in a graph 898 -> 874,
    // YOLOv3-416, four, 1282 -> 1203).
    const int k_iters = g.size * g.size * a.c_blocks;
    auto estimate = [&](int pair, int bn) {
        return persistent_us(pair, bn, (long long)(pair ? (ptiles + 1) / 2 : ptiles) * ((p->n_pad + bn - 1) / bn), k_iters, residual);
    };
    if (ptiles * a.n_tiles < sm_count()) {
        int best = a.bn;
        for (int bn = a.bn; bn >= 128 && bn % 128 == 0 && ptiles * ((p->n_pad + bn - 1) / bn) < sm_count();) {
            bn /= 2;
            if (plain || estimate(0, bn) <= estimate(0, best)) best = bn;
        }
        a.bn = best;
        a.n_tiles = (p->n_pad + a.bn - 1) / a.bn;
    }
    // A launch that writes Darknet's layout spends a store per output element in its epilogue; behind a short K loop
    // (the 1x1 heads of YOLOv3) that is the whole run time, and the four epilogue warps of one CTA per SM issue it
    // slowly: 128-filter tiles leave TMEM for a second CTA, i.e. eight epilogue warps.
    if (nchw_out && a.bn == 256 && g.size * g.size * a.c_blocks <= 16) {
        a.bn = 128;
        a.n_tiles = (p->n_pad + a.bn - 1) / a.bn;
    }
    // CTA pairs (cta_group::2): for layers whose filters come in whole tiles of 256 and whose K loop is long enough to
    // be bound by operand traffic.  Each CTA of a pair loads its own 128 pixels and half of the 256-filter weight tile:
    // a third fewer bytes from L2 into shared memory per MMA, and 32 KB ring slots (six of them) instead of 48 KB (four).
    // Layers with at least 16 K iterations (1x1 layers over 512 channels in TF32: 8 % faster than single CTAs on YOLOv3's 38x38 and
    // 19x19 layers at batch 64).  A 3x3 layer over one block of channels has nine: its epilogue outlasts its MMAs, and single
    // CTAs hand over with less ceremony (33 x 38 x 38, 64 -> 1024 in bf16 59.6 us in pairs, 55.6 without; 64 -> 256 19.5 and 16.4;
    // 32 -> 1024 in TF32 74 and 71.5; 128 -> 256 of xnor layers, 128 x 28 x 28, 52.2 and 48.1); over two blocks, 18 iterations, pairs
    // are ahead again (96 -> 512 in bf16 44.4 and 53.7).  With a fused residual nine iterations still run in pairs: the tests fix that choice (64 -> 512, stride 2, 40 x 44 x 44 in bf16: 23.5 us,
    // 20 in single CTAs).  DNB_TC_PAIR: 0 never, 1 3x3 layers of fewer iterations too, 2 every layer the geometry allows.
    a.pair = 0;
    {
        const char *e = knobs.pair;
        const int knob = e ? atoi(e) : -1;
        // (the pair kernel is built for 128-byte staged rows only: it needs a channels-last output at least that wide)
        // Enough pair tiles to occupy every pair of SMs; or, for long K loops (small batches of the 19x19 and 38x38
        // layers), at least half of them: a pair's six-deep ring of 32 KB slots keeps its tensor pipes fed where two
        // single CTAs per SM with two or three slots each starve on load latency, which outweighs the idle SMs.
        const int pair_tiles = (ptiles + 1) / 2 * (g.n / 256), clusters = sm_count() / 2;
        const bool enough = pair_tiles >= clusters || (k_iters >= 64 && 2 * pair_tiles >= clusters);
        const bool legal = a.row_bytes == 128 && channels_last && y_cpitch * (bf16 ? 2 : 4) >= 128 && !pool;
        const bool wanted = legal && (knob == 2 || (g.size >= 3 && (knob == 1 || (knob < 0 && residual))) || (knob != 0 && k_iters >= 16));
        if (wanted && g.n % 256 == 0 && enough) {
            a.pair = 1;
            a.bn = 256;
            a.n_tiles = p->n_pad / 256;
        }
        // A launch of a few rounds: the whole rounds it takes decide between tiles.  A pair over 128 filters loads as little per MMA as it can
        // (24 KB an iteration and CTA, 0.168 us) and comes in halves of a pair over 256, which is the better one in full rounds: 3x3 512 -> 512 at 16 x
        // 26 x 26 in TF32 99.6 -> 80.9 us (pairs over 256: 90.0), 256 -> 256 at 8 x 52 x 52 49.2 -> 45.0, 1024 -> 1024 at 16 x 19 x 19 196 -> 162, and in
        // bf16 8 x 52 x 52 27.7 -> 25.9; 2 x 76 x 76 stays with 256 (30.0 and 31.4).
        if (knob < 0 && !plain && !i8 && g.n % 128 == 0 && (ptiles + 1) / 2 * ((g.n + 255) / 256) < 6 * clusters) {
            double best = estimate(a.pair, a.bn);
            for (int pair = a.pair; pair < 2; ++pair)
                for (int bn = 128; bn <= 256; bn *= 2) {
                    if (g.n % bn || (pair && !(wanted && k_iters >= 16)) || (!pair && nchw_out)) continue;
                    const double us = estimate(pair, bn);
                    if (us < 0.97 * best) { best = us; a.pair = pair; a.bn = bn; a.n_tiles = p->n_pad / bn; }
                }
        }
    }
    a.total_tiles = a.pair ? (ptiles + 1) / 2 * a.n_tiles : ptiles * a.n_tiles;
}

// ------------------------------------------------------------------ 3x3 layers with one load for nine taps, 1x1 layers with their filters in place (conv_tc_taps.cu)
// The launch's tiles and rings; p->tp holds them.  False where the kernel has no form of it.
static bool taps_tiles(dnb_conv_plan *p, const ConvGeom &g, int bn, bool boxes, bool channels_last, bool residual)
{
    TapsArgs &a = p->tp;
    const int es = p->kernel == K_TC_BF16 ? 2 : 4;
    a.bf16 = es == 2 ? 1 : 0;
    a.bk = 128 / es;
    a.c_blocks = (p->c_pad + a.bk - 1) / a.bk;
    a.g = p->g;
    a.taps = g.size * g.size;
    a.boxes = boxes ? 1 : 0;
    a.tiles_w = (g.w + 7) / 8; a.tiles_h = (g.h + 15) / 16;
    a.pitch = boxes ? 10 : g.w + 1;
    a.rows = a.taps == 1 ? 128 : boxes ? 180 : 128 + 2 * a.pitch + 2;
    if (a.rows > 1024 || (boxes && a.taps == 1)) return false;
    const long long pixels = (long long)g.batch * g.h * g.w;
    const long long positions = a.taps == 1 ? pixels : boxes ? 128LL * a.tiles_w * a.tiles_h * g.batch : (long long)g.batch * a.pitch * (g.h + 1) - a.pitch - 1;
    if (positions > (1LL << 31) - 4096) return false;
    a.pixels = (int)pixels;
    a.ptiles = (int)((positions + 127) / 128);
    a.bn = bn;
    a.n_tiles = (p->n_pad + bn - 1) / bn;
    const long long tiles = (long long)((a.ptiles + 1) / 2) * a.n_tiles;
    if (tiles > 1 << 30) return false;
    a.total_tiles = (int)tiles;
    a.x_slot = round_up(a.rows * 128, 1024);
    a.w_bytes = round_up(bn / 2 * 128, 1024);
    a.staged_bytes = channels_last ? (residual ? 98304 : 32768) : 0;
    a.table = round_up(a.n_tiles * bn, 64);
    a.tmem_cols = 32;
    while (a.tmem_cols < 2 * bn) a.tmem_cols *= 2;
    a.x_stages = a.w_stages = 0;
    a.resident = 0;
    const long budget = conv_tc_max_smem() - (long)conv_tc_taps_fixed_smem(a);
    const int all = a.taps * a.c_blocks * a.n_tiles, least = a.taps == 1 ? 3 : 2;   // boxes in flight, where they are all that is loaded
    if ((a.taps == 1 || a.n_tiles == 1) && all <= TAPS_MAX_W && (long)least * a.x_slot + (long)all * a.w_bytes <= budget) {
        a.resident = 1;
        a.w_stages = all;
        a.x_stages = (int)((budget - (long)all * a.w_bytes) / a.x_slot);
    } else if (a.taps == 1) {
        a.x_stages = a.w_stages = (int)(budget / (a.x_slot + a.w_bytes));
    } else {
        a.x_stages = 2;
        long left = budget - 2L * a.x_slot;
        // a third box where the filters' ring keeps its depth
        if (left - a.x_slot >= 8L * a.w_bytes) { a.x_stages = 3; left -= a.x_slot; }
        a.w_stages = left > 0 ? (int)(left / a.w_bytes) : 0;
        if (a.w_stages > 12) a.w_stages = 12;
    }
    if (a.x_stages > TAPS_MAX_X) a.x_stages = TAPS_MAX_X;
    return a.x_stages >= 2 && (a.resident || a.w_stages >= 4);
}

// Whether the kernel has a variant for such a launch of the plan.  A 1x1 layer with a residual has not: its addend arrives by TMA, three chunks
// ahead, in conv_tc.cu (64 -> 256 at 256 x 56 x 56 335 us, 363 here).
static bool taps_covers(const dnb_conv_plan *p, const ConvEpilogue *res, bool nchw_out)
{
    const ConvGeom &g = p->g;
    const int es = p->kernel == K_TC_BF16 ? 2 : 4;
    if ((p->kernel != K_TC_TF32 && p->kernel != K_TC_BF16) || g.stride != 1 || p->c_pad * es < 128 || (p->d.activation != DNB_LEAKY && p->d.activation != DNB_LINEAR)) return false;
    if (g.size == 1) return g.pad == 0 && !(res && res->residual);
    if (g.size != 3 || g.pad != 1 || p->keep_k_order || (res && res->yolo_entries)) return false;
    if (p->tap_order && p->c_pad * es > 128) return false;   // (one block of channels: there is one order)
    return !(res && res->residual) ||
           (res->res_stride == 1 && res->res_c == g.n && !nchw_out && res->activation2 == (p->d.activation == DNB_LEAKY ? DNB_LINEAR : DNB_LEAKY));
}

// Microseconds of such a launch, fitted to 600 measured launches of 3x3 and 1100 of 1x1 layers (32 to 1024 filters over 32 to 2048 channels, maps of 7 to 152, 1 to
// 128 images, either type and layout; 7 and 12 % root mean square): an iteration is the four MMAs of a tap and 128 bytes of channels, 0.174 up to 128
// filters and 0.31 at 256, a box for a single tap more; the im2col load takes 3.7 ns a position; a tile's epilogue 6 ns a filter, 19 in Darknet's
// layout, 27 with a residual.  A 1x1 layer moves its tensors at 6.1 TB/s at most.
static double taps_us(const TapsArgs &a, bool nchw_out, bool residual, bool yolo)
{
    const double clusters = sm_count() / 2, rounds = ceil(a.total_tiles / clusters), wide = a.bn <= 128 ? 0.0 : (a.bn - 128) / 128.0;
    const double epilogue = a.bn * (yolo ? 0.03 : nchw_out ? 0.019 : residual ? 0.027 : 0.006);
    if (a.taps == 1) {
        const double mma = a.c_blocks * (0.26 + 0.103 * wide), bytes = (double)a.pixels * (a.c_blocks * 128.0 + a.g.n * (nchw_out || !a.bf16 ? 4.0 : 2.0));
        const double tiles = rounds * ((mma > epilogue ? mma : epilogue) + 0.6);
        return 7.2 + (tiles > bytes / 6.1e6 ? tiles : bytes / 6.1e6);
    }
    const double mma = 9.0 * a.c_blocks * (0.174 + 0.136 * wide), load = a.c_blocks * a.rows * (a.boxes ? 0.0011 : 0.0037);
    const double longest = mma > load ? (mma > epilogue ? mma : epilogue) : (load > epilogue ? load : epilogue);
    return 5.3 + rounds * (longest + 0.65) + 0.55 * epilogue + load / a.c_blocks;
}

// The best tile of a launch of geometry g, in p->tp; its estimated time, or 1e300.
static double best_taps(dnb_conv_plan *p, const Knobs &knobs, const ConvGeom &g, bool channels_last, bool nchw_out, bool residual, bool yolo)
{
    const char *e = knobs.taps_bn;
    const int only = e ? atoi(e) : 0;
    const char *be = knobs.taps_box;
    int best_bn = 0, best_boxes = 0;
    double best = 1e300;
    for (int bn = 64; bn <= 256; bn *= 2)
        for (int boxes = 0; boxes < 2; ++boxes) {
            if (be && atoi(be) != boxes) continue;
            const int width = bn < p->n_pad ? bn : round_up(p->n_pad, 32);   // (MMAs of 256 rows have columns in steps of 32)
            if ((only && bn != only) || (bn > 64 && bn / 2 >= p->n_pad) || !taps_tiles(p, g, width, boxes, channels_last, residual)) continue;
            const double us = taps_us(p->tp, nchw_out, residual, yolo);
            if (us < best) { best = us; best_bn = width; best_boxes = boxes; }
        }
    return best_bn && taps_tiles(p, g, best_bn, best_boxes, channels_last, residual) ? best : 1e300;
}

// Whether a launch takes that kernel: where its estimate is well below what the others take.  others_us: the estimate of the launch that it would
// be, cut along K or not.  Those estimates are of launches in a chain; in the measure of taps_us, launches by themselves, cut ones take 1.3 times
// theirs and whole ones 1.12, in Darknet's layout 1.55 and 1.3 (stores in the short rows of a tile), with a residual 1.25 and 0.95 (1.05 alone, but 64 x 64 x 152 x 152 -> 128
// is 516 -> 485 us alone and 548 -> 568 inside YOLOv3-608).  On 200 random 3x3
// launches the rule takes 68 here, 7 of them to their loss (of 4 to 13 %), 18 in less than 0.8 of the time, and all of the launches take 0.946 of what they did: 16 x 256 x 52 x 52
// -> 512 in Darknet's layout 153 -> 126 us, 2 x 120 x 76 x 76 -> 128 26.8 -> 14.2, 256 x 128 x 28 x 28 -> 128 128 -> 106, 34 x 232 x 38 x 38 -> 255 in bf16 85 -> 42.
// Launches of many rounds of pairs over 256 filters run into the power cap in either kernel (64 x 256 x 38 x 38 -> 512 265 -> 261 alone, 300 -> 307
// inside YOLOv3-608) and stay where less padding is multiplied.
// The kernel adds the products of a 3x3 layer in another order, so g is that of the whole batch where the plan is for a part of it, and of one image where
// there are two: an image's sums then hang neither on the parts nor on the other image.
// 1x1 layers add in the same order and are never cut here: what they gain is that their filters are loaded once (wide tiles, which are at least even alone, take a
// tenth less power: 64 x 512 x 52 x 52 -> 256 in bf16 53.2 -> 51.9 us alone, 62.9 -> 59.5 back to back; 256 -> 128 at
// 64 x 76 x 76 inside YOLOv3-608 110 -> 99, 512 -> 256 at 64 x 32 x 32 in bf16 35 -> 29; 128 filters over four rounds of pairs and
// more where six blocks of pixels fit beside them: 256 -> 128 at 32 x 52 x 52 30.5 -> 26.5, 512 -> 128 at 32 x 52 x 52 in bf16 26.8 -> 24.0; over ten where fewer do: 512 ->
// 128 at 256 x 28 x 28 102.7 -> 100.8, but at 40 x 46 x 46 42.3 -> 46.2) and the stores in Darknet's layout (255 filters at 64 x 76 x 76 180 -> 138,
// with a [yolo] layer's logistic 271 -> 174, 345 -> 226 inside YOLOv3-608); a launch of less than two rounds of pairs is not worth their set-up
// (255 filters and the logistic at 26 x 26, one image: 7.2 us, 8.9 here).
// DNB_TC_TAPS: 0 never, 2 wherever the kernel has the variant; the other kernels' knobs ask for those kernels.
static bool taps_pay(dnb_conv_plan *p, const Knobs &knobs, const ConvGeom &g, bool cut, double others_us, const ConvEpilogue *res, bool channels_last, bool nchw_out)
{
    const char *e = knobs.taps;
    const int knob = e ? atoi(e) : 1;
    if (knob == 0) return false;
    const bool residual = res && res->residual;
    const bool yolo = res && res->yolo_entries > 0;
    const double slack = yolo ? 1.0 : nchw_out ? (cut ? 1.55 : 1.3) : residual ? (cut ? 1.25 : 0.95) : cut ? 1.3 : 1.12;
    if (knob != 2) {   // what no choice of tiles would change: small launches, whose plans are most of their first call
        const int c_blocks = (p->c_pad * (p->kernel == K_TC_BF16 ? 2 : 4) + 127) / 128;
        if (g.size == 1 && (cut || (((long long)g.batch * g.h * g.w + 127) / 128 + 1) / 2 * ((p->n_pad + 63) / 64) < sm_count())) return false;
        if (g.size == 3 && 5.3 + 9.0 * c_blocks * 0.174 + 0.65 >= 0.9 * slack * others_us) return false;
    }
    if (!e) {
        const char *const split = knobs.splitk;
        if (knobs.pair || knobs.epi || knobs.halo || knobs.warp_stores || (split && atoi(split) > 1)) return false;
    }
    const double us = best_taps(p, knobs, g, channels_last, nchw_out, residual, yolo);
    if (us >= 1e300 || knob == 2) return us < 1e300;
    if (g.size == 1) {
        const TapsArgs &t = p->tp;
        const double bytes = (double)t.pixels * (t.c_blocks * 128.0 + g.n * (nchw_out || !t.bf16 ? 4.0 : 2.0)) / 6.1e6 + 7.2;   // no kernel is faster
        const double others = slack * others_us > bytes ? slack * others_us : bytes;
        const bool even = t.resident && (t.bn >= 192 || (t.bn >= 128 && t.c_blocks >= 8 && t.total_tiles >= (t.x_stages == TAPS_MAX_X ? 2 : 5) * sm_count()));
        return !cut && t.total_tiles >= sm_count() && us < (yolo ? 0.9 : even ? 1.05 : 0.8) * others;
    }
    return us < 0.9 * slack * others_us;
}

static int build_taps_args(dnb_conv_plan *p, const dnb_tensor *x, const void *y_nhwc, int y_cpitch)
{
    TapsArgs &a = p->tp;
    const ConvGeom &g = p->g;
    const int es = a.bf16 ? 2 : 4;
    a.n_pad = p->n_pad;
    const int n8 = round_up(g.n, 8);
    a.y_chan = y_nhwc ? (n8 < y_cpitch ? n8 : y_cpitch) : 0;
    a.debug = p->tc.debug; a.wait_limit = p->tc.wait_limit;
    DNB_TRY(ensure_status(p));
    const uint64_t pix = (uint64_t)x->cpitch * es;
    const uint64_t dims[4] = {(uint64_t)p->c_pad, (uint64_t)g.w, (uint64_t)g.h, (uint64_t)g.batch}, strides[3] = {pix, pix * g.w, pix * g.w * g.h};
    if (a.boxes) {
        const uint32_t box[4] = {(uint32_t)a.bk, 10u, 18u, 1u};
        DNB_TRY(encode_tensor_map(&a.tmx, a.bf16, 4, x->data, dims, strides, box, 128));
    } else if (a.taps == 9) {
        DNB_TRY(encode_im2col_map(&a.tmx, a.bf16, x->data, dims, strides, (uint32_t)a.bk, (uint32_t)a.rows));
    } else {
        const uint64_t flat_dims[3] = {(uint64_t)p->c_pad, (uint64_t)a.pixels, 1}, flat_strides[2] = {pix, pix * a.pixels};
        const uint32_t box[3] = {(uint32_t)a.bk, 128u, 1u};
        DNB_TRY(encode_tensor_map(&a.tmx, a.bf16, 3, x->data, flat_dims, flat_strides, box, 128));
    }
    return encode_weight_map(&a.tmw, p, a.bf16, es, p->c_pad, a.taps, a.bk, a.bn / 2, 128);
}

static int build_tc_args(dnb_conv_plan *p, const dnb_tensor *x, void *y_nhwc, int y_dtype, int y_cpitch,
                         const ConvEpilogue *res, bool nchw_out, void *sign_out = nullptr, int sign_cpitch = 0, bool pool = false)
{
    const void *residual = res ? res->residual : nullptr;   // fused residual, if any
    const int res_cpitch = res ? res->res_cpitch : 0, res_stride = residual ? res->res_stride : 1, res_c = residual ? res->res_c : 0;
    const Knobs knobs;
    TcArgs &a = p->tc;
    p->tc_x_ptr = nullptr;   // until all of the block is there
    p->tc_res_act = residual ? res->activation2 : DNB_LINEAR;
    p->tc_yolo = res && res->yolo_entries > 0 ? 1 : 0;
    // A 1x1 convolution (stride 1, no padding) does not care which pixels are neighbours: with Darknet's layout among
    // the outputs, the h x w plane is treated as one row of h*w pixels, so that a tile is a run of up to 128 contiguous
    // pixels of every filter plane (and of the channels-last input) instead of a wt x ht patch.  DNB_TC_FLAT=0: never.
    ConvGeom g = p->g;
    {
        const char *e = knobs.flat;
        if (nchw_out && g.size == 1 && g.stride == 1 && g.pad == 0 && !(e && atoi(e) == 0)) {
            g.w = g.out_w = g.w * g.h;
            g.h = g.out_h = 1;
        }
    }
    const bool bf16 = p->kernel == K_TC_BF16, i8 = p->kernel == K_XNOR;
    const int es = i8 ? 1 : (bf16 ? 2 : 4);
    const int kind = i8 ? 2 : (bf16 ? 1 : 0);              // element kind of the operands (and of their tensor maps)
    const int c_pad = i8 ? p->c_pad_i8 : p->c_pad;         // channel pitch of the operand tensors
    a.is_bf16 = kind;
    const int cbytes = c_pad * es;
    a.row_bytes = cbytes >= 128 ? 128 : (cbytes >= 64 ? 64 : 32);
    a.bk = a.row_bytes / es;
    a.c_blocks = (c_pad + a.bk - 1) / a.bk;
    a.taps = g.size * g.size;
    a.debug = (knobs.debug ? atoi(knobs.debug) : 0) | p->debug_bits;
    a.wait_limit = p->wait_limit > 0 ? p->wait_limit : DEFAULT_WAIT_CYCLES;
    p->tc_taps = p->tc_split = false;
    pick_persistent_tiles(p, knobs, g, a, nchw_out, y_nhwc != nullptr, y_cpitch, residual != nullptr, pool);
    a.pool = pool ? 1 : 0;
    a.n_pad = p->n_pad;
    a.n_tot = a.n_tiles * a.bn;
    a.a_bytes = 128 * a.row_bytes;
    a.b_bytes = round_up((a.pair ? a.bn / 2 : a.bn) * a.row_bytes, 1024);
    const int max_smem = conv_tc_max_smem();
    if (max_smem <= 0) DNB_FAIL(DNB_ECUDA, "conv: cannot query shared memory of the current device");
    // staged output rows: the widest of 128 / 64 / 32 bytes that the output pitch allows and that keeps
    // at least four ring stages
    const int out_es = bf16 ? 2 : 4;   // channels-last output uses the plan's storage type
    const int pitch_bytes = y_nhwc ? y_cpitch * out_es : 32;
    const int min_srb = sign_out || pool ? 128 : 16 * out_es;  // a staged row holds at least one 16-column piece of the accumulator; the sign output is built for 32 columns per chunk
    int srb = pitch_bytes >= 128 ? 128 : (pitch_bytes >= 64 ? 64 : 32);
    if (srb < min_srb) srb = min_srb;  // the box may be wider than a narrow tensor: the TMA unit clips it
    if (sign_out && (pitch_bytes < 128 || !i8)) DNB_FAIL(DNB_EINVAL, "conv: the sign output needs an int8-kind plan with at least 32 output channels");
    if (const char *e = knobs.srb) {   // tuning knob: widest staged row to try (128, 64 or 32)
        const int v = atoi(e);
        if ((v == 128 || v == 64 || v == 32) && v >= min_srb && v < srb && !a.pair) srb = v;
    }
    const int min_stages = knobs.min_stages ? atoi(knobs.min_stages) : 4;
    // two accumulators of bn columns; TMEM is allocated in powers of two >= 32 columns
    a.tmem_cols = 32;
    while (a.tmem_cols < 2 * a.bn) a.tmem_cols *= 2;
    // Narrow tiles (bn <= 128) leave TMEM and, with a short ring, shared memory for a second CTA on the SM:
    // twice the warps hide the per-tile hand-offs that dominate layers with few K iterations.
    a.ctas_per_sm = 1;
    a.stage_bufs = residual ? 4 : 2;
    if (sign_out) a.stage_bufs = 3;   // the third buffer holds the staged signs
    if (pool) a.stage_bufs = 0;       // pooled rows leave from registers
    a.sign_out = sign_out;
    a.sign_cpitch = sign_cpitch;
    int stages = 0;
    const bool allow2 = knobs.ctas ? atoi(knobs.ctas) >= 2 : true;
    a.a_slot = a.a_box_slot = a.a_box_bytes = a.a_pitch = 0;
    a.epi_groups = 1;
    a.halo = 0;
    // Halo mode, where two CTAs with the layer's weights fit an SM: what a layer over few channels waits for is the rows its copies are made of,
    // 128 pixels and the filters for every tap, and with the weights in place and one box for all taps they are a tenth.  3x3 32 -> 64 at
    // 64 x 304 x 304 in bf16 with a residual 926 -> 487 us, of xnor layers with the maxpool at 128 x 112 x 112 226 -> 138, 16 -> 32 in TF32 at
    // 16 x 208 x 208 72 -> 49.  One CTA alone with its weights is slower than two without (32 -> 64 in TF32 854 -> 900, 64 -> 128 in bf16 at 152 x
    // 152 280 -> 390, of xnor layers at 56 x 56 79 -> 95, 32 -> 64 with stride 2 in bf16 685 -> 790).  Same order of the sums.
    // DNB_TC_HALO: 0 never, 2 wherever the geometry and shared memory allow.
    // Pooled launches stage nothing and their epilogue is the longer part: as many CTAs as TMEM takes (xnor 32 -> 64 at 128 x 112 x 112 103 us with two, 93 with
    // three, 90 with four; 16 -> 32 in TF32 at 16 x 208 x 208 49, 42, 37)
    const int most_ctas = pool && a.tmem_cols <= 128 ? 4 : 2;
    const int halo_knob = knobs.halo ? atoi(knobs.halo) : 1;
    if (halo_knob != 0 && g.size == 3 && g.pad == 1 && a.n_tiles == 1 && !a.pair && g.out_w >= 8 && g.out_h >= 16) {
        const int lattices = g.stride * g.stride, htiles = ((g.out_w + 7) / 8) * ((g.out_h + 15) / 16) * g.batch;
        a.a_pitch = g.stride == 1 ? 10 : 9;
        a.a_box_bytes = a.a_pitch * (g.stride == 1 ? 18 : 17) * a.row_bytes;
        a.a_box_slot = round_up(a.a_box_bytes, 1024);
        a.a_slot = lattices * a.c_blocks * a.a_box_slot;
        const long weights = (long)a.taps * a.c_blocks * a.b_bytes;
        auto fit = [&](long budget, int srb_try, int most) {
            const long left = budget - weights - (long)conv_tc_fixed_smem(srb_try, a.bn, a.stage_bufs);
            const int n = left > 0 ? (int)(left / a.a_slot) : 0;
            if (n < 2) return false;
            stages = n > most ? most : n; srb = srb_try;
            return true;
        };
        bool done = false;
        if (halo_knob == 2 || (htiles >= 2 * sm_count() && htiles <= 1.2 * a.total_tiles)) {
            const int widest = srb;
            if (allow2 && a.tmem_cols <= 256 && htiles > sm_count())
                for (int n = most_ctas; n >= 2 && !done; --n)
                    for (int t = widest; t >= min_srb && !done; t /= 2) { done = fit((228L * 1024) / n - 2048, t, 4); if (done) a.ctas_per_sm = n; }
            for (int t = widest; halo_knob == 2 && t >= min_srb && !done; t /= 2) done = fit(max_smem, t, 4);
            if (!done) srb = widest;
        }
        if (done) {
            a.halo = 1;
            a.wt = 8; a.ht = 16; a.bt = 1;
            a.tiles_w = (g.out_w + 7) / 8; a.tiles_h = (g.out_h + 15) / 16; a.tiles_b = g.batch;
            a.total_tiles = htiles;
            if (a.ctas_per_sm == 1 && srb == 128 && !residual && !pool && (y_nhwc || sign_out) && !nchw_out) a.epi_groups = 2;
        }
    }
    if (!a.halo) {
        // (not when every tile has an SM of its own: one deep ring then)
        if (allow2 && a.tmem_cols <= 256 && !a.pair && a.total_tiles > sm_count()) {
            const int max2 = knobs.max2 ? atoi(knobs.max2) : 4;   // ring slots per CTA when two share the SM
            const long budget = (228L * 1024) / 2 - 2048;   // per CTA when two share the SM (1 KB each is reserved by the system)
            for (int srb2 = srb; srb2 >= min_srb; srb2 /= 2) {   // narrower staged rows if that is what makes two CTAs fit
                const int s2 = (int)((budget - (long)conv_tc_fixed_smem(srb2, a.bn, a.stage_bufs)) / (a.a_bytes + a.b_bytes));
                if (s2 >= 2) { a.ctas_per_sm = 2; stages = s2 > max2 ? max2 : s2; srb = srb2; break; }
            }
        }
        // A CTA alone on its SM may have two groups of epilogue warps, if three ring slots and their 128-byte staged rows fit:
        //  * pairs with a residual, always: 3x3 128 -> 256 at 64 x 76 x 76 in TF32 329 -> 306 us, 360 -> 311 under the power cap; 512 -> 2048
        //    at 256 x 7 x 7 87 -> 73
        //  * pairs of less than 32 K iterations, whose epilogue is as long as their MMAs: 3x3 128 -> 256 at 8 x 52 x 52 in bf16 25.4 -> 24.0;
        //    over 36 iterations and more the second group only disturbs (282 -> 284, 260 -> 264)
        //  * Darknet's layout, a store instruction per value: 1024 -> 255 at 64 x 19 x 19 87 -> 56
        //  * xnor layers: 256 -> 128 at 128 x 28 x 28 28.1 -> 26.6, 512 -> 256 at 14 x 14 21.0 -> 19.0
        // Other single CTAs are bound by memory (512 -> 256 at 64 x 52 x 52 in bf16 52 and 52), with a residual they want its tiles by TMA, three
        // chunks ahead (64 -> 256 at 256 x 56 x 56 342 us, 416 through this path).  DNB_TC_EPI=1: one group (pairs with a residual: two).
        const int loop = g.size * g.size * a.c_blocks, epi_knob = knobs.epi ? atoi(knobs.epi) : 2;
        const bool two = pool ? false : residual ? a.pair != 0 : epi_knob != 1 && (a.pair ? loop < 32 : nchw_out || i8);
        if (a.ctas_per_sm == 1 && two && (a.pair || !knobs.srb) && (!y_nhwc || srb == 128)) {
            const int bufs = y_nhwc ? a.stage_bufs : 0;
            const int fit = (int)((max_smem - (long)conv_tc_fixed_smem(128, a.bn, bufs)) / (a.a_bytes + a.b_bytes));
            if (fit >= 3) { a.epi_groups = 2; a.stage_bufs = bufs; stages = fit; srb = 128; }
        }
        if (a.ctas_per_sm == 1 && a.epi_groups == 1) {
            // The depth of the ring is what hides the operand loads' latency: four slots before wide staged rows.
            // The exception is a fused residual behind a short K loop, where the epilogue (one round of barrier,
            // residual wait and store per staged chunk) would outlast the tile's MMAs: fewer, wider chunks then.
            const int k_iters = g.size * g.size * a.c_blocks;
            const bool short_k_rule = knobs.shortk ? atoi(knobs.shortk) != 0 : true;
            const int short_k = bf16 ? 32 : 64;   // measured: 76x76x128 -> 256 layers want the wide rows in both modes, 38x38x256 -> 512 only in TF32
            const int want = (residual && k_iters < short_k && min_stages > 3 && short_k_rule) ? 3 : min_stages;
            for (;; srb /= 2) {
                stages = (int)((max_smem - (long)conv_tc_fixed_smem(srb, a.bn, a.stage_bufs)) / (a.a_bytes + a.b_bytes));
                if (stages >= want || srb == min_srb) break;
            }
        }
    }
    if (stages > 8) stages = 8;
    if (const char *e = knobs.stages) {
        const int v = atoi(e);
        if (v >= 2 && v <= stages) stages = v;
    }
    if (stages < 2) DNB_FAIL(DNB_ECUDA, "conv: %d bytes of shared memory are too few for the operand ring", max_smem);
    a.stages = stages;
    a.store_row_bytes = srb;
    {   // DNB_TC_WARP_STORES=1 (experiment, off): every epilogue warp stores its own 32 rows and the four warps meet once
        // per tile instead of twice per chunk.  Measured on YOLOv3-608 b64: the layers' event times drop by 0.5 %, the
        // step replayed as one CUDA graph takes 2 % longer (18.5 -> 18.9 ms), batch 8 and ResNet-50 do not move.
        const char *e = knobs.warp_stores;
        a.warp_stores = e ? (atoi(e) != 0) : 0;
    }
    // A launch that leaves SMs idle, or whose few tiles have a long K loop: one tile per cluster, K cut across it
    // (conv_tc_split.cu).  Chosen where its estimate is below the persistent kernel's, which overlaps a tile's epilogue with the
    // next one's MMAs and therefore wins once every SM has a few tiles.  DNB_TC_SPLITK: 0 never, N forces N ranges (tests).
    const int split_knob = knobs.splitk ? atoi(knobs.splitk) : -1, pair_knob = knobs.pair ? atoi(knobs.pair) : 1;
    const bool may_cut = split_knob != 0 && !pool && (i8 || !p->keep_k_order) && (split_knob > 1 || pair_knob != 2);
    // pixels of a 1x1 layer in one row: of the whole batch where nothing is stored per image
    auto flat = [&](ConvGeom sg) {
        if (sg.size == 1 && sg.stride == 1 && sg.pad == 0) {
            sg.w = sg.out_w = sg.w * sg.h * (nchw_out ? 1 : sg.batch);
            sg.h = sg.out_h = 1;
            if (!nchw_out) sg.batch = 1;
        }
        return sg;
    };
    auto cut_at = [&](const ConvGeom &at) {   // the cut launch of that geometry, no ranges where it is not cut
        const int k_iters = at.size * at.size * a.c_blocks;
        SplitQuery q;
        q.row_bytes = a.row_bytes; q.k_iters = k_iters; q.n_pad = p->n_pad; q.max_smem = max_smem;
        q.pair_ok = pair_knob > 0 && a.row_bytes == 128 && at.n % 256 == 0 && k_iters >= 16;
        q.residual = residual != nullptr;
        q.long_sum = at.c * at.size * at.size >= 8192;
        if (split_knob > 1) return choose_split(q, flat(at), split_knob < 8 ? split_knob : 8, true, at.batch);
        // decided at one image for two images also (see choose_split)
        ConvGeom dg = at;
        if (at.batch == 2) dg.batch = 1;
        TcArgs da = a;
        pick_persistent_tiles(p, knobs, dg, da, nchw_out, y_nhwc != nullptr, y_cpitch, residual != nullptr, false, true);
        SplitPlan sp = choose_split(q, flat(dg), 0, false, dg.batch);
        if (!(sp.cost < uncut_us(da, k_iters, q.residual))) sp = SplitPlan();
        else if (at.batch == 2) sp = choose_split(q, flat(at), sp.splits, false, 2);
        return sp;
    };
    const SplitPlan cut = may_cut && !a.halo ? cut_at(g) : SplitPlan();
    if (!pool && !i8 && taps_covers(p, res, nchw_out)) {
        const int whole = p->whole_batch > g.batch ? p->whole_batch : g.batch;
        ConvGeom dg = g;
        dg.batch = whole <= 2 ? 1 : whole;
        SplitPlan dcut = cut;
        TcArgs da = a;
        if (dg.batch != g.batch || a.halo) {   // (nor does the choice hang on whether this part has its weights in place)
            dcut = may_cut ? cut_at(dg) : SplitPlan();
            pick_persistent_tiles(p, knobs, dg, da, nchw_out, y_nhwc != nullptr, y_cpitch, residual != nullptr);
        }
        double others = dcut.splits ? dcut.cost : persistent_us(da.pair, da.bn, da.total_tiles, a.taps * a.c_blocks, residual != nullptr, res && res->yolo_entries);
        if (!dcut.splits && !da.pair && da.bn > 128 && da.bn <= 192) others *= 0.85;   // (that estimate is of 256 filters)
        // (the tile that it was decided with is there already, unless it is that of another batch)
        p->tc_taps = taps_pay(p, knobs, dg, dcut.splits != 0, others, res, y_nhwc != nullptr, nchw_out) &&
                     (dg.batch == g.batch || best_taps(p, knobs, g, y_nhwc != nullptr, nchw_out, residual != nullptr, res && res->yolo_entries) < 1e300);
    }
    if (p->tc_taps) DNB_TRY(build_taps_args(p, x, y_nhwc, y_cpitch));
    else if (cut.splits) DNB_TRY(build_split_args(p, x, flat(g), cut, kind, es, y_nhwc, y_cpitch, sign_out, sign_cpitch));
    if (p->tc_split || p->tc_taps) {
        p->tc_sign_out = sign_out;
        p->tc_x_ptr = x->data; p->tc_x_cpitch = x->cpitch; p->tc_y_ptr = y_nhwc; p->tc_y_cpitch = y_cpitch; p->tc_y_dtype = y_dtype;
        p->tc_res_ptr = residual; p->tc_res_cpitch = res_cpitch; p->tc_res_c = res_c; p->tc_res_stride = res_stride; p->tc_nchw_out = nchw_out ? 1 : 0; p->tc_pool = 0;
        return DNB_OK;
    }
    a.g = g;
    DNB_TRY(ensure_status(p));
    a.status = p->status;
    {
        const uint32_t box[4] = {(uint32_t)a.bk, (uint32_t)(a.halo ? a.a_pitch : a.wt), (uint32_t)(a.halo ? a.a_box_bytes / (a.a_pitch * a.row_bytes) : a.ht), (uint32_t)a.bt};
        DNB_TRY(encode_input_maps(a.tmx, g, x, kind, es, c_pad, box, a.row_bytes));
        DNB_TRY(encode_weight_map(&a.tmw, p, kind, es, c_pad, a.taps, a.bk, a.pair ? a.bn / 2 : a.bn, a.row_bytes));
    }
    if (y_nhwc && !pool) {
        const size_t opix = (size_t)y_cpitch * out_es;
        // the channel extent is the layer's own (padded to 8), the pitch whatever the tensor has: the output may be a
        // channel range of a wider tensor (a [route] output), and the boxes must not spill into its neighbour
        const int y_chan = round_up(g.n, 8) < y_cpitch ? round_up(g.n, 8) : y_cpitch;
        uint64_t dims[4] = {(uint64_t)y_chan, (uint64_t)g.out_w, (uint64_t)g.out_h, (uint64_t)g.batch};
        uint64_t strides[3] = {opix, opix * g.out_w, opix * g.out_w * g.out_h};
        uint32_t box[4] = {(uint32_t)(srb / out_es), (uint32_t)a.wt, (uint32_t)a.ht, (uint32_t)a.bt};
        DNB_TRY(encode_tensor_map(&a.tmy, bf16, 4, y_nhwc, dims, strides, box, srb));
        {   // the 32 consecutive rows of one epilogue warp: wt*ht*bt = 128 in powers of two, so they are a box too
            const int w2 = a.wt < 32 ? a.wt : 32, h2 = a.ht < 32 / w2 ? a.ht : 32 / w2, b2 = 32 / (w2 * h2);
            uint32_t wbox[4] = {(uint32_t)(srb / out_es), (uint32_t)w2, (uint32_t)h2, (uint32_t)b2};
            DNB_TRY(encode_tensor_map(&a.tmy_warp, bf16, 4, y_nhwc, dims, strides, wbox, srb));
        }
        if (residual) {
            // every res_stride-th pixel of the residual; channels it does not have are the TMA unit's zero fill
            const size_t rpix = (size_t)res_cpitch * out_es;
            const int r_chan = round_up(res_c, 8) < res_cpitch ? round_up(res_c, 8) : res_cpitch;
            const uint64_t rw = res_stride > 1 ? (uint64_t)res->res_w : (uint64_t)g.out_w, rh = res_stride > 1 ? (uint64_t)res->res_h : (uint64_t)g.out_h;
            uint64_t rdims[4] = {(uint64_t)r_chan, (uint64_t)g.out_w, (uint64_t)g.out_h, (uint64_t)g.batch};
            uint64_t rstrides[3] = {rpix * res_stride, rpix * rw * res_stride, rpix * rw * rh};
            DNB_TRY(encode_tensor_map(&a.tmr, bf16, 4, const_cast<void *>(residual), rdims, rstrides, box, srb));
        }
    }
    if (sign_out && !pool) {
        uint64_t dims[4] = {(uint64_t)sign_cpitch, (uint64_t)g.out_w, (uint64_t)g.out_h, (uint64_t)g.batch};
        uint64_t strides[3] = {(uint64_t)sign_cpitch, (uint64_t)sign_cpitch * g.out_w, (uint64_t)sign_cpitch * g.out_w * g.out_h};
        uint32_t box[4] = {32u, (uint32_t)a.wt, (uint32_t)a.ht, (uint32_t)a.bt};
        DNB_TRY(encode_tensor_map(&a.tms, 2, 4, sign_out, dims, strides, box, 32));
    }
    p->tc_sign_out = sign_out;
    p->tc_x_ptr = x->data;
    p->tc_x_cpitch = x->cpitch;
    p->tc_y_ptr = y_nhwc;
    p->tc_y_cpitch = y_cpitch;
    p->tc_y_dtype = y_dtype;
    p->tc_res_ptr = residual;
    p->tc_res_cpitch = res_cpitch;
    p->tc_res_c = res_c;
    p->tc_res_stride = res_stride;
    p->tc_nchw_out = nchw_out ? 1 : 0;
    p->tc_pool = pool ? 1 : 0;
    return DNB_OK;
}

// A tensor-core xnor layer reads its input as int8 signs.  Where the layer before it can write them as it writes its
// own f32 output (another tensor-core xnor layer, from its epilogue; a maxpool layer), the sign pass over the f32 tensor
// disappears.  conv_plan_expect_signs prepares the consumer (its operand buffer is allocated and returned; it skips its
// own pass whenever it is given `tensor`, the channels-last tensor that carries the producer's output) and
// conv_plan_link_signs also tells a producing xnor plan.  DNB_XNOR_SIGNS=0: never.
int8_t *conv_plan_expect_signs(dnb_conv_plan *consumer, const void *tensor, int batch, int c, int h, int w)
{
    const char *e = getenv("DNB_XNOR_SIGNS");
    if (e && atoi(e) == 0) return nullptr;
    if (!consumer || !tensor || consumer->kernel != K_XNOR || !consumer->xnor_tc) return nullptr;
    const ConvGeom &b = consumer->g;
    if (c != b.c || h != b.h || w != b.w || batch != b.batch || c % 32 || consumer->c_pad_i8 != c) return nullptr;
    const size_t need = (size_t)b.batch * b.h * b.w * consumer->c_pad_i8;
    if (need > consumer->x_i8_bytes) {
        cudaFree(consumer->x_i8);
        consumer->x_i8 = nullptr; consumer->x_i8_bytes = 0;
        if (cudaMalloc((void **)&consumer->x_i8, need) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        consumer->x_i8_bytes = need;
        consumer->tc_x_ptr = nullptr;
    }
    consumer->signs_given = true;
    consumer->signs_of = tensor;
    return consumer->x_i8;
}

bool conv_plan_link_signs(dnb_conv_plan *producer, dnb_conv_plan *consumer, const void *tensor, bool pooled)
{
    if (!producer || !((producer->kernel == K_XNOR && producer->xnor_tc) || (pooled && producer->stem_tc && producer->g.n == 32))) return false;   // a first layer with its maxpool writes them too
    const ConvGeom &a = producer->g;
    if (!conv_plan_expect_signs(consumer, tensor, a.batch, a.n, pooled ? a.out_h / 2 : a.out_h, pooled ? a.out_w / 2 : a.out_w)) return false;
    producer->sign_consumer = consumer;
    return true;
}

// ------------------------------------------------------------------ forward
static int check_conv_io(const dnb_conv_plan *p, const dnb_tensor *x, const dnb_tensor *y, const dnb_tensor *y2)
{
    const ConvGeom &g = p->g;
    DNB_TRY(check_tensor(x, "conv input"));
    DNB_TRY(check_tensor(y, "conv output"));
    if (y2) DNB_TRY(check_tensor(y2, "conv second output"));
    if (x->n != g.batch || x->c != g.c || x->h != g.h || x->w != g.w)
        DNB_FAIL(DNB_EINVAL, "conv: input is %dx%dx%dx%d, plan expects %dx%dx%dx%d", x->n, x->c, x->h, x->w, g.batch, g.c, g.h, g.w);
    const dnb_tensor *outs[2] = {y, y2};
    for (int i = 0; i < 2; ++i) {
        const dnb_tensor *o = outs[i];
        if (!o) continue;
        if (o->n != g.batch || o->c != g.n || o->h != g.out_h || o->w != g.out_w)
            DNB_FAIL(DNB_EINVAL, "conv: output is %dx%dx%dx%d, plan produces %dx%dx%dx%d", o->n, o->c, o->h, o->w, g.batch, g.n, g.out_h, g.out_w);
    }
    if (y2 && y2->layout == y->layout) DNB_FAIL(DNB_EINVAL, "conv: the second output must use the other layout");
    return DNB_OK;
}

struct Residual {
    const dnb_tensor *add = nullptr;
    float alpha = 1.f, beta = 1.f;
    int activation = DNB_LINEAR;
    float *keep = nullptr;
    bool pool = false;      // y is the output of the 2x2 maxpool after the convolution
    int yolo_entries = 0;   // instead of a residual: the [yolo] layer's activations, entries per anchor
};

static int conv_forward_impl(dnb_conv_plan *p, const dnb_tensor *x, const dnb_tensor *y, const dnb_tensor *y2,
                             int32_t *acc_out, cudaStream_t s, const Residual *res = nullptr)
{
    if (!p) DNB_FAIL(DNB_EINVAL, "conv: null plan");
    if (!p->params_set) DNB_FAIL(DNB_EINVAL, "conv: dnb_conv_plan_set_params has not been called");
    DNB_TRY(check_current_device(p->device, "conv"));
    const ConvGeom &g = p->g;
    void *y_nhwc = nullptr;
    float *y_nchw = nullptr;
    int y_dtype = DNB_F32, y_cpitch = 0;
    const dnb_tensor *outs[2] = {y, y2};
    for (int i = 0; i < 2; ++i) {
        const dnb_tensor *o = outs[i];
        if (!o) continue;
        if (o->layout == DNB_NHWC) { y_nhwc = o->data; y_dtype = o->dtype; y_cpitch = o->cpitch; }
        else y_nchw = (float *)o->data;
    }
    ConvEpilogue ep{p->scale, p->shift, p->d.activation, 0, nullptr, 0, DNB_LINEAR, 1.f, 1.f, 0, 0};
    if (res && res->yolo_entries > 0) {
        if (p->kernel != K_TC_TF32 && p->kernel != K_TC_BF16)
            DNB_FAIL(DNB_EUNSUPPORTED, "conv + yolo: only tensor-core plans fuse the yolo activations (this plan is %s)", kKernelNames[p->kernel]);
        ep.yolo_entries = res->yolo_entries;
    }
    if (res && res->add) {
        if (p->kernel != K_TC_TF32 && p->kernel != K_TC_BF16)
            DNB_FAIL(DNB_EUNSUPPORTED, "conv + shortcut: only tensor-core plans fuse the residual (this plan is %s)", kKernelNames[p->kernel]);
        ep.residual = res->add->data; ep.res_cpitch = res->add->cpitch; ep.activation2 = res->activation;
        ep.res_c = res->add->c; ep.res_h = res->add->h; ep.res_w = res->add->w; ep.res_stride = res->add->w / g.out_w;
        ep.res_out_h = g.out_h; ep.res_out_w = g.out_w;
        ep.alpha = res->alpha; ep.beta = res->beta;
    }
    // f32 channels-last results of a TF32 network feed the next tensor-core layer: round them once here (the tensor
    // core would truncate them instead, a bias that adds up over a network's depth).  A copy in Darknet's layout
    // written by the same launch holds the same rounded values.
    ep.round_tf32 = (p->mode == DNB_MODE_TF32 && y_nhwc && y_dtype == DNB_F32) ? 1 : 0;
    const bool pool = res && res->pool;

    if (pool && p->kernel == K_DIRECT && !(x->dtype == DNB_F32 && y_nhwc && y_cpitch == g.n)) DNB_FAIL(DNB_EINVAL, "conv + maxpool: the first layer's tensors");
    if (p->kernel == K_DIRECT && p->stem_tc && x->dtype == DNB_F32 && y_nhwc && !y_nchw && y_cpitch == g.n) {
        StemTcArgs a;
        a.x = (const float *)x->data;
        if (x->layout == DNB_NHWC) { a.xs_c = 1; a.xs_w = x->cpitch; a.xs_h = (long long)g.w * x->cpitch; a.xs_b = (long long)g.h * a.xs_h; }
        else { a.xs_w = 1; a.xs_h = g.w; a.xs_c = (long long)g.h * g.w; a.xs_b = (long long)g.c * a.xs_c; }
        a.w = p->w_direct; a.npg_pad = p->npg_pad;
        a.y = y_nhwc; a.y_dtype = y_dtype; a.y_cpitch = y_cpitch;
        DNB_TRY(ensure_status(p));
        a.status = p->status;
        a.wait_limit = p->wait_limit > 0 ? p->wait_limit : DEFAULT_WAIT_CYCLES;
        a.g = g; a.ep = ep;
        a.pool = pool ? 1 : 0;
        a.keep = pool && x->layout == DNB_NCHW ? res->keep : nullptr;
        dnb_conv_plan *const next = p->sign_consumer;
        a.signs = pool && next && y_nhwc == next->signs_of ? next->x_i8 : nullptr;
        // in the im2col order where layers take the signs of what follows from it (see conv_stem_rows.cu), else from the patch, whose
        // offsets inside an image take rows of less than 2^25 values
        const bool rows = (p->keep_k_order || a.xs_h >= (1LL << 31) / 64) && conv_stem_rows_covers(g, y_dtype);
        return rows ? launch_conv_stem_rows(a, s) : launch_conv_stem_tc(a, s);
    }
    if (on_fp32_tc(p) && x->dtype == DNB_F32 && (!y_nhwc || y_dtype == DNB_F32)) {
        Fp32TcArgs a;
        DNB_TRY(build_fp32_tc_args(p, x, y_nhwc, y_cpitch, y_nchw, ep, a));
        return launch_conv_fp32_tc(a, s);
    }
    if (p->kernel == K_DIRECT) {   // also a first-layer plan asked for Darknet's layout or given bf16 input
        DirectArgs a;
        a.x = x->data; a.x_dtype = x->dtype;
        if (x->layout == DNB_NHWC) { a.xs_c = 1; a.xs_w = x->cpitch; a.xs_h = (long long)g.w * x->cpitch; a.xs_b = (long long)g.h * a.xs_h; }
        else { a.xs_w = 1; a.xs_h = g.w; a.xs_c = (long long)g.h * g.w; a.xs_b = (long long)g.c * a.xs_c; }
        a.wpk = p->w_direct; a.npg_pad = p->npg_pad;
        a.y_nhwc = y_nhwc; a.y_dtype = y_dtype; a.y_cpitch = y_cpitch; a.y_nchw = y_nchw;
        a.in_order = p->keep_k_order ? 1 : 0;
        a.g = g; a.ep = ep;
        return launch_conv_direct(a, s);
    }
    if (p->kernel == K_XNOR && p->xnor_tc) {
        // tensor-core xnor: the input's signs as an int8 channels-last tensor (one pass over the input), then the
        // implicit-GEMM kernel in its int8 kind; out-of-image taps are the TMA unit's zero fill, i.e. they add nothing,
        // as in the reference, where the padding is applied after the binarisation (src/im2col.c:3-12)
        const size_t need = (size_t)g.batch * g.h * g.w * p->c_pad_i8;
        if (need > p->x_i8_bytes) {
            cudaFree(p->x_i8);
            p->x_i8 = nullptr; p->x_i8_bytes = 0;
            DNB_CUDA(cudaMalloc((void **)&p->x_i8, need));
            p->x_i8_bytes = need;
            p->tc_x_ptr = nullptr;
        }
        // (the xnor layer before this one, if the network linked the two, has written the signs from its epilogue)
        const bool given = p->signs_given && x->layout == DNB_NHWC && x->data == p->signs_of;
        if (!given) DNB_TRY(launch_pack_sign_i8(x, p->x_i8, p->c_pad_i8, s));
        dnb_tensor xin{p->x_i8, DNB_NHWC, DNB_F32, g.batch, g.c, g.h, g.w, p->c_pad_i8};   // dtype unused: the plan's kind says int8
        if (y_nhwc && y_dtype != DNB_F32) DNB_FAIL(DNB_EINVAL, "conv: an xnor plan writes channels-last output as f32");
        float *nchw = acc_out ? reinterpret_cast<float *>(acc_out) : y_nchw;
        void *nhwc = acc_out ? nullptr : y_nhwc;
        // signs for the next xnor layer, when this launch writes the very tensor that layer reads
        dnb_conv_plan *next = p->sign_consumer;
        void *sign_out = (next && nhwc && nhwc == next->signs_of && next->x_i8) ? next->x_i8 : nullptr;
        if (p->tc_x_ptr != xin.data || p->tc_y_ptr != nhwc || p->tc_y_cpitch != (nhwc ? y_cpitch : 0) || !p->status || p->tc_nchw_out != (nchw ? 1 : 0) ||
            p->tc_sign_out != sign_out || p->tc_pool != (pool ? 1 : 0))
            DNB_TRY(build_tc_args(p, &xin, nhwc, DNB_F32, nhwc ? y_cpitch : 0, nullptr, nchw != nullptr, sign_out, sign_out ? next->c_pad_i8 : 0, pool));
        if (p->tc_split) {
            SplitArgs &a = p->sp;
            a.y_nhwc = nhwc; a.y_cpitch = nhwc ? y_cpitch : 0; a.y_nchw = nchw;
            a.ep = ep;
            a.ep.scale = p->scale_i8; a.ep.round_tf32 = 0; a.ep.raw_acc = acc_out ? 1 : 0;
            if (acc_out) a.ep.activation = DNB_LINEAR;
            a.status = p->status;
            return launch_conv_tc_split(a, s);
        }
        TcArgs &a = p->tc;
        a.y_nhwc = nhwc; a.y_dtype = DNB_F32; a.y_cpitch = nhwc ? y_cpitch : 0; a.y_nchw = nchw;
        ep.scale = p->scale_i8;
        ep.round_tf32 = 0;
        ep.raw_acc = acc_out ? 1 : 0;
        if (acc_out) ep.activation = DNB_LINEAR;
        a.ep = ep;
        a.status = p->status;
        return launch_conv_tc(a, s);
    }
    if (p->kernel == K_XNOR) {
        const size_t need = (size_t)g.batch * g.h * g.w * p->cwords * sizeof(uint32_t);
        if (need > p->x_bits_bytes) {
            cudaFree(p->x_bits);
            p->x_bits = nullptr; p->x_bits_bytes = 0;
            DNB_CUDA(cudaMalloc((void **)&p->x_bits, need));
            p->x_bits_bytes = need;
        }
        DNB_TRY(launch_pack_sign_bits(x, p->x_bits, p->cwords, s));
        XnorArgs a;
        a.xbits = p->x_bits; a.wbits = p->w_bits; a.cwords = p->cwords; a.wmean = p->w_mean; a.acc_out = acc_out;
        a.y_nhwc = y_nhwc; a.y_dtype = y_dtype; a.y_cpitch = y_cpitch; a.y_nchw = y_nchw;
        a.g = g; a.ep = ep; a.ep.round_tf32 = 0;
        return launch_conv_xnor(a, s);
    }
    // tensor-core path: channels-last input of the plan's storage type
    const int want = p->kernel == K_TC_BF16 ? DNB_BF16 : DNB_F32;
    dnb_tensor xin = *x;
    if (x->layout == DNB_NCHW) {
        const size_t need = (size_t)g.batch * g.h * g.w * p->c_pad * elem_size(want);
        if (need > p->x_nhwc_bytes) {
            cudaFree(p->x_nhwc_scratch);
            p->x_nhwc_scratch = nullptr; p->x_nhwc_bytes = 0;
            DNB_CUDA(cudaMalloc(&p->x_nhwc_scratch, need));
            p->x_nhwc_bytes = need;
        }
        xin.data = p->x_nhwc_scratch; xin.layout = DNB_NHWC; xin.dtype = want; xin.cpitch = p->c_pad;
        DNB_TRY(launch_convert(x, &xin, want == DNB_F32, 0, 0, s));
    } else if (x->dtype != want) {
        DNB_FAIL(DNB_EINVAL, "conv: channels-last input is %s, this plan (%s) reads %s", x->dtype == DNB_BF16 ? "bf16" : "f32",
                 kKernelNames[p->kernel], want == DNB_BF16 ? "bf16" : "f32");
    }
    if (y_nhwc && y_dtype != want)
        DNB_FAIL(DNB_EINVAL, "conv: a %s plan writes channels-last output as %s", kKernelNames[p->kernel], want == DNB_BF16 ? "bf16" : "f32");
    if (p->tc_x_ptr != xin.data || p->tc_x_cpitch != xin.cpitch || p->tc_y_ptr != y_nhwc || p->tc_y_cpitch != y_cpitch ||
        p->tc_y_dtype != y_dtype || !p->status || p->tc_res_ptr != ep.residual || p->tc_res_cpitch != ep.res_cpitch ||
        (ep.residual && (p->tc_res_c != ep.res_c || p->tc_res_stride != ep.res_stride || p->tc_res_act != ep.activation2)) || p->tc_yolo != (ep.yolo_entries > 0 ? 1 : 0) ||
        p->tc_nchw_out != (y_nchw ? 1 : 0) || p->tc_pool != (pool ? 1 : 0))
        DNB_TRY(build_tc_args(p, &xin, y_nhwc, y_dtype, y_cpitch, &ep, y_nchw != nullptr, nullptr, 0, pool));
    if (p->tc_split) {
        SplitArgs &a = p->sp;
        a.y_nhwc = y_nhwc; a.y_cpitch = y_cpitch; a.y_nchw = y_nchw;
        a.ep = ep;
        a.status = p->status;
        return launch_conv_tc_split(a, s);
    }
    if (p->tc_taps) {
        TapsArgs &a = p->tp;
        a.y_nhwc = y_nhwc; a.y_cpitch = y_cpitch; a.y_nchw = y_nchw;
        a.ep = ep;
        a.status = p->status;
        return launch_conv_tc_taps(a, s);
    }
    TcArgs &a = p->tc;
    a.y_nhwc = y_nhwc; a.y_dtype = y_dtype; a.y_cpitch = y_cpitch; a.y_nchw = y_nchw;
    a.ep = ep;
    a.status = p->status;   // a network points its plans at the status word of the step being enqueued
    return launch_conv_tc(a, s);
}

extern "C" int dnb_conv_forward(dnb_conv_plan *p, const dnb_tensor *x, const dnb_tensor *y, const dnb_tensor *y2, void *stream)
{
    if (!p) DNB_FAIL(DNB_EINVAL, "conv: null plan");
    DNB_TRY(check_conv_io(p, x, y, y2));
    return conv_forward_impl(p, x, y, y2, nullptr, (cudaStream_t)stream);
}

// Convolution followed by the residual add of a [shortcut] layer, one launch:
// y = act2(alpha * act(conv(x)) + beta * add).
extern "C" int dnb_conv_shortcut_forward(dnb_conv_plan *p, const dnb_tensor *x, const dnb_tensor *add, const dnb_tensor *y,
                                         float alpha, float beta, int activation2, void *stream)
{
    if (!p || !add) DNB_FAIL(DNB_EINVAL, "conv + shortcut: null argument");
    DNB_TRY(check_conv_io(p, x, y, nullptr));
    DNB_TRY(check_tensor(add, "conv + shortcut residual"));
    if (activation2 < 0 || activation2 > DNB_SELU) DNB_FAIL(DNB_EINVAL, "conv + shortcut: activation %d", activation2);
    const int want = p->kernel == K_TC_BF16 ? DNB_BF16 : DNB_F32;
    if (add->layout != DNB_NHWC || y->layout != DNB_NHWC || add->dtype != want)
        DNB_FAIL(DNB_EINVAL, "conv + shortcut: residual and output must be channels-last in the plan's storage type");
    if (add->n != y->n || add->c != y->c || add->h != y->h || add->w != y->w)
        DNB_FAIL(DNB_EUNSUPPORTED, "conv + shortcut: the residual must have the output's extents (other shapes: dnb_shortcut_forward)");
    return conv_shortcut_general(p, x, add, y, alpha, beta, activation2, (cudaStream_t)stream);
}

// What the epilogue covers: a map that is a whole multiple of the output's, and where channels are fewer, whole staged chunks
// of them.  An addend smaller than the output (scattered with shortcut_cpu's `sample`) has its own pass.
bool conv_shortcut_fusable(const dnb_conv_plan *p, const dnb_tensor *add, const dnb_tensor *y, float alpha)
{
    if (!p || (p->kernel != K_TC_TF32 && p->kernel != K_TC_BF16)) return false;
    const int want = p->kernel == K_TC_BF16 ? DNB_BF16 : DNB_F32;
    if (add->layout != DNB_NHWC || y->layout != DNB_NHWC || add->dtype != want || y->dtype != want || add->n != y->n) return false;
    if (add->c == y->c && add->h == y->h && add->w == y->w) return true;
    const int stride = add->w / y->w;
    if (stride < 1 || add->w != stride * y->w || add->h != stride * y->h) return false;
    return add->c == y->c || (add->c < y->c && add->c % 64 == 0 && alpha == 1.f);
}

int conv_shortcut_general(dnb_conv_plan *p, const dnb_tensor *x, const dnb_tensor *add, const dnb_tensor *y, float alpha, float beta, int activation2, cudaStream_t s)
{
    DNB_TRY(check_conv_io(p, x, y, nullptr));
    DNB_TRY(check_tensor(add, "conv + shortcut residual"));
    Residual r;
    r.add = add; r.alpha = alpha; r.beta = beta; r.activation = activation2;
    return conv_forward_impl(p, x, y, nullptr, nullptr, s, &r);
}

// Convolution followed by the [yolo] layer that reads it, one launch: forward_yolo_layer_gpu at inference copies
// its input and applies the logistic to the x, y, objectness and class entries of every anchor
// (src/yolo_layer.c:347-357); here the convolution's epilogue does that and writes the [yolo] layer's NCHW output.
extern "C" int dnb_conv_yolo_forward(dnb_conv_plan *p, const dnb_tensor *x, const dnb_tensor *y, int anchors, int classes, void *stream)
{
    if (!p) DNB_FAIL(DNB_EINVAL, "conv + yolo: null plan");
    DNB_TRY(check_conv_io(p, x, y, nullptr));
    if (anchors < 1 || classes < 0 || p->g.n != anchors * (classes + 5))
        DNB_FAIL(DNB_EINVAL, "conv + yolo: %d filters are not %d anchors of %d entries", p->g.n, anchors, classes + 5);
    if (y->layout != DNB_NCHW || y->dtype != DNB_F32) DNB_FAIL(DNB_EINVAL, "conv + yolo: the output is Darknet's layout (NCHW f32)");
    if (p->d.activation != DNB_LINEAR) DNB_FAIL(DNB_EUNSUPPORTED, "conv + yolo: the convolution's own activation must be linear (as in every yolo cfg)");
    if (p->g.n % 256 == 0) DNB_FAIL(DNB_EUNSUPPORTED, "conv + yolo: %d filters (whole tiles of 256 may run as CTA pairs, which have no yolo epilogue)", p->g.n);
    Residual r;
    r.yolo_entries = classes + 5;
    return conv_forward_impl(p, x, y, nullptr, nullptr, (cudaStream_t)stream, &r);
}

// The launch that the layer would have by itself must be the persistent kernel's, in single CTAs: where it is cut along K or
// runs in pairs, small maps of deep layers, the pass that is saved is not worth another kernel (512 -> 1024 at 14 x 14, 128 images: 12 us
// of 1300).  Where it fills the GPU: 3x3 32 -> 64 at 64 x 112 x 112 in TF32 103 + 49 -> 96 us
// with the pass; three such passes of Darknet-19 with xnor layers, 128 x 224 x 224, 1352 -> 1176 us a step.
bool conv_pool_fusable(dnb_conv_plan *p, bool in_order)
{
    if (p->pool_fits) return p->pool_fits > 0;
    p->pool_fits = -1;
    const ConvGeom &g = p->g;
    const bool bf16 = p->kernel == K_TC_BF16, i8 = p->kernel == K_XNOR && p->xnor_tc;
    if (p->stem_tc) {
        const int dtype = p->mode == DNB_MODE_BF16 ? DNB_BF16 : DNB_F32;
        if (!conv_stem_pool_covers(g, dtype, p->d.activation) || g.w >= (1 << 25) || (in_order && (g.w >= (1 << 22) || !conv_stem_rows_pool_covers(g, dtype)))) return false;   // (32-bit offsets inside a tile's patch)
        p->pool_fits = 1;
        return true;
    }
    if (p->kernel != K_TC_TF32 && !bf16 && !i8) return false;
    if (p->d.activation != DNB_LEAKY || g.out_h % 2 || g.out_w % 2 || g.n * (bf16 ? 2 : 4) < 128 || g.n % 8) return false;
    const Knobs knobs;
    TcArgs a;
    const int es = i8 ? 1 : bf16 ? 2 : 4, c_pad = i8 ? p->c_pad_i8 : p->c_pad;
    a.row_bytes = c_pad * es >= 128 ? 128 : c_pad * es >= 64 ? 64 : 32;
    a.bk = a.row_bytes / es;
    a.c_blocks = (c_pad + a.bk - 1) / a.bk;
    pick_persistent_tiles(p, knobs, g, a, false, true, g.n, false);
    const int k_iters = g.size * g.size * a.c_blocks;
    if (a.pair || a.total_tiles < (k_iters <= 12 ? sm_count() / 2 : sm_count())) return false;
    p->pool_fits = 1;
    return true;
}

int conv_pool_forward(dnb_conv_plan *p, const dnb_tensor *x, const dnb_tensor *y, float *keep, cudaStream_t s)
{
    const ConvGeom &g = p->g;
    DNB_TRY(check_tensor(x, "conv + maxpool input"));
    DNB_TRY(check_tensor(y, "conv + maxpool output"));
    if (x->n != g.batch || x->c != g.c || x->h != g.h || x->w != g.w || y->n != g.batch || y->c != g.n || y->h != g.out_h / 2 || y->w != g.out_w / 2 || y->layout != DNB_NHWC)
        DNB_FAIL(DNB_EINVAL, "conv + maxpool: extents or layout");
    Residual r;
    r.pool = true;
    r.keep = keep;
    return conv_forward_impl(p, x, y, nullptr, nullptr, s, &r);
}

extern "C" int dnb_conv_xnor_accumulate(dnb_conv_plan *p, const dnb_tensor *x, int32_t *acc, void *stream)
{
    if (!p || !acc) DNB_FAIL(DNB_EINVAL, "xnor accumulate: null argument");
    if (p->kernel != K_XNOR) DNB_FAIL(DNB_EINVAL, "xnor accumulate: the plan is not an xnor plan");
    DNB_TRY(check_tensor(x, "conv input"));
    const ConvGeom &g = p->g;
    if (x->n != g.batch || x->c != g.c || x->h != g.h || x->w != g.w) DNB_FAIL(DNB_EINVAL, "xnor accumulate: input extents differ from the plan");
    return conv_forward_impl(p, x, nullptr, nullptr, acc, (cudaStream_t)stream);
}

// Device status word of the tensor-core kernel: 0, or the code of the bounded
// wait that expired (DNB_ETIMEOUT is returned to the caller in that case).
extern "C" int dnb_conv_plan_check_status(dnb_conv_plan *p)
{
    if (!p || !p->status) return DNB_OK;
    int v = 0;
    DNB_CUDA(cudaMemcpy(&v, p->status, sizeof(int), cudaMemcpyDeviceToHost));
    if (v) {
        cudaMemset(p->status, 0, sizeof(int));
        DNB_FAIL(DNB_ETIMEOUT, "conv: a device-side wait expired (code %d: 101 ring slot free, 102 operands landed, 103 accumulator free, 104 accumulator ready, 105 residual tile, 106 shared memory window not 1024-byte aligned)", v);
    }
    return DNB_OK;
}
