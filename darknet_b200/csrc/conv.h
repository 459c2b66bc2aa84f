// Internal argument blocks of the convolution kernels and the plan object.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include <vector>

#include "common.h"

namespace dnb {

// Default bound of the kernels' device-side waits: about one second of SM clock cycles.
constexpr long long DEFAULT_WAIT_CYCLES = 2000000000LL;

// ---- conv_direct.cu
struct DirectArgs {
    const void *x;                       // input, any layout through element strides
    int x_dtype;
    long long xs_b, xs_c, xs_h, xs_w;    // element strides of x
    const float *wpk;                    // weights [groups][K][npg_pad], K = c/groups*size*size
    int npg_pad;                         // filters per group rounded up to 32
    void *y_nhwc;                        // optional NHWC output
    int y_dtype, y_cpitch;
    float *y_nchw;                       // optional NCHW f32 output
    int in_order;                        // add the products in the order c, kh, kw whatever the layout (keep_k_order)
    ConvGeom g;
    ConvEpilogue ep;
};
int launch_conv_direct(const DirectArgs &a, cudaStream_t s);

// ---- conv_stem_tc.cu : first layer (3x3 over at most 3 channels, 5x5 and 7x7 over RGB) on tcgen05, rows read straight from the image's patch
struct alignas(64) StemTcArgs {
    CUtensorMap tmy;                     // channels-last output, boxes of 8 x 4 pixels and one row segment
    int seg_bytes, segs;                 // a pixel's output row in segments of 32, 64 or 128 bytes
    const float *x;                      // f32 input, any layout through element strides
    long long xs_b, xs_c, xs_h, xs_w;
    const float *w;                      // weights [K][npg_pad], K = c*9 (the direct kernel's packing)
    int npg_pad;
    void *y;                             // channels-last output, pitch == n
    int y_dtype, y_cpitch;
    int n_pad, tmem_cols, tiles, tiles_w, tiles_h;   // filled by the launcher
    int pool;                            // 1: y is the 2x2 stride-2 maxpool's output
    float *keep;                         // pooled output: where a copy of the images (Darknet's layout) goes, or null
    int8_t *signs;                       // pooled output of conv_stem_rows.cu: its signs, 32 bytes a pixel, or null
    int npix, tma_store;                 // ... of conv_stem_rows.cu: output pixels; rows leave through tmy (else plain stores)
    int *status;
    long long wait_limit;                // bound of every device-side wait, SM clock cycles
    ConvGeom g;
    ConvEpilogue ep;
};
bool conv_stem_tc_covers(const ConvGeom &g);
bool conv_stem_pool_covers(const ConvGeom &g, int y_dtype, int activation);
int launch_conv_stem_tc(StemTcArgs a, cudaStream_t s);

// ---- conv_stem_rows.cu : the same layers with their products added in the im2col order (networks with xnor layers)
bool conv_stem_rows_covers(const ConvGeom &g, int y_dtype);
bool conv_stem_rows_pool_covers(const ConvGeom &g, int y_dtype);
int launch_conv_stem_rows(StemTcArgs a, cudaStream_t s);

// The shared memory that a CTA with `cols` columns of TMEM asks for: its `bytes`, or its columns' share of the SM's (228 KB, 1 KB of
// it reserved per CTA, against 512 columns) if that is more.  Whatever CTAs then meet on an SM, of this kernel or another one,
// of this stream or another one, their columns fit together and no tcgen05.alloc ever waits.  One that waits can wait
// for good: a CTA of a cluster keeps its columns until its peers are done, so clusters of two networks on two streams, each holding
// what a peer of the other waits for on another SM, would never end, and no bounded wait covers an allocation.
size_t tmem_smem(size_t bytes, int cols);

// ---- conv_tc.cu : implicit GEMM on tcgen05 / TMEM, operands by TMA
struct alignas(64) TcArgs {
    CUtensorMap tmx[4];   // activation maps: one per (row parity, column parity) lattice of a strided conv
    CUtensorMap tmw;      // weights [taps][n_pad][c_pad], channels innermost
    CUtensorMap tmy;      // NHWC output, written by TMA stores from the staging rows
    CUtensorMap tmr;      // fused residual (tmy's box over the pixels that are added), loaded tile by tile in the epilogue
    CUtensorMap tmy_warp; // the same output as 32-pixel boxes: the rows one epilogue warp stages (per-warp stores)
    CUtensorMap tms;      // sign output (int8 channels-last, the next xnor layer's operand): 32-channel boxes of the same pixels as tmy
    int is_bf16;          // operand kind: 0 kind::tf32 on f32 operands, 1 kind::f16 on bf16 operands, 2 kind::i8 on int8 sign tensors (xnor)
    int row_bytes;        // bytes of channels per pipeline stage row: 128, 64 or 32 (= swizzle span)
    int bk;               // channels per stage row (row_bytes / element size)
    int c_blocks;         // ceil(c_pad / bk)
    int taps;             // size*size
    int bn;               // filters per tile: multiple of 16, <= 256
    int n_tiles;          // ceil(n / bn)
    int wt, ht, bt;       // output pixels per tile along w, h, batch; wt*ht*bt == 128
    int tiles_w, tiles_h, tiles_b;
    int total_tiles;      // n_tiles * tiles_w * tiles_h * tiles_b
    int stages;           // depth of the shared-memory ring
    // Halo mode (3x3, padding 1, one filter tile, tiles of 8 x 16 pixels): the layer's weights stay in shared memory, and ONE box of (8+2) x (16+2)
    // pixels per channel block (stride 2: of 9 x 17 of each of the four lattices) serves all nine taps: the MMA's A descriptor starts at row
    // kh*10 + kw of the box, its 8-row groups are 10 rows apart.  A tile then asks for a tenth of the rows it did, tap by tap
    // and with its weights.  `stages` tiles' boxes are a ring of a_slot bytes each.
    int halo, a_slot, a_box_slot, a_box_bytes, a_pitch;
    int tmem_cols;        // TMEM columns the CTA allocates: a power of two >= 2*bn (two accumulators)
    int debug;            // timing experiments only (DNB_TC_DEBUG): 1 no residual loads, 2 no output stores, 4 no wait before a residual request (one group), 8 empty epilogue, 16 no MMAs;
                          // 32 (dnb_conv_plan_set_diagnostics): each CTA withholds the last operand load of its first tile, so a bounded wait runs out
    long long wait_limit; // bound of every device-side wait, SM clock cycles
    int stage_bufs;       // staging buffers of the epilogue: 2, or 4 with a fused residual (it lands in them first), 3 with signs, 0 where two groups write Darknet's layout only
    int pair;             // 1: clusters of two CTAs share every MMA (cta_group::2); total_tiles then counts PAIRS of pixel tiles,
                          // b_bytes and the weight map's box cover half a filter tile, bn is 128 or 256
    int ctas_per_sm;      // 2 for narrow tiles (TMEM and shared memory are sized so that two CTAs share an SM), up to 4 for pooled ones, else 1
    int pool;             // 1: y_nhwc (and sign_out) are the 2x2 stride-2 maxpool's output, plain stores; wt and ht are even, wt at most 16
    int epi_groups;       // groups of four epilogue warps: 2 where a CTA has its SM to itself and staged rows are 128 bytes, else 1
    int a_bytes, b_bytes; // shared-memory bytes of one stage's activation / weight tile (1024-multiples)
    int store_row_bytes;  // bytes of one staged output row (128, 64 or 32) = swizzle span of tmy
    int n_pad;            // length of the scale / shift vectors
    int n_tot;            // n_tiles * bn rounded up: entries of the shared scale / shift copies
    void *y_nhwc;
    int y_dtype, y_cpitch;
    float *y_nchw;
    int *status;          // device word: 0, or the code of the wait that expired
    int warp_stores;      // one group, 1: every epilogue warp stores its own 32 rows (tmy_warp); 0: one store per chunk by one thread (tmy)
    void *sign_out;       // int8 kind: also write the output's signs here ([b][h][w][sign_cpitch] bytes), or null
    int sign_cpitch;
    ConvGeom g;
    ConvEpilogue ep;
};
int launch_conv_tc(const TcArgs &a, cudaStream_t s);
size_t conv_tc_smem_bytes(const TcArgs &a);
size_t conv_tc_fixed_smem(int store_row_bytes, int bn, int stage_bufs);
int conv_tc_max_smem();

// ---- conv_tc_split.cu : the same convolution for launches that do not fill the GPU, one tile per cluster, K cut across it
struct alignas(64) SplitArgs {
    CUtensorMap tmx[4];   // as in TcArgs; boxes of wt x ht x bt pixels
    CUtensorMap tmw;
    int kind;             // 0 tf32, 1 bf16, 2 int8 signs
    int pair;             // clusters of 2 * splits CTAs working in pairs; tiles then counts PAIRS of pixel tiles
    int splits;           // K ranges = CTAs (pairs) per tile, 2..8
    int tiles;            // output tiles = clusters
    int row_bytes, bk, c_blocks, taps, bn, n_tiles;
    int wt, ht, bt, rows; // a tile's pixels, rows = wt*ht*bt <= 128
    int tiles_w, tiles_h;
    int stages, a_bytes, b_bytes;
    int work_bytes;       // ring or accumulator dump, whichever is larger
    int tmem_cols;        // power of two >= bn
    int n_write;          // channels written: n rounded to 8 for channels-last output, n for Darknet's layout alone
    void *y_nhwc;
    int y_cpitch;
    float *y_nchw;
    void *sign_out;
    int sign_cpitch;
    int *status;
    int debug;
    long long wait_limit;
    ConvGeom g;
    ConvEpilogue ep;
};
int launch_conv_tc_split(const SplitArgs &a, cudaStream_t s);
size_t conv_tc_split_smem(int stages, int stage_bytes, int bn, int *work_bytes);
int conv_tc_split_resident(int pair, int cluster);

// ---- conv_tc_taps.cu : 3x3 layers with stride 1 in CTA pairs, one load of pixels for all nine taps
constexpr int TAPS_MAX_X = 6, TAPS_MAX_W = 36;
struct alignas(64) TapsArgs {
    CUtensorMap tmx;      // im2col map: the input with a column of zeros before each row and a row of zeros before each image
    CUtensorMap tmw;      // weights, half a filter tile of 128 bytes of channels
    int bf16;             // operands and channels-last output bf16, else f32 (TF32 products)
    int taps, pixels;     // 9, or 1 (1x1 layers); of those the pixels of the whole batch
    int bk, c_blocks;     // channels of a block (128 bytes), blocks
    int bn, n_tiles;      // filters per tile, a multiple of 32
    int boxes;            // 1: tiles are boxes of 8 x 16 pixels, a load one of 10 x 18, by tiles_w and tiles_h of an image; 0: 128 positions in a row
    int tiles_w, tiles_h;
    int pitch, rows;      // positions of a row (w + 1, of a box 10); of a tile's load (128 + 2 * pitch + 2, of a box 180)
    int ptiles;           // pixel tiles
    int total_tiles;      // pairs of them times n_tiles
    int x_stages, x_slot; // ring of pixel boxes, bytes of one
    int w_stages, w_bytes;// ring of filter tiles
    int resident;         // 1: the ring holds all of the layer's filters, loaded once
    int staged_bytes;     // rows of the eight epilogue warps: 4 KB each, 12 with a residual, none for Darknet's layout alone
    int table;            // entries of the scale and shift tables in shared memory
    int tmem_cols, n_pad;
    int y_chan;           // channels written to y_nhwc
    void *y_nhwc;
    int y_cpitch;
    float *y_nchw;
    int *status;
    int debug;
    long long wait_limit;
    ConvGeom g;
    ConvEpilogue ep;
};
int launch_conv_tc_taps(const TapsArgs &a, cudaStream_t s);
size_t conv_tc_taps_smem(const TapsArgs &a);
size_t conv_tc_taps_fixed_smem(const TapsArgs &a);   // what its rings leave

// ---- conv_fp32_tc.cu : fp32 convolution by three bf16 parts of every operand on the tensor cores, sums in fp32 registers
struct alignas(64) Fp32TcArgs {
    CUtensorMap tmx[4];   // as in TcArgs; boxes of 32 channels x wt x ht x bt pixels
    CUtensorMap tmy;      // channels-last output, boxes of 32 channels (16 where bn is 32) and the tile's pixels
    CUtensorMap tmw;      // [c_blocks*taps][3][n_pad][32]: the weights' three parts
    int c_blocks, taps, last_slices;   // last_slices: MMAs of 16 channels in the last block of 32
    int bn, n_tiles;      // filters per tile: 32, 64 or 128
    int wt, ht, bt, tiles_w, tiles_h, total_tiles;
    int n_pad;
    const float *x;       // the input and its element strides (planes, and sums that are added up again)
    long long xs_b, xs_c, xs_h, xs_w;
    int planes;           // 1: the input is a Darknet tensor, no tmx
    uint32_t smallest;    // bits of the smallest input, but zero, that the parts stand for
    const float *w;       // the CUDA-core kernel's weights
    int npg_pad;
    float *y_nhwc, *y_nchw;
    int *status;
    int debug;
    long long wait_limit;
    ConvGeom g;
    ConvEpilogue ep;
};
int launch_conv_fp32_tc(const Fp32TcArgs &a, cudaStream_t s);

// cuTensorMapEncodeTiled through the runtime's driver entry point (no libcuda link).
int encode_tensor_map(CUtensorMap *map, int elem_kind /* 0 f32, 1 bf16, 2 bytes */, int rank, void *base, const uint64_t *dims,
                      const uint64_t *strides_bytes /* rank-1 */, const uint32_t *box, int swizzle_bytes);

// Map for loads in im2col mode of an NHWC tensor: `rows` pixels of `chan` channels (128 bytes, 128-byte swizzle) along the bounding box that has one column
// before each row and one row before each image.
int encode_im2col_map(CUtensorMap *map, int elem_kind, void *base, const uint64_t *dims, const uint64_t *strides_bytes, uint32_t chan, uint32_t rows);

// ---- conv_xnor.cu : bit-packed popcount GEMM
struct XnorArgs {
    const uint32_t *xbits;   // [b][h][w][cwords] sign bits of the input (1 = x > 0)
    const uint32_t *wbits;   // [n][taps][cwords] sign bits of the weights (1 = w > 0)
    int cwords;              // ceil(c / 32); unused high bits are 0 in both operands
    const float *wmean;      // [n] mean |w| per filter
    int32_t *acc_out;        // optional NCHW int32 accumulators
    void *y_nhwc;
    int y_dtype, y_cpitch;
    float *y_nchw;
    ConvGeom g;
    ConvEpilogue ep;
};
int launch_conv_xnor(const XnorArgs &a, cudaStream_t s);
// sign bits of an NHWC (f32/bf16) or NCHW f32 tensor into [b][h][w][cwords]
int launch_pack_sign_bits(const dnb_tensor *x, uint32_t *bits, int cwords, cudaStream_t s);
// signs of the same tensors as int8 (+1 where x > 0, else -1; 0 in the padding channels) into [b][h][w][cpad], cpad a
// multiple of 32: the operand of the tensor-core xnor convolution
int launch_pack_sign_i8(const dnb_tensor *x, int8_t *out, int cpad, cudaStream_t s);

}  // namespace dnb

// The plan object behind the C ABI.
struct dnb_conv_plan {
    dnb_conv_desc d;
    int mode;
    int kernel;              // 0 tc_tf32, 1 tc_bf16, 2 direct_fp32, 3 xnor_popc
    dnb::ConvGeom g;
    int n_pad;               // filters rounded up to 16
    int c_pad;               // input channels rounded up to 8 (cpitch the kernel expects of NHWC input)
    bool params_set;
    bool stem_tc;            // a direct plan whose channels-last f32-input launches use the tensor-core first-layer kernel
    // derived device tensors
    float *scale, *shift;    // [n_pad] folded batchnorm / bias
    void *w_tc;              // [taps][n_pad][c_pad] f32 (TF32-rounded) or bf16
    float *w_direct;         // [groups][K][npg_pad]
    __nv_bfloat16 *w_parts;  // [c_blocks][taps][3][n_pad][32]: the weights' three bf16 parts (full-precision plans on the tensor cores)
    uint32_t *w_bits;        // [n][taps][cwords]
    float *w_mean;           // [n]
    int npg_pad, cwords;
    // scratch owned by the plan
    void *x_nhwc_scratch;    // NHWC copy of an NCHW input handed to a tensor-core plan
    size_t x_nhwc_bytes;
    uint32_t *x_bits;        // packed input of an xnor plan
    size_t x_bits_bytes;
    // xnor on the tensor cores (kind::i8): int8 sign tensors instead of packed bits
    bool xnor_tc;            // this xnor plan runs the tensor-core kernel (DNB_XNOR_TC=0 keeps the popcount kernel)
    int c_pad_i8;            // input channels rounded up to 32
    int8_t *w_i8;            // [taps][n_pad][c_pad_i8] signs of the weights
    float *scale_i8;         // [n_pad] mean|w| * folded batchnorm scale
    int8_t *x_i8;            // int8 signs of the input, scratch
    size_t x_i8_bytes;
    int *status;             // device status word of the tensor-core kernel
    bool borrowed;           // the parameter tensors belong to another plan (conv_plan_for_batch)
    bool status_shared;      // the word belongs to a network object (one word for all its plans)
    // tensor-core launch block, rebuilt when the input pointer changes
    dnb::TcArgs tc;
    const void *tc_x_ptr;
    int tc_x_cpitch;
    const void *tc_y_ptr;    // NHWC output the store map was built for
    const void *tc_res_ptr;  // fused residual the load map was built for (NULL: none)
    int tc_res_cpitch, tc_res_c, tc_res_stride, tc_res_act;
    int tc_yolo;             // the cached launch block was built for a launch with a [yolo] layer's logistic
    int tc_y_cpitch, tc_y_dtype;
    // xnor layers in a row (tensor-core kind): the producer's epilogue writes the consumer's int8 operand
    dnb_conv_plan *sign_consumer;   // this plan also fills that plan's x_i8 (set by the network object), or null
    bool signs_given;               // this plan's x_i8 is filled by the layer before it: no sign pass of its own
    const void *signs_of;           // ... as long as the input it is given is this tensor
    void *tc_sign_out;              // the sign output the cached launch block was built for
    bool keep_k_order;       // sum K in one order whatever the batch (dense layers of a network with xnor layers): no split, first layers in the im2col order
    bool tc_split;           // launches use the one-tile-per-cluster kernel and its block below
    dnb::SplitArgs sp;
    bool tc_taps;            // ... or conv_tc_taps.cu and its block
    dnb::TapsArgs tp;
    int whole_batch;         // of the plan that this one is a part of (see taps_pay), its own otherwise
    bool tap_order;          // sums over taps, then blocks of channels, on whichever kernel: not conv_tc_taps.cu
    bool status_in_block;    // the status word lies behind the weights
    bool fp32_tc;            // this full-precision plan's layer is one that conv_fp32_tc.cu is made for
    uint32_t fp32_smallest;  // ... its smallest input (see there), or 0 where its weights keep it on the CUDA cores
    int tc_pool;             // the cached launch block writes the pooled output
    int pool_fits;           // conv_pool_fusable's answer: 0 not asked yet, 1 yes, -1 no
    int tc_nchw_out;         // the cached launch block was built for a launch that also writes Darknet's layout
    int device;
    long long wait_limit;    // bound of the kernels' waits in cycles (0: the default, about one second)
    int debug_bits;          // OR-ed into the launch block's debug field (dnb_conv_plan_set_diagnostics)
};

// dnb_conv_shortcut_forward with an addend that may have fewer channels and a map that is a whole multiple of the output's
bool conv_shortcut_fusable(const dnb_conv_plan *p, const dnb_tensor *add, const dnb_tensor *y, float alpha);
int conv_shortcut_general(dnb_conv_plan *p, const dnb_tensor *x, const dnb_tensor *add, const dnb_tensor *y, float alpha, float beta, int activation2, cudaStream_t s);

// Convolution and the 2x2 maxpool with stride 2 after it in one launch (first-layer or persistent tensor-core kernel, leaky activation, even maps): y is the
// maxpool's output.  conv_pool_fusable: whether the layer is one of those, and its launch one that fills the GPU.
// in_order: the layer will be one of a network with xnor layers.
bool conv_pool_fusable(dnb_conv_plan *p, bool in_order);
// keep: a first layer also copies its input, a Darknet tensor, there (null: it does not).
int conv_pool_forward(dnb_conv_plan *p, const dnb_tensor *x, const dnb_tensor *y, float *keep, cudaStream_t s);

dnb_conv_plan *conv_plan_for_batch(const dnb_conv_plan *p, int batch);

// producers of a tensor-core xnor layer's int8 operand (see conv_plan.cu)
int8_t *conv_plan_expect_signs(dnb_conv_plan *consumer, const void *tensor, int batch, int c, int h, int w);
bool conv_plan_link_signs(dnb_conv_plan *producer, dnb_conv_plan *consumer, const void *tensor, bool pooled = false);
