// Host-side launch interface of the CUDA kernels (internal to the library).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <vector>
#include "common.cuh"

namespace n2d2b {

struct ConvGeom {
    int B, H, W, C;      // input, NHWC
    int oH, oW, O;       // output, NHWC
    int kH, kW, sY, sX, pT, pL, dY, dX;
    int groups, Cg, Og;  // channels / outputs per group
};

struct PoolGeom {
    int B, H, W, C, oH, oW;
    int pH, pW, sY, sX, padY, padX;
    int is_max;
};

struct SumInputs {
    const void* ptr[4];
    int dtype[4];
    int is_unsigned[4];
    int n;
};

// Fused residual: after the cell's own requantisation t, out = requant2(t + res)
struct Residual {
    const void* ptr;   // int8 NHWC, same shape as the output; nullptr = none
    int is_unsigned;
    QuantDev q2;
};

// CUDA-core direct convolution (any geometry, groups, dilation); weights OHWI int8.
cudaError_t launch_conv_direct(const void* in, int in_unsigned, const int8_t* w, const ConvGeom& g,
                               const QuantDev& q, const Residual& r, void* out, int out_dtype,
                               cudaStream_t s);
// Depthwise convolution, C % 16 == 0; weights re-laid as [kH][kW][C].
struct FastQuant;
// `fast` (when enabled): the proved 32-bit rescale; 3x3 filters then take the dot-product kernel
cudaError_t launch_conv_depthwise(const void* in, int in_unsigned, const int8_t* w_hwc, const ConvGeom& g,
                                  const QuantDev& q, const FastQuant& fast, void* out, cudaStream_t s);
// 3x3 depthwise layers, stride 1 or 2, on the 32-bit or floating-point epilogue
// Bytes on which the input of launch_conv_depthwise has to start: the widest load of the kernel it takes
int depthwise_alignment(const ConvGeom& g, const FastQuant& fast);
bool depthwise3x3_eligible(const ConvGeom& g);
cudaError_t launch_depthwise3x3(const void* in, int in_unsigned, const int8_t* w_hwc, const ConvGeom& g, const FastQuant& fast, void* out,
                                int num_sms, cudaStream_t s);
cudaError_t launch_pool(const void* in, int in_unsigned, const PoolGeom& g, void* out, cudaStream_t s);
cudaError_t launch_pool_i32(const void* in, const PoolGeom& g, void* out, cudaStream_t s);
cudaError_t launch_elemwise_sum(const SumInputs& ins, size_t pixels, int C, const QuantDev& q,
                                void* out, int out_dtype, cudaStream_t s);
// Stand-alone rescale of int32 [pixels][C] to 8 bits.  words: host constants, [5][C] of the 32-bit form (form 0, with valid
// clamps) or the floating-point form (1), or [7][C] bias, p0, p1, fscale, clip_thr, clip_val, clip_f (form 2, exact 64-bit);
// q: the scalar fields of QuantDev (its pointers are not used)
cudaError_t launch_rescale_i32(const int32_t* in, void* out, size_t pixels, int C, int form, const int32_t* words, const QuantDev& q,
                               cudaStream_t s);
// Top-1 class per pixel (first maximum wins) of [pixels][C] scores; values may be nullptr.
// [rows][ld] bytes -> [rows][C] bytes (C <= ld): drops the zero columns a padded cell computed
cudaError_t launch_drop_padded_columns(const uint8_t* src, int ld, uint8_t* dst, int C, size_t rows, cudaStream_t s);
// labels / values: [images][topN][hw]; pixels = images * hw score vectors of C entries; C <= 16384
cudaError_t launch_topn(const void* scores, int dtype, int is_unsigned, size_t pixels, size_t hw, int C, int topN, int32_t* labels,
                        int32_t* values, cudaStream_t s);
cudaError_t launch_argmax(const void* scores, int dtype, int is_unsigned, size_t pixels, int C, int32_t* labels, int32_t* values,
                          cudaStream_t s);
// Float stimuli NCHW -> trunc(x * factor) clamped to [lo, hi], 8-bit NHWC.
cudaError_t launch_quantize_stimuli(const float* in, int B, int C, int H, int W, float factor, int lo, int hi, void* out, cudaStream_t s);
// Fully connected on CUDA cores: in [B][K], w [O][K] int8.
cudaError_t launch_fc_direct(const void* in, int in_unsigned, const int8_t* w, int B, int K, int O,
                             const QuantDev& q, void* out, int out_dtype, cudaStream_t s);

// Per-channel constants of the 32-bit epilogue y = (clamp(acc, lo, hi) * mult + add) >> shift, which is
// exact whenever the host could bound every intermediate to 32 bits (see build_fast_quant in net.cu).
struct FastQuant {
    const int* fq = nullptr;    // [5][cpad]: lo, hi, mult, add, shift of the cell
    const int* fq2 = nullptr;   // the same for a fused residual sum
    int cpad = 0;
    int t_lo = 0, t_hi = 0;     // range the cell's own output saturates to
    int out_unsigned = 0;       // final 8-bit range
    bool need_clamp = true;     // false: no product can leave 32 bits and saturation is the final pack's
    int form = 0;               // EF_WIDE: first rescale in 64 bits, row 0 of fq holds the upper words of the addends, row 1 the bound
                                // of the rescaled value (with need_clamp: values are clamped to [0, bound]);
                                // EF_FLOAT: floating-point scaling (both stages of a residual cell); 0: the 32-bit form
    bool dp4a = false;          // residual stage as a byte dot product (multipliers <= 255, native 8-bit ranges)
    bool dp_t_unsigned = false; //   the cell's own output is packed as unsigned bytes (natively, or shifted by +128)
    int dp_a_signed = 1;        //   signedness of the (t, r) byte vector
    bool unit_multiplier = false;   // every multiplier of the cell's own 32-bit rescale is 1
    bool monotone = false;      // no multiplier of the cell's own rescale is negative: it never decreases
    bool enabled = false;
};

// ---- stride-2 first layer through space-to-depth (tcgen05 kind::i8, no gather) ----
struct StemS2dPlan {
    CUtensorMap tmA;      // re-laid image [B][Hs][Ws][16] as (8-byte words, rows, images); box = one band
    const int8_t* w;      // weights in the canonical unswizzled K-major layout (device)
    int BN, KH, KWp, Wp;
    int R, bands;
    int row_stride;       // convolution rows between bands
    int pool_k, pool_s, P, pool_oH, pool_oW;   // fused max pooling (P = pooled rows per band; 0 = none)
    int cbuf_alloc;       // bytes of one band-sized output buffer of the fused pooling
    int band_bytes, band_alloc, w_bytes;
    int in_unsigned;
    int num_sms;
    int band_batch;       // images the band height was chosen for
    int late_layer;       // weights and constants are written by the kernel before
    const void* s2d;      // the re-laid image
    int max_batch;
    void* encode;         // cuTensorMapEncodeTiled
    size_t smem_bytes;
};
// Chooses the band height for a call of `batch` images (a no-op when it is the plan's already)
int stem_s2d_set_batch(StemS2dPlan* plan, const ConvGeom& g, int batch);
bool stem_s2d_eligible(const ConvGeom& g);
bool stem_s2d_pool_eligible(const ConvGeom& g, const PoolGeom& p);
void stem_s2d_dims(const ConvGeom& g, int* Hs, int* Ws);
// Image shift, filter rows and (even) filter columns after space-to-depth
void stem_s2d_filter(const ConvGeom& g, int* P, int* KH, int* KWp);
size_t stem_s2d_weight_bytes(const ConvGeom& g);
void stem_s2d_arrange_weights(const ConvGeom& g, const int8_t* w_ohwi, int8_t* dst);
cudaError_t launch_s2d_image(const void* in, const ConvGeom& g, int batch, void* out, cudaStream_t s);
// The layer as parameters of the kernel that re-lays the image; weights OHWI, constants [5][O]
struct S2dLayer {
    int O, kH, kW, C, offy, offx, KH, KWp, BN, blocks;
    int8_t* w_dst;
    int* const_dst;       // [5][256]
    int consts[5 * 128];
    int8_t w[28 * 1024];
};
static_assert(sizeof(S2dLayer) <= 32000, "kernel parameters end at 32764 bytes");
cudaError_t launch_s2d_layer_and_image(S2dLayer* l, const void* in, const ConvGeom& g, int batch, void* out, cudaStream_t s);
// pool: a max pooling folded into the kernel (stem_s2d_pool_eligible); `out` of the launch is then the pooled tensor
int stem_s2d_make_plan(StemS2dPlan* plan, const void* d_s2d, const int8_t* d_w_arranged, const ConvGeom& g, int max_batch,
                       int in_unsigned, int num_sms, const char** why, const PoolGeom* pool = nullptr);
cudaError_t launch_stem_s2d(const StemS2dPlan& plan, const ConvGeom& g, int n_base, const FastQuant& fast, void* out,
                            int* status_word, cudaStream_t s);

// ---- stride-2 first layer of 64 channels with the 3x3 / 2 max pooling behind it (monotone rescales only) ----
struct StemPoolPlan {
    CUtensorMap tmX;      // re-laid image as (8-byte words, rows, images); box = two rows
    const int8_t* w;
    int KH, KWp, Wp, w_bytes, poH, poW, in_unsigned, num_sms;
    size_t smem_bytes;
};
bool stem_pool_eligible(const ConvGeom& g, const PoolGeom& p);
size_t stem_pool_weight_bytes(const ConvGeom& g);
void stem_pool_arrange_weights(const ConvGeom& g, const int8_t* w_ohwi, int8_t* dst);
int stem_pool_make_plan(StemPoolPlan* plan, const void* d_s2d, const int8_t* d_w_arranged, const ConvGeom& g, const PoolGeom& p, int max_batch,
                        int in_unsigned, int num_sms, const char** why);
bool stem_pool_takes_image(const StemPoolPlan& plan, const ConvGeom& g, const void* in);
cudaError_t launch_stem_pool(const StemPoolPlan& plan, const ConvGeom& g, int n_base, const void* raw, const FastQuant& fast, void* out, int* status_word,
                             cudaStream_t s);

// ---- stride-1 convolution from a shared-memory input patch (tcgen05 kind::i8) ----
struct PatchPlan {
    CUtensorMap tmA;      // NHWC activations, box = one patch: C x Wp x (R + halo rows) x 1 image
    CUtensorMap tmB;      // weights [O][taps*C], box = one tap of all outputs
    int BN;               // accumulator columns: 64 or 128
    int Wp;               // patch width in pixels: oW + (kW-1)*dX
    int R, bands;         // output rows per band, bands per image
    int patch_bytes;      // bytes of one patch load
    int patch_alloc;      // bytes reserved per patch buffer
    int b_stream;         // weights stream through a ring (too large to stay resident)
    int bring;            // slots of that ring (one filter tap each)
    int nbuf;             // patch buffers
    int in_unsigned;
    int num_sms;
    int late_weights;     // the weights are the previous kernel's output (see IgemmPlan)
    int G;                // channel groups: 1, or the block-diagonal groups of a depthwise layer
    const void* proj_in;  // a 1x1 projection of this tensor beside the layer, and their sum (patch_add_projection); nullptr: none
    CUtensorMap tmA2, tmB2;
    int proj_unsigned, proj_alloc, proj_bytes;
    int band_batch;       // images the band height was chosen for
    const void* in;       // the activations (max_batch images)
    int max_batch;
    void* encode;         // cuTensorMapEncodeTiled
    size_t smem_bytes;
};
// Chooses the band height for a call of `batch` images (a no-op when it is the plan's already)
int patch_set_batch(PatchPlan* plan, const ConvGeom& g, int batch);
// dense stride-1 layers with 32 / 64 / 128 input channels, and depthwise stride-1 layers whose channels are a
// multiple of 32 (run as block-diagonal groups of 64 or 32 channels)
bool patch_eligible(const ConvGeom& g);
int patch_groups(const ConvGeom& g);
size_t patch_dw_weight_bytes(const ConvGeom& g);
void patch_dw_arrange_weights(const ConvGeom& g, const int8_t* w_ct, int8_t* dst);
void patch_permute_weights(const int8_t* w, int8_t* dst, int O, size_t row_bytes);
int patch_make_plan(PatchPlan* plan, const void* in, const int8_t* w, const ConvGeom& g, int in_unsigned, int num_sms,
                    const char** why);
// n_base: first image of this call within the tensors the plan was encoded for (`out` = the tensor's base)
bool patch_takes_residual(const ConvGeom& g);
cudaError_t launch_patch(const PatchPlan& plan, const ConvGeom& g, int n_base, const Residual& r, const FastQuant& fast, void* out,
                         int* status_word, cudaStream_t s, const FastQuant* branch = nullptr);
// Whether the kernel computes the projection `p` beside the layer `g` and the sum of both; adds it to the layer's plan (max_batch images of `in`)
bool patch_takes_projection(const ConvGeom& g, const ConvGeom& p);
int patch_add_projection(PatchPlan* plan, const void* in, const int8_t* w, const ConvGeom& g, int in_unsigned, const char** why);

// ---- 3x3 depthwise layer and the 1x1 layer behind it (dwpw_tcgen05.cu) ----
struct DwPwPlan {
    CUtensorMap tmA;      // NHWC input, box = one patch row of bk channels
    CUtensorMap tmB;      // 1x1 weights [N][C], rows permuted in blocks of 32
    ConvGeom d;           // the depthwise layer
    int N, bk, num_sms;
    const void* dw_words; // its weights (dwpw_arrange_depthwise), device
    // the split of a call of `batch` images (dwpw_set_batch; fields as in DwPwArgs)
    int batch, units, seg, segs_per_row, rt, groups, nsplit, bn, passes, item, parts, pitch, patch_bytes, np, subs, a_sub, na, dw_shared,
        b_bytes, nb;
    size_t smem_bytes;
};
bool dwpw_eligible(const ConvGeom& d, const ConvGeom& p);
bool dwpw_faster(const ConvGeom& d, int N, int batch, int num_sms);
bool dwpw_takes_forms(const FastQuant& dw, const FastQuant& pw);
size_t dwpw_depthwise_words(const ConvGeom& d);
void dwpw_arrange_depthwise(const ConvGeom& d, const int8_t* w, uint32_t* dst);
int dwpw_make_plan(DwPwPlan* plan, const void* in, const void* dw_words, const int8_t* w, const ConvGeom& d, int N, int max_batch, int num_sms, const char** why);
// Splits a call of `batch` images (a no-op when the plan is for that many already)
int dwpw_set_batch(DwPwPlan* plan, int batch);
cudaError_t launch_dwpw(const DwPwPlan& plan, int n_base, const FastQuant& dw, const FastQuant& pw, void* out, int* status_word, cudaStream_t s);

// ---- tensor-core implicit GEMM (tcgen05 kind::i8) ----
struct IgemmPlan {
    CUtensorMap tmA;      // activations: 2-D tiled [M][K] or 4-D im2col NHWC
    CUtensorMap tmB;      // weights [N][Ktot], K-major
    CUtensorMap tmO;      // output [M][N] bytes, box = 32 rows x BN/2 (TMA store of the epilogue)
    CUtensorMap tmR;      // residual operand, same geometry (TMA load of the epilogue)
    int has_out_maps;
    int a_im2col;         // 0: 2-D tiled, 1: im2col
    int M, N;             // GEMM extents (output pixels, output channels)
    int Cin, taps;        // K = taps * Cin, walked tap by tap
    int BK;               // bytes of K per pipeline stage: 32, 64 or 128 (also the swizzle width)
    int BN;               // tile N: 64, 128 or 256
    int stages;
    int parts;            // epilogue warps that share a tile's columns per TMEM lane quadrant: 4, 2 or 1 (a warp then takes BN / parts columns)
    int grouped;          // depthwise layer as block-diagonal groups: column block n reads input channels [n * BN, (n + 1) * BN)
    int b_resident;       // weights of the CTA's column block stay in shared memory for the whole launch
    int res_slots;        // fused residual: staging regions per epilogue warp (2 or 4), 0 without a residual
    int w4;               // weights are packed 4-bit values in HBM ([N][Ktot / 2] bytes, even element in the high nibble)
    int perm;             // weight rows stored permuted inside blocks of this many output channels (32 or 16; 0 = not)
    int pair;             // large-K layer with 256-column tiles: CTAs take two 128-row tiles per weight slab
    CUtensorMap tmO32;    // output [M][N] bytes, box = 32 rows x 32 columns (the pair kernel's two-pass store)
    size_t pair_smem_bytes;
    int a_unsigned;
    // im2col geometry
    int oW, oH, kW, sX, sY, pL, pT, dX, dY;
    int grid;             // CTAs to launch
    int num_sms;
    int late_weights;     // the weights are the previous kernel's output: not before griddepcontrol.wait
    size_t smem_bytes;
};
// depthwise layers the kernel takes as block-diagonal groups (channels a multiple of 64, or 32): channels per group,
// bytes and layout of the block-diagonal weight matrix [C][taps][group]
int igemm_dw_group(const ConvGeom& g);
size_t igemm_dw_weight_bytes(const ConvGeom& g);
void igemm_dw_arrange_weights(const ConvGeom& g, const int8_t* w_ct, int8_t* dst);
// Encodes the tensor maps for `in`/`w` and fills the tiling. Returns 0, or -1 with `why` set.
// force_pair: take the 256-row variant wherever its structure allows, whatever the layer's size (tests)
int igemm_make_plan(IgemmPlan* plan, const void* in, const int8_t* w, const void* out, const void* res,
                    const ConvGeom& g, int in_unsigned, int force_im2col, int force_bn, int num_sms, const char** why,
                    int force_pair = 0, int w4 = 0);
// Points a plan at buffers that only the forward pass knows (either may be nullptr: left as it is).  The maps cover g.B images and no
// more: the last tile's rows beyond them read as zero, where a map over max_batch images would read past the caller's buffer.
int igemm_bind_buffers(IgemmPlan* plan, const void* in, const void* res, const ConvGeom& g, const char** why);
// Whether a launch of this plan takes the 32-bit epilogue; such a cell's weight rows must be stored in the
// permuted order (igemm_permute_weights with igemm_perm_block(plan)) and plan.perm set to that block size.
bool igemm_uses_fast_epilogue(const IgemmPlan& plan, const FastQuant& fast, bool has_residual, int out_dtype);
int igemm_perm_block(const IgemmPlan& plan);
void igemm_permute_weights(const int8_t* w, int8_t* dst, int N, size_t row_bytes, int perm_block);
// m_base: first output row (pixel) of this call within the tensors the plan was encoded for; `out` and the
// residual stay the tensors' base pointers
// rows: where the output's rows go instead, stored from the registers without the columns the plan was padded with (only where igemm_writes_rows)
cudaError_t launch_igemm(const IgemmPlan& plan, const QuantDev& q, const Residual& r, const FastQuant& fast,
                         void* out, int out_dtype, int m_base, int* status_word, cudaStream_t s, void* rows = nullptr, int columns = 0);
// Whether a launch of plan.M rows stores from the registers and so may write rows of `columns` bytes
bool igemm_writes_rows(const IgemmPlan& plan, int columns);
// Whether it runs on clusters of CTAs that share a tile
bool igemm_takes_clusters(const IgemmPlan& plan);

// ---- two convolutions and the sum of their outputs (igemm_dual.cu) ----
struct DualPlan {
    IgemmPlan a, b;       // maps, extents and tiling of the branch and of the projection
    int stages, slot_bytes, resident;
    size_t smem_bytes;
};
int dual_make_plan(DualPlan* plan, const void* in_a, const int8_t* w_a, const ConvGeom& ga, int a_unsigned, const void* in_b, const int8_t* w_b, const ConvGeom& gb,
                   int b_unsigned, const void* out, int num_sms, const char** why);
// fb: the projection's rescale with the sum's; m_base: first output row of the call's images; gb.B images
cudaError_t launch_dual(const DualPlan& plan, const ConvGeom& gb, const FastQuant& fa, const FastQuant& fb, int branch_unsigned, int m_base, int late_weights,
                        int* status_word, cudaStream_t s);

// ---- a 1x1 expansion to 256 channels with its residual sum, and the 1x1 layer behind it (igemm_chain.cu) ----
struct ChainPlan {
    IgemmPlan a;          // maps of the expansion's operands, its output and its residual
    CUtensorMap tmB2;     // weights of the layer behind, box = 64 of its inputs x all outputs
    int C, N2, slots, y_unsigned;
    size_t smem_bytes;
};
bool chain_eligible(const ConvGeom& g, const ConvGeom& p);
int chain_make_plan(ChainPlan* plan, const void* in, const int8_t* w, const void* y, const void* res, const ConvGeom& g, int in_unsigned, const int8_t* w_next,
                    const ConvGeom& p, int y_unsigned, int num_sms, const char** why);
// M rows from row m_base on; out: the next layer's tensor
cudaError_t launch_chain(const ChainPlan& plan, int M, const FastQuant& fast, int res_unsigned, const FastQuant& next, void* out, int m_base, int* status_word,
                         cudaStream_t s);

// Widens packed 4-bit weights [rows_src][8 words / 2 bytes] into int8 [rows][8 words] in the row order a kernel expects, several cells' in one launch.  Row n
// of the destination is real channel perm_real_channel(n, ng_dst); ng_src says how the packed rows are ordered (0: naturally).
// Destination rows of channels that do not exist are zero.
struct WidenJob {
    const uint8_t* packed;
    int8_t* dst;
    int rows_src, ng_src, rows, ng_dst;
    unsigned words;       // 8-byte words of a destination row
};
cudaError_t launch_widen_int4(const WidenJob* jobs, int count, cudaStream_t s);

// ---- first-layer convolution (<= 4 input channels) on the tensor cores ----
struct StemPlan {
    CUtensorMap tmB;      // arranged weights [O][nkb*128]
    void* encode;         // cuTensorMapEncodeTiled (the output map is encoded per launch)
    int nkb;
    int BN;
    int stages;
    int in_unsigned;
    int num_sms;
    size_t smem_bytes;
};
bool stem_eligible(const ConvGeom& g);
size_t stem_weight_bytes(const ConvGeom& g);
void stem_arrange_weights(const ConvGeom& g, const int8_t* w_ohwi, int8_t* dst);
int stem_make_plan(StemPlan* plan, const int8_t* d_w_arranged, const ConvGeom& g, int in_unsigned, int num_sms,
                   const char** why);
// Re-lays [pixels][C] (C <= 4) as [pixels][4] with zero fill.
// [batch][H][W][C] -> [batch][Hp][Wp][4] with the zero padding written out (dimensions from stem_padded_dims)
void stem_padded_dims(const ConvGeom& g, int* Hp, int* Wp);
cudaError_t launch_pad_image(const void* in, const ConvGeom& g, int batch, void* out, cudaStream_t s);
cudaError_t launch_stem(const StemPlan& plan, const void* in4, const ConvGeom& g, const FastQuant& fast, void* out,
                        int* status_word, cudaStream_t s);

// ---- a whole small network in one kernel (small_net.cu) ----
static constexpr int SMALL_NET_CELLS = 12;
struct SmallCell {
    int pool, is_max, last;
    int O, Opad, oH, oW, kH, kW;
    int words;                      // 32-bit words of a filter row's run of kW * C bytes
    int step_x, step_y, step_ky;    // bytes from one output pixel / output row / filter row to the next in the padded input
    int copy_stride;                // bytes between the moved copies of the input of a cell whose windows start on any byte
    int log_split;                  // a window's words are dealt out to 2^log_split threads
    int in_off, out_off, out_row;   // activation area: this cell's input, where its output goes, bytes per output row there
    int out_copies, out_copy_stride;    // copies of the output that the next cell wants
    int w_off, cst_off;             // weights and constants in the blob
    int form;                       // rescale: 0, EF_WIDE, EF_FLOAT, or -1 for the exact 64-bit one (q)
    int in_unsigned, out_unsigned;
    int inH, inW, sY, sX, padY, padX;   // pooling
    unsigned rcp_O, rcp_oW;             // reciprocals of Opad / 2 (channels for a pooling) and oW
    QuantDev q;
};
struct SmallNetArgs {
    SmallCell cell[SMALL_NET_CELLS];
    int nb_cells;
    const uint8_t* blob;
    int blob_bytes, act_stride;
    int in_bytes, in_place, in_pitch, in_row, in_words, in_copies, in_copy_stride;
    int out_bytes;
};
struct SmallNetPlan {
    std::vector<SmallCell> cells;
    std::vector<uint8_t> blob;      // weights and constants of every cell, as the kernel keeps them in shared memory
    int act_bytes = 0;              // activations of one image
    int in_bytes = 0, in_place = 0, in_pitch = 0, in_row = 0, in_words = 0, in_copies = 1, in_copy_stride = 0;
    int out_bytes = 0;
    int group = 1;                  // images per pass the shared memory holds: 4 or 1
};
void small_net_add_conv(SmallNetPlan* p, const ConvGeom& g, int in_unsigned, int out_unsigned, const int8_t* w, int form, const int32_t* consts,
                        int cpad, const QuantDev& q);
void small_net_add_pool(SmallNetPlan* p, const PoolGeom& g, int in_unsigned);
void small_net_link(SmallNetPlan* p, int in_off, int copies, int copy_stride, int pT, int pL, int pitch, int row_bytes, int pixel, int H, int W, int C);
bool small_net_finish(SmallNetPlan* p, int out_bytes);
// out: the network's final tensor, out2: the caller's copy of it (or nullptr)
cudaError_t launch_small_net(const SmallNetPlan& p, const void* d_blob, const void* in, int batch, void* out, void* out2, int num_sms,
                             cudaStream_t s);

}  // namespace n2d2b
