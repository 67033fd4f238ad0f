// First layer by space-to-depth: the re-layout of the image and the host side (the kernel: stem_s2d_kernel.cuh)
#include <cstring>
#include <vector>
#include <algorithm>
#include "stem_s2d_kernel.cuh"

namespace n2d2b {

// [B][H][W][C] (C <= 4) -> [B][Hs][Ws][2][2][4]: block (dy, dx) of pixel (Y, X) = input pixel
// (2Y + dy - P, 2X + dx - P), zero outside the image and in the unused channels.  One block per output row.
struct S2dImage {
    const uint8_t* in;
    uint4* out;
    int C, H, W, Hs, Ws, P;
    int rows;                          // output rows of all images
    unsigned threads_per_row, total;   // word form: threads of a row and of all (0: not eligible)
};

__device__ __forceinline__ void s2d_image_bytes(const S2dImage& im, int block, int blocks)
{
    const uint8_t* __restrict__ in = im.in;
    uint4* __restrict__ out = im.out;
    const int C = im.C, H = im.H, W = im.W, Hs = im.Hs, Ws = im.Ws, P = im.P;
    const bool words = C == 4 && ((uintptr_t)in & 3) == 0;   // (the image is the caller's buffer)
    for (int row = block; row < im.rows; row += blocks) {
        const int n = row / Hs, Y = row - n * Hs;
        const uint8_t* img = in + (size_t)n * H * W * C;
        uint4* orow = out + (size_t)row * Ws;
        for (int X = threadIdx.x; X < Ws; X += blockDim.x) {
            uint32_t v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int y = 2 * Y + (q >> 1) - P, x = 2 * X + (q & 1) - P;
                uint32_t px = 0;
                if (y >= 0 && y < H && x >= 0 && x < W) {
                    const uint8_t* p = img + ((size_t)y * W + x) * C;
                    if (words) px = __ldg((const uint32_t*)p);
                    else if (C == 4) px = __ldg(p) | ((uint32_t)__ldg(p + 1) << 8) | ((uint32_t)__ldg(p + 2) << 16) | ((uint32_t)__ldg(p + 3) << 24);
                    else if (C == 3) px = __ldg(p) | ((uint32_t)__ldg(p + 1) << 8) | ((uint32_t)__ldg(p + 2) << 16);
                    else if (C == 2) px = __ldg(p) | ((uint32_t)__ldg(p + 1) << 8);
                    else px = __ldg(p);
                }
                v[q] = px;
            }
            orow[X] = make_uint4(v[0], v[1], v[2], v[3]);
        }
    }
}

// The same for three channels and rows of whole 32-bit words (width a multiple of four).  A thread owns the two output pixels whose
// blocks are four adjacent input pixels, 12 bytes of each of two rows: six word loads and a handful of byte permutes where the
// general kernel takes 24 byte loads with their conditions (1024 images of 224 x 224: 130 us, instruction-bound, against 65).
__device__ __forceinline__ void s2d_image_words(const S2dImage& im, unsigned block, unsigned blocks)
{
    const uint8_t* __restrict__ in = im.in;
    const int H = im.H, W = im.W, Hs = im.Hs, Ws = im.Ws, P = im.P;
    const unsigned threads_per_row = im.threads_per_row;
    const unsigned row_words = (unsigned)W * 3u / 4u;
    for (unsigned i = block * blockDim.x + threadIdx.x; i < im.total; i += blocks * blockDim.x) {
        const unsigned row = i / threads_per_row, n = row / (unsigned)Hs;
        const int Y = (int)(row - n * (unsigned)Hs), x0 = 4 * (int)(i - row * threads_per_row) - (P + 3) / 4 * 4;
        const int X = (x0 + P) / 2;   // first of the two output pixels; -1 where P is no multiple of four
        unsigned px[2][4];
#pragma unroll
        for (int dy = 0; dy < 2; ++dy) {
            const int y = 2 * Y + dy - P;
            unsigned w0 = 0, w1 = 0, w2 = 0;
            if ((unsigned)y < (unsigned)H && (unsigned)x0 < (unsigned)W) {
                const unsigned* p = (const unsigned*)in + (size_t)(n * (unsigned)H + (unsigned)y) * row_words + (unsigned)x0 * 3u / 4u;
                w0 = __ldg(p);
                w1 = __ldg(p + 1);
                w2 = __ldg(p + 2);
            }
            px[dy][0] = w0 & 0xffffffu;
            px[dy][1] = __byte_perm(w0, w1, 0x0543) & 0xffffffu;
            px[dy][2] = __byte_perm(w1, w2, 0x0432) & 0xffffffu;
            px[dy][3] = w2 >> 8;
        }
        uint4* o = im.out + (size_t)row * Ws + X;
        if (X >= 0 && X < Ws) o[0] = make_uint4(px[0][0], px[0][1], px[1][0], px[1][1]);
        if (X + 1 < Ws) o[1] = make_uint4(px[0][2], px[0][3], px[1][2], px[1][3]);
    }
}

template <bool WORDS>
__global__ void __launch_bounds__(256) s2d_image_kernel(const S2dImage im)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    if (WORDS) s2d_image_words(im, blockIdx.x, gridDim.x);
    else s2d_image_bytes(im, (int)blockIdx.x, (int)gridDim.x);
}

// The same with the layer itself in the launch's parameters (callers that own no device memory): the first blocks write the weights
// in the order of stem_s2d_arrange_weights and the constants, the others the image.  Neither host copies nor their
// waits: a call with eight 224 x 224 images went from 48.4 us to 23.6.
__global__ void __launch_bounds__(256) s2d_layer_and_image_kernel(const __grid_constant__ S2dLayer l, const S2dImage im)
{
    pdl_launch_dependents();
    pdl_wait();
    if ((int)blockIdx.x >= l.blocks) {
        if (im.total) s2d_image_words(im, blockIdx.x - l.blocks, gridDim.x - l.blocks);
        else s2d_image_bytes(im, (int)blockIdx.x - l.blocks, (int)gridDim.x - l.blocks);
        return;
    }
    const int i0 = (int)(blockIdx.x * blockDim.x + threadIdx.x), step = l.blocks * (int)blockDim.x;
    for (int i = i0; i < 5 * l.O; i += step) l.const_dst[i / l.O * 256 + i % l.O] = l.consts[i];
    const int row_words = l.BN * l.KWp * 4, words = l.KH * row_words, group = l.KWp * 32;   // 32-bit words: one tap's channels each
    for (int d = i0; d < words; d += step) {
        const int Y = d / row_words, r = d - Y * row_words, n8 = r / group, q = r - n8 * group;
        const int X = q >> 5, n = n8 * 8 + ((q >> 2) & 7), dy = (q >> 1) & 1, dx = q & 1;
        const int o = perm_real_channel(n, 4), ky = 2 * Y + dy - l.offy, kx = 2 * X + dx - l.offx;
        unsigned w = 0;
        if (o < l.O && ky >= 0 && ky < l.kH && kx >= 0 && kx < l.kW) {
            const int8_t* src = l.w + ((o * l.kH + ky) * l.kW + kx) * l.C;
            for (int c = 0; c < l.C; ++c) w |= (unsigned)(uint8_t)src[c] << (8 * c);
        }
        ((unsigned*)l.w_dst)[d] = w;
    }
}

// ----------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// filter extents after space-to-depth; `off` = 1 when the padding is odd (the image is shifted by one more
// pixel so that every output's window starts on an even pixel)
void stem_s2d_filter(const ConvGeom& g, int* P, int* KH, int* KWp)
{
    const int offy = g.pT & 1, offx = g.pL & 1;
    *P = g.pT + offy;
    *KH = (g.kH + offy + 1) / 2;
    const int kw = (g.kW + offx + 1) / 2;
    *KWp = (kw + 1) & ~1;   // an MMA covers two pixels
}

// cbuf_alloc: bytes of one band-sized output buffer of the fused-pooling variant (0: per-warp staging regions)
static size_t s2d_smem_bytes(int w_bytes, int BN, int band_alloc, int cbuf_alloc = 0)
{
    const size_t b = ((size_t)w_bytes + 1023) & ~(size_t)1023;
    return 1024 + b + 2 * (size_t)band_alloc + (cbuf_alloc ? 2 * (size_t)cbuf_alloc : (size_t)Z_EPI_WARPS * 32 * BN)
         + (4 + 2 * Z_SLOTS + 2 + 2) * 8 + 32 + FAST_NP * 256 * 4 + 64;
}

static int s2d_band_alloc(int Wp, int KH, int KWp, int R)
{
    const int tiles = (R * Wp + ZBM - 1) / ZBM;
    const int reach = tiles * ZBM + (KH - 1) * Wp + KWp;   // last tile's rows, the filter's extent and the overlap
    const int box = (R + KH - 1) * Wp;
    const int px = reach > box ? reach : box;
    return (px * 16 + 1023) & ~1023;
}

bool stem_s2d_eligible(const ConvGeom& g)
{
    if (g.groups != 1 || g.C > 4 || g.sX != 2 || g.sY != 2 || g.dX != 1 || g.dY != 1) return false;
    if (g.pT != g.pL || g.kH > 16 || g.kW > 16) return false;
    if (g.O % 32 != 0 || g.O > 128 || g.oW < 2 || g.oH < 1) return false;
    int P, KH, KWp;
    stem_s2d_filter(g, &P, &KH, &KWp);
    const int Wp = g.oW + KWp - 1;
    if (Wp * 2 > 256) return false;   // one row of the band is one row of the TMA box (8-byte elements)
    const int BN = g.O <= 64 ? 64 : 128;
    const int w_bytes = KH * BN * KWp * 16;
    if (w_bytes > 64 * 1024) return false;
    return s2d_smem_bytes(w_bytes, BN, s2d_band_alloc(Wp, KH, KWp, 1)) <= 226 * 1024;
}

void stem_s2d_dims(const ConvGeom& g, int* Hs, int* Ws)
{
    int P, KH, KWp;
    stem_s2d_filter(g, &P, &KH, &KWp);
    *Hs = g.oH + KH - 1;
    *Ws = g.oW + KWp - 1;
}

size_t stem_s2d_weight_bytes(const ConvGeom& g)
{
    int P, KH, KWp;
    stem_s2d_filter(g, &P, &KH, &KWp);
    const int BN = g.O <= 64 ? 64 : 128;
    return (size_t)KH * BN * KWp * 16;
}

// OHWI int8 weights -> per filter row of the re-laid problem a BN x (KWp*16) block in the canonical
// unswizzled K-major order [n / 8][k / 16][n % 8][k % 16], k = X * 16 + (dy * 2 + dx) * 4 + c.  Row n of a block holds
// output channel perm_real_channel(n, 4): the order the epilogue's fragment layout wants (see perm_block).
void stem_s2d_arrange_weights(const ConvGeom& g, const int8_t* w_ohwi, int8_t* dst)
{
    int P, KH, KWp;
    stem_s2d_filter(g, &P, &KH, &KWp);
    const int BN = g.O <= 64 ? 64 : 128;
    const int offy = P - g.pT, offx = P - g.pL;
    const size_t row_block = (size_t)BN * KWp * 16;
    memset(dst, 0, (size_t)KH * row_block);
    for (int n = 0; n < BN; ++n) {
        const int o = perm_real_channel(n, 4);
        if (o >= g.O) continue;
        for (int ky = 0; ky < g.kH; ++ky)
            for (int kx = 0; kx < g.kW; ++kx)
                for (int c = 0; c < g.C; ++c) {
                    const int yy = ky + offy, xx = kx + offx;       // tap position in the shifted image
                    const int Y = yy >> 1, dy = yy & 1, X = xx >> 1, dx = xx & 1;
                    const int k = X * 16 + (dy * 2 + dx) * 4 + c;
                    const size_t off = (size_t)Y * row_block + (size_t)(n / 8) * (KWp * 128) + (size_t)(k / 16) * 128
                                     + (size_t)(n % 8) * 16 + (size_t)(k % 16);
                    dst[off] = w_ohwi[(((size_t)o * g.kH + ky) * g.kW + kx) * g.C + c];
                }
    }
}

static S2dImage s2d_image_of(const void* in, const ConvGeom& g, int batch, void* out)
{
    S2dImage im;
    int KH, KWp;
    stem_s2d_filter(g, &im.P, &KH, &KWp);
    stem_s2d_dims(g, &im.Hs, &im.Ws);
    im.in = (const uint8_t*)in;
    im.out = (uint4*)out;
    im.C = g.C; im.H = g.H; im.W = g.W;
    im.rows = batch * im.Hs;
    // three channels and whole words per row (the padding is even): groups of four input pixels, the first at -(P + 3) / 4 * 4
    im.threads_per_row = (unsigned)(((im.P + 3) / 4 * 4 - im.P + 2 * im.Ws + 3) / 4);
    const long long total = (long long)im.rows * im.threads_per_row;
    const bool words = g.C == 3 && g.W % 4 == 0 && im.P % 2 == 0 && ((uintptr_t)in & 3) == 0 && total < (1ll << 31) && (long long)batch * g.H < (1ll << 31);
    im.total = words ? (unsigned)total : 0u;
    return im;
}

static int s2d_image_blocks(const S2dImage& im)
{
    return im.total ? (int)std::min((im.total + 255u) / 256u, 32u * (unsigned)current_sms()) : std::min(im.rows, 1 << 20);
}

cudaError_t launch_s2d_image(const void* in, const ConvGeom& g, int batch, void* out, cudaStream_t s)
{
    const S2dImage im = s2d_image_of(in, g, batch, out);
    if (im.rows == 0) return cudaSuccess;
    if (im.total) return launch_pdl(s2d_image_kernel<true>, s2d_image_blocks(im), 256, 0, s, im);
    return launch_pdl(s2d_image_kernel<false>, s2d_image_blocks(im), im.Ws >= 128 ? 128 : ((im.Ws + 31) / 32) * 32, 0, s, im);
}

// `l` comes with its weights, constants and destinations
cudaError_t launch_s2d_layer_and_image(S2dLayer* l, const void* in, const ConvGeom& g, int batch, void* out, cudaStream_t s)
{
    const S2dImage im = s2d_image_of(in, g, batch, out);
    int P;
    stem_s2d_filter(g, &P, &l->KH, &l->KWp);
    l->O = g.O; l->kH = g.kH; l->kW = g.kW; l->C = g.C;
    l->offy = P - g.pT; l->offx = P - g.pL;
    l->BN = g.O <= 64 ? 64 : 128;
    l->blocks = (l->KH * l->BN * l->KWp * 4 + 255) / 256;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(l->blocks + s2d_image_blocks(im)));
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[2] = {(void*)l, (void*)&im};   // (30 KB of parameters: not copied around)
    return cudaLaunchKernelExC(&cfg, (const void*)s2d_layer_and_image_kernel, args);
}

// A max pooling this kernel can fold in: square window, same stride both ways, no padding, 8-bit channels in whole
// 16-byte units.
bool stem_s2d_pool_eligible(const ConvGeom& g, const PoolGeom& p)
{
    if (!(stem_s2d_eligible(g) && p.is_max && p.pH == p.pW && p.sY == p.sX && p.padY == 0 && p.padX == 0 && p.pH >= 1 && p.pH <= 4
          && p.sY >= 1 && p.sY <= p.pH && p.H == g.oH && p.W == g.oW && p.C == g.O && g.O % 16 == 0 && p.oH >= 1 && p.oW >= 1))
        return false;
    // one pooled row per band must fit shared memory
    int P0, KH, KWp;
    stem_s2d_filter(g, &P0, &KH, &KWp);
    const int Wp = g.oW + KWp - 1, BN = g.O <= 64 ? 64 : 128, R = p.pH;
    const int cbuf = ((R * Wp + ZBM - 1) / ZBM) * ZBM * BN;
    return s2d_smem_bytes(KH * BN * KWp * 16, BN, s2d_band_alloc(Wp, KH, KWp, R), cbuf) <= 226 * 1024;
}

static int s2d_use_bands(StemS2dPlan* plan, const ConvGeom& g, int R);

int stem_s2d_make_plan(StemS2dPlan* plan, const void* d_s2d, const int8_t* d_w_arranged, const ConvGeom& g, int max_batch,
                       int in_unsigned, int num_sms, const char** why, const PoolGeom* pool)
{
    static const char* kWhy = "";
    *why = kWhy;
    if (!stem_s2d_eligible(g)) { *why = "geometry outside the space-to-depth first-layer kernel"; return -1; }
    cudaDriverEntryPointQueryResult qr;
    void* fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) != cudaSuccess || !fn) {
        *why = "cuTensorMapEncodeTiled is not available from the CUDA driver";
        return -1;
    }
    memset(plan, 0, sizeof(*plan));
    int P;
    stem_s2d_filter(g, &P, &plan->KH, &plan->KWp);
    plan->BN = g.O <= 64 ? 64 : 128;
    plan->Wp = g.oW + plan->KWp - 1;
    plan->w_bytes = plan->KH * plan->BN * plan->KWp * 16;
    plan->w = d_w_arranged;
    plan->in_unsigned = in_unsigned;
    plan->num_sms = num_sms;
    plan->s2d = d_s2d;
    plan->max_batch = max_batch;
    plan->encode = fn;
    if (pool) {
        // the most pooled rows per band that fit: fewer bands recompute fewer overlapping convolution rows
        if (!stem_s2d_pool_eligible(g, *pool)) { *why = "pooling outside the fused first-layer kernel"; return -1; }
        int best_R = 0;
        for (int P = 1; P <= pool->oH; ++P) {
            const int R = (P - 1) * pool->sY + pool->pH;
            if (R + plan->KH - 1 > 256) break;
            const int cbuf = ((R * plan->Wp + ZBM - 1) / ZBM) * ZBM * plan->BN;
            if (s2d_smem_bytes(plan->w_bytes, plan->BN, s2d_band_alloc(plan->Wp, plan->KH, plan->KWp, R), cbuf) > 226 * 1024) break;
            best_R = R;
            plan->P = P;
            plan->cbuf_alloc = cbuf;
        }
        if (best_R == 0) { *why = "no band of the fused pooling fits shared memory"; return -1; }
        plan->pool_k = pool->pH; plan->pool_s = pool->sY; plan->pool_oH = pool->oH; plan->pool_oW = pool->oW;
        plan->row_stride = plan->P * pool->sY;
        plan->bands = (pool->oH + plan->P - 1) / plan->P;
        if (s2d_use_bands(plan, g, best_R)) { *why = "cuTensorMapEncodeTiled failed for the re-laid image"; return -1; }
        return 0;
    }
    if (stem_s2d_set_batch(plan, g, max_batch)) { *why = "no band height of the first layer fits"; return -1; }
    return 0;
}

// Bands of R rows: sizes and the tensor map
static int s2d_use_bands(StemS2dPlan* plan, const ConvGeom& g, int R)
{
    plan->R = R;
    const int box_rows = R + plan->KH - 1;
    plan->band_bytes = box_rows * plan->Wp * 16;
    plan->band_alloc = s2d_band_alloc(plan->Wp, plan->KH, plan->KWp, R);
    plan->smem_bytes = s2d_smem_bytes(plan->w_bytes, plan->BN, plan->band_alloc, plan->cbuf_alloc);
    int Hs, Ws;
    stem_s2d_dims(g, &Hs, &Ws);
    // the re-laid image as (8-byte words of a row, rows, images): one box = one band, rows below the image read as zero
    const cuuint64_t dims[3] = {(cuuint64_t)Ws * 2, (cuuint64_t)Hs, (cuuint64_t)plan->max_batch};
    const cuuint64_t strides[2] = {(cuuint64_t)Ws * 16, (cuuint64_t)Ws * 16 * Hs};
    const cuuint32_t box[3] = {(cuuint32_t)plan->Wp * 2, (cuuint32_t)box_rows, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return ((EncodeTiledFn)plan->encode)(&plan->tmA, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, (void*)plan->s2d, dims, strides, box, estr,
                                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -1;
}

// The band height: fewest tiles per image, or a CTA's shortest run at small batches (see patch_set_batch).  One 224 x 224 image in three bands
// of 38 rows: 20 us, in 112 bands of one row: 8 us.
int stem_s2d_set_batch(StemS2dPlan* plan, const ConvGeom& g, int batch)
{
    if (plan->P || plan->band_batch == batch) return 0;
    int best_R = 0;
    for (int even = 0; even < 2; ++even) {
        long long best = 0;
        for (int R = 1; R <= g.oH; ++R) {
            if (R + plan->KH - 1 > 256) break;
            if (s2d_smem_bytes(plan->w_bytes, plan->BN, s2d_band_alloc(plan->Wp, plan->KH, plan->KWp, R)) > 226 * 1024) break;
            const int bands = (g.oH + R - 1) / R, rest = g.oH - (bands - 1) * R, tall = (R * plan->Wp + ZBM - 1) / ZBM;
            const long long cost = even ? ((long long)batch * bands + plan->num_sms - 1) / plan->num_sms * (tall + 1)
                                        : (long long)(bands - 1) * tall + (rest * plan->Wp + ZBM - 1) / ZBM;
            if (best == 0 || cost <= best) { best_R = R; best = cost; }
        }
        if (best_R == 0 || (long long)batch * ((g.oH + best_R - 1) / best_R) >= 2 * plan->num_sms) break;
    }
    if (best_R == 0) return -1;
    plan->band_batch = batch;
    if (best_R == plan->R) return 0;
    plan->row_stride = best_R;
    plan->bands = (g.oH + best_R - 1) / best_R;
    return s2d_use_bands(plan, g, best_R);
}

cudaError_t launch_stem_s2d(const StemS2dPlan& plan, const ConvGeom& g, int n_base, const FastQuant& fast, void* out,
                            int* status_word, cudaStream_t s)
{
    S2dArgs a;
    memset(&a, 0, sizeof(a));
    a.B = g.B; a.oH = g.oH; a.oW = g.oW; a.N = g.O; a.BN = plan.BN;
    if (a.B == 0) return cudaSuccess;
    a.KH = plan.KH; a.KWp = plan.KWp; a.Wp = plan.Wp; a.R = plan.R; a.bands = plan.bands;
    a.row_stride = plan.row_stride;
    a.pool_k = plan.pool_k; a.pool_s = plan.pool_s; a.P = plan.P; a.pool_oH = plan.pool_oH; a.pool_oW = plan.pool_oW;
    a.cbuf_alloc = plan.cbuf_alloc;
    a.n_base = n_base;
    a.band_bytes = plan.band_bytes; a.band_alloc = plan.band_alloc; a.w_bytes = plan.w_bytes;
    a.rcp_Wp = (unsigned)(((1ull << 32) + (unsigned)plan.Wp - 1) / (unsigned)plan.Wp);
    a.idesc = (2u << 4) | ((plan.in_unsigned ? 0u : 1u) << 7) | (1u << 10) | ((unsigned)(plan.BN >> 3) << 17)
            | ((unsigned)(ZBM >> 4) << 24);
    a.tmem_cols = (unsigned)(Z_SLOTS * plan.BN);
    a.w = plan.w;
    a.late_layer = plan.late_layer;
    a.out = out;
    a.status = status_word;
    a.fq = fast.fq;
    a.cpad = fast.cpad;
    a.out_unsigned = fast.out_unsigned;
    static const StemS2dKernel kernels[6][3] = N2D2B_STEM_S2D_KERNELS(false);
    static SmemLimitSet limits[2][6][3];
    const long long items = (long long)a.B * a.bands;
    const int grid = (int)(items < plan.num_sms ? items : plan.num_sms);
    const int shape = (plan.KH == 4 && plan.KWp == 4) ? 1 : ((plan.KH == 2 && plan.KWp == 2) ? 2 : 0);
    const int form = (fast.form == EF_WIDE ? 4 : (fast.form == EF_FLOAT ? 2 : 0)) + (fast.need_clamp ? 1 : 0), pool = plan.P ? 1 : 0;
    const StemS2dKernel kernel = (pool ? stem_s2d_pool_kernels : kernels)[form][shape];
    if (cudaError_t e = raise_smem_limit(kernel, limits[pool][form][shape])) return e;
    return launch_pdl(kernel, grid, Z_THREADS, plan.smem_bytes, s, plan.tmA, a);
}

}  // namespace n2d2b
