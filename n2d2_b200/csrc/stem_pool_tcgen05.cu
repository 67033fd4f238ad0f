// Host side of the first layer whose accumulators are pooled (the kernel: stem_pool_kernel.cuh)
#include <cstring>
#include <algorithm>
#include "stem_pool_kernel.cuh"

namespace n2d2b {

// ----------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static size_t sp_weight_block(int KWp) { return (size_t)128 * KWp * 16; }

static size_t sp_smem_bytes(int KH, int KWp, int Wp)
{
    const size_t w = ((KH + 1) * sp_weight_block(KWp) + 1023) & ~(size_t)1023;
    return 1024 + w + (size_t)SP_RING * ((2 * Wp * 16 + 127) & ~127) + 1024 + (2 * SP_RING + 2 * SP_SLOTS + 1) * 8 + 16;
}

bool stem_pool_eligible(const ConvGeom& g, const PoolGeom& p)
{
    if (!stem_s2d_eligible(g) || g.O != SP_CHANNELS || g.oW > 128) return false;
    if (!p.is_max || p.pH != 3 || p.pW != 3 || p.sY != 2 || p.sX != 2 || p.padY != 0 || p.padX != 0) return false;
    if (p.H != g.oH || p.W != g.oW || p.C != g.O || p.oH < 1 || p.oW < 1 || 2 * p.oH + 1 > g.oH || 2 * p.oW + 1 > g.oW) return false;
    int P, KH, KWp;
    stem_s2d_filter(g, &P, &KH, &KWp);
    return sp_smem_bytes(KH, KWp, g.oW + KWp - 1) <= 226 * 1024;
}

size_t stem_pool_weight_bytes(const ConvGeom& g)
{
    int P, KH, KWp;
    stem_s2d_filter(g, &P, &KH, &KWp);
    return (KH + 1) * sp_weight_block(KWp);
}

// OHWI int8 weights -> per image row ky of a row pair a 128 x (KWp * 16) block in the canonical unswizzled K-major order
// [m / 8][k / 16][m % 8][k % 16].  Row m = 32 Q + 16 r + c is channel 16 Q + c of the pair's row r, whose filter starts r image
// rows further down.
void stem_pool_arrange_weights(const ConvGeom& g, const int8_t* w_ohwi, int8_t* dst)
{
    int P, KH, KWp;
    stem_s2d_filter(g, &P, &KH, &KWp);
    const int offy = P - g.pT, offx = P - g.pL;
    const size_t block = sp_weight_block(KWp);
    memset(dst, 0, (KH + 1) * block);
    for (int m = 0; m < 128; ++m) {
        const int o = 16 * (m / 32) + m % 16, r = (m / 16) & 1;
        for (int ky = 0; ky < g.kH; ++ky)
            for (int kx = 0; kx < g.kW; ++kx)
                for (int c = 0; c < g.C; ++c) {
                    const int yy = ky + offy, xx = kx + offx;       // tap position in the shifted image
                    const int k = (xx >> 1) * 16 + ((yy & 1) * 2 + (xx & 1)) * 4 + c;
                    dst[((yy >> 1) + r) * block + (size_t)(m / 8) * (KWp * 128) + (size_t)(k / 16) * 128 + (size_t)(m % 8) * 16 + k % 16]
                        = w_ohwi[(((size_t)o * g.kH + ky) * g.kW + kx) * g.C + c];
                }
    }
}

// The kernel re-lays the images of this call itself (see RAW): three channels, whole words per row, and bands of four pooled rows and
// more - in short ones the latency of the first loads and the rows that bands share cost more than the other kernel (ResNet-50 at one
// image 276 us against 280)
bool stem_pool_takes_image(const StemPoolPlan& plan, const ConvGeom& g, const void* in)
{
    int P, KH, KWp;
    stem_s2d_filter(g, &P, &KH, &KWp);
    return (long long)g.B * plan.poH >= 4ll * plan.num_sms && g.C == 3 && g.W % 4 == 0 && P % 2 == 0 && ((uintptr_t)in & 3) == 0 && (long long)g.B * g.H < (1ll << 31)
        && (P + 3) / 4 * 4 - P + 2 * plan.Wp + 3 <= 4 * 80;
}

int stem_pool_make_plan(StemPoolPlan* plan, const void* d_s2d, const int8_t* d_w_arranged, const ConvGeom& g, const PoolGeom& p, int max_batch,
                        int in_unsigned, int num_sms, const char** why)
{
    static const char* kWhy = "";
    *why = kWhy;
    if (!stem_pool_eligible(g, p)) { *why = "geometry outside the first-layer kernel with pooling"; return -1; }
    cudaDriverEntryPointQueryResult qr;
    void* fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) != cudaSuccess || !fn) {
        *why = "cuTensorMapEncodeTiled is not available from the CUDA driver";
        return -1;
    }
    memset(plan, 0, sizeof(*plan));
    int P;
    stem_s2d_filter(g, &P, &plan->KH, &plan->KWp);
    plan->Wp = g.oW + plan->KWp - 1;
    plan->w = d_w_arranged;
    plan->w_bytes = (int)stem_pool_weight_bytes(g);
    plan->in_unsigned = in_unsigned;
    plan->num_sms = num_sms;
    plan->poH = p.oH;
    plan->poW = p.oW;
    plan->smem_bytes = sp_smem_bytes(plan->KH, plan->KWp, plan->Wp);
    int Hs, Ws;
    stem_s2d_dims(g, &Hs, &Ws);
    // the re-laid image as (8-byte words of a row, rows, images): one box = two rows
    const cuuint64_t dims[3] = {(cuuint64_t)Ws * 2, (cuuint64_t)Hs, (cuuint64_t)max_batch};
    const cuuint64_t strides[2] = {(cuuint64_t)Ws * 16, (cuuint64_t)Ws * 16 * Hs};
    const cuuint32_t box[3] = {(cuuint32_t)plan->Wp * 2, 2, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    if (((EncodeTiledFn)fn)(&plan->tmX, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, (void*)d_s2d, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
        *why = "cuTensorMapEncodeTiled failed for the re-laid image";
        return -1;
    }
    return 0;
}

// raw: the call's images as they are (stem_pool_takes_image), or nullptr: re-laid in the plan's buffer
cudaError_t launch_stem_pool(const StemPoolPlan& plan, const ConvGeom& g, int n_base, const void* raw, const FastQuant& fast, void* out, int* status_word,
                             cudaStream_t s)
{
    if (g.B == 0) return cudaSuccess;
    StemPoolArgs a;
    memset(&a, 0, sizeof(a));
    a.poH = plan.poH; a.poW = plan.poW;
    a.KH = plan.KH; a.KWp = plan.KWp; a.Wp = plan.Wp;
    // the tallest bands that give the busiest CTA the fewest row pairs, one more per band than it has pooled rows
    long long best = 0;
    for (int P = 1; P <= plan.poH; ++P) {
        const long long items = (long long)g.B * ((plan.poH + P - 1) / P), cost = (items + plan.num_sms - 1) / plan.num_sms * (P + 1);
        if (best == 0 || cost <= best) { best = cost; a.P = P; }
    }
    a.bands = (plan.poH + a.P - 1) / a.P;
    if ((long long)g.B * a.bands >= (1ll << 31)) return cudaErrorInvalidValue;
    a.items = g.B * a.bands;
    a.n_base = n_base;
    a.raw = (const uint8_t*)raw;
    a.H = g.H;
    a.W = g.W;
    int KH, KWp;
    stem_s2d_filter(g, &a.shift, &KH, &KWp);
    a.groups_per_row = ((a.shift + 3) / 4 * 4 - a.shift + 2 * plan.Wp + 3) / 4;
    a.chunk_alloc = (2 * plan.Wp * 16 + 127) & ~127;
    a.w_bytes = plan.w_bytes;
    const int N = (g.oW + 15) & ~15;
    // instruction descriptor: D = s32, A = s8 weights, B = u8 / s8 positions, both K-major
    a.idesc = (2u << 4) | (1u << 7) | ((plan.in_unsigned ? 0u : 1u) << 10) | ((unsigned)(N >> 3) << 17) | ((128u >> 4) << 24);
    a.w = plan.w;
    a.out = (uint8_t*)out;
    a.status = status_word;
    a.fq = fast.fq;
    a.cpad = fast.cpad;
    a.out_lo = fast.out_unsigned ? 0 : -128;
    a.out_hi = fast.out_unsigned ? 255 : 127;
    typedef const StemPoolKernel (*Table)[3][4];
    static const Table forms[6] = {stem_pool_int, stem_pool_int_clamped, stem_pool_float, stem_pool_float_clamped, stem_pool_wide,
                                    stem_pool_wide_clamped};
    static SmemLimitSet limits[6][2][3][4];
    const int shape = plan.KH == 4 && plan.KWp == 4 ? 1 : (plan.KH == 2 && plan.KWp == 2 ? 2 : 0);
    const int form = (fast.form == EF_WIDE ? 4 : (fast.form == EF_FLOAT ? 2 : 0)) + (fast.need_clamp ? 1 : 0);
    const int per_lane = (plan.poW + 7) / 8, hp = per_lane <= 4 ? 0 : (per_lane <= 6 ? 1 : (per_lane <= 7 ? 2 : 3));
    const int grid = a.items < plan.num_sms ? a.items : plan.num_sms;
    const StemPoolKernel kernel = forms[form][raw ? 1 : 0][shape][hp];
    if (cudaError_t e = raise_smem_limit(kernel, limits[form][raw ? 1 : 0][shape][hp])) return e;
    return launch_pdl(kernel, grid, raw ? SP_THREADS_RAW : SP_THREADS, plan.smem_bytes, s, plan.tmX, a);
}

}  // namespace n2d2b
