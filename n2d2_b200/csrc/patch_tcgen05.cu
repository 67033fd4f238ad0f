// Host side of the patch kernel: which layers it takes, its plans and launch (and its kernels of the 32-bit rescale)
#include <cstring>
#include "patch_kernel.cuh"

namespace n2d2b {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// weights of up to this size stay resident; larger ones stream tap by tap through a ring of `bring` blocks, and
// the epilogue then stages 32 columns per pass so that the ring can be deep: its loads cross the L2 with a
// latency of thousands of cycles, and what is in flight bounds what arrives
static constexpr size_t P_RESIDENT_MAX = 96 * 1024;
static bool patch_streams(int taps, int C, int BN) { return (size_t)taps * BN * C > P_RESIDENT_MAX; }

// (`spare` caps the band height of two buffers: with that space given to the patches, the 64-channel 55 x 55 layers went from
// five bands of 11 rows to 22 + 22 + 11 and ran 18 % slower.  More buffers may use it.)
// proj_alloc: bytes of a projection's band beside every patch (0: none)
static size_t patch_smem_bytes(int taps, int C, int BN, int patch_alloc, int bring = P_BRING_MIN, int nbuf = 2, int proj_alloc = 0)
{
    const int blocks = patch_streams(taps, C, BN) ? bring : taps;
    const size_t b = (((size_t)(blocks + (proj_alloc ? 1 : 0)) * BN * C) + 1023) & ~(size_t)1023;
    const size_t spare = nbuf == 2 && !proj_alloc ? (size_t)P_EPI_WARPS * 32 * (patch_streams(taps, C, BN) ? 32 : BN) : 0;
    return 1024 + b + nbuf * (size_t)(patch_alloc + proj_alloc) + spare + (2 * P_BUFS_MAX + 2 * P_SLOTS + 2 + 2 * P_BRING_MAX) * 8 + 32
         + FAST_NP * 256 * 4 + 64;
}

// bytes a patch buffer must hold for bands of R rows: the tiles of a band read 128-row operands that start
// up to (kH-1)*dY*Wp + (kW-1)*dX rows after the tile's first position
static int patch_alloc_bytes(const ConvGeom& g, int Wp, int R)
{
    const int tiles = (R * Wp + PBM - 1) / PBM;
    const int reach = tiles * PBM + (g.kH - 1) * g.dY * Wp + (g.kW - 1) * g.dX;
    const int box = (R + (g.kH - 1) * g.dY) * Wp;
    const int rows = reach > box ? reach : box;
    return (rows * g.C + 1023) & ~1023;
}

// Channels per block-diagonal group of a depthwise layer (0: not a layer this kernel takes as groups)
static int patch_dw_group(const ConvGeom& g)
{
    if (g.groups <= 1 || g.groups != g.C || g.O != g.C || g.Cg != 1 || g.Og != 1) return 0;
    if (g.C % 64 == 0) return 64;
    if (g.C % 32 == 0) return 32;
    return 0;
}

// The geometry of one group of a depthwise layer as the dense layer the kernel sees
static ConvGeom patch_group_geom(const ConvGeom& g)
{
    ConvGeom e = g;
    const int cg = patch_dw_group(g);
    if (cg) { e.C = cg; e.O = cg; e.groups = 1; e.Cg = cg; e.Og = cg; }
    return e;
}

int patch_groups(const ConvGeom& g) { const int cg = patch_dw_group(g); return cg ? g.C / cg : 1; }

bool patch_eligible(const ConvGeom& g0)
{
    if (g0.groups != 1 && (!patch_dw_group(g0) || patch_groups(g0) > 64)) return false;
    const ConvGeom g = patch_group_geom(g0);
    if (g.groups != 1 || g.sX != 1 || g.sY != 1) return false;
    if (g.C != 32 && g.C != 64 && g.C != 128) return false;
    if (g.O % 32 != 0 || g.O > 128) return false;
    if (g.kH * g.kW < 2) return false;   // a 1x1 layer gains nothing from a patch
    const int BN = g.O <= 64 ? 64 : 128;
    const int Wp = g.oW + (g.kW - 1) * g.dX;
    if (Wp > 256 || Wp < 2 || g.oH < 1) return false;
    if ((g.kH - 1) * g.dY + 1 > 256) return false;
    // at least one output row per band must fit
    return patch_smem_bytes(g.kH * g.kW, g.C, BN, patch_alloc_bytes(g, Wp, 1)) <= 226 * 1024;
}

// Weight rows ([O][taps * C] bytes) in the order the kernel's epilogue expects
void patch_permute_weights(const int8_t* w, int8_t* dst, int O, size_t row_bytes)
{
    for (int n = 0; n < O; ++n) memcpy(dst + (size_t)n * row_bytes, w + (size_t)perm_real_channel(n, 4) * row_bytes, row_bytes);
}

// Depthwise weights [C][taps] as the block-diagonal matrix of the grouped form: row o = [taps][group channels] with
// the tap's weight at column o % group and zeros elsewhere; rows in the epilogue's order.
size_t patch_dw_weight_bytes(const ConvGeom& g) { return (size_t)g.C * g.kH * g.kW * patch_dw_group(g); }
void patch_dw_arrange_weights(const ConvGeom& g, const int8_t* w_ct, int8_t* dst)
{
    const int cg = patch_dw_group(g), taps = g.kH * g.kW;
    const size_t row_bytes = (size_t)taps * cg;
    memset(dst, 0, (size_t)g.C * row_bytes);
    for (int n = 0; n < g.C; ++n) {
        const int o = perm_real_channel(n, 4);
        for (int t = 0; t < taps; ++t) dst[(size_t)n * row_bytes + (size_t)t * cg + (o % cg)] = w_ct[(size_t)o * taps + t];
    }
}

// bytes of a projection's band of R rows: whole tiles of positions
static int patch_proj_alloc(const ConvGeom& g, int Wp, int R) { return (R * Wp + PBM - 1) / PBM * PBM * g.C; }

bool patch_takes_projection(const ConvGeom& g, const ConvGeom& p)
{
    return patch_takes_residual(g) && p.groups == 1 && p.C == 64 && p.O == 64 && p.kH == 1 && p.kW == 1 && p.sX == 1 && p.sY == 1 && p.pT == 0 && p.pL == 0 && p.oH == g.oH
        && p.oW == g.oW && p.H == g.oH && p.W == g.oW;
}

int patch_add_projection(PatchPlan* plan, const void* in, const int8_t* w, const ConvGeom& g0, int in_unsigned, const char** why)
{
    static const char* kWhy = "";
    *why = kWhy;
    if (((uintptr_t)in & 15) || ((uintptr_t)w & 15)) { *why = "operands must be 16-byte aligned"; return -1; }
    const cuuint64_t dims[2] = {64, 64};
    const cuuint64_t strides[1] = {64};
    const cuuint32_t box[2] = {64, 64};
    const cuuint32_t estr[2] = {1, 1};
    if (((EncodeTiledFn)plan->encode)(&plan->tmB2, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)w, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                      CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
        *why = "cuTensorMapEncodeTiled failed for the projection's weights";
        return -1;
    }
    plan->proj_in = in;
    plan->proj_unsigned = in_unsigned;
    plan->band_batch = plan->R = 0;   // the bands are chosen anew, with the projection's beside them
    if (patch_set_batch(plan, g0, plan->max_batch)) { *why = "no band height fits shared memory"; return -1; }
    return 0;
}

int patch_make_plan(PatchPlan* plan, const void* in, const int8_t* w, const ConvGeom& g0, int in_unsigned, int num_sms,
                    const char** why)
{
    static const char* kWhy = "";
    *why = kWhy;
    if (!patch_eligible(g0)) { *why = "geometry outside the patch kernel"; return -1; }
    const ConvGeom g = patch_group_geom(g0);   // one group (the layer itself when it is dense)
    if (((uintptr_t)in & 15) || ((uintptr_t)w & 15)) { *why = "operands must be 16-byte aligned"; return -1; }
    cudaDriverEntryPointQueryResult qr;
    void* fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) != cudaSuccess || !fn) {
        *why = "cuTensorMapEncodeTiled is not available from the CUDA driver";
        return -1;
    }
    memset(plan, 0, sizeof(*plan));
    const int taps = g.kH * g.kW;
    plan->BN = g.O <= 64 ? 64 : 128;
    plan->Wp = g.oW + (g.kW - 1) * g.dX;
    plan->in_unsigned = in_unsigned;
    plan->num_sms = num_sms;
    plan->G = patch_groups(g0);
    plan->b_stream = patch_streams(taps, g.C, plan->BN) ? 1 : 0;
    plan->in = in;
    plan->max_batch = g.B;
    plan->encode = fn;
    const CUtensorMapSwizzle swz = g.C == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                                              : (g.C == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    CUresult rc;
    {   // weights [O][taps*C], one box = one tap of all outputs (rows beyond O read as zero)
        const cuuint64_t dims[2] = {(cuuint64_t)taps * g.C, (cuuint64_t)g0.O};
        const cuuint64_t strides[1] = {(cuuint64_t)taps * g.C};
        const cuuint32_t box[2] = {(cuuint32_t)g.C, (cuuint32_t)plan->BN};
        const cuuint32_t estr[2] = {1, 1};
        rc = ((EncodeTiledFn)fn)(&plan->tmB, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)w, dims, strides, box, estr,
                                 CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (rc != CUDA_SUCCESS) { *why = "cuTensorMapEncodeTiled failed for the weights"; return -1; }
    }
    if (patch_set_batch(plan, g0, g.B)) { *why = "no band height fits shared memory"; return -1; }
    return 0;
}

// Rows per band: among the heights that fit shared memory (and the 256-row TMA box), the one that wastes the fewest
// 128-position tiles per image; ties go to the taller band (fewer halo rows re-read).  When that leaves the SMs fewer than two bands
// each, a CTA's longest run decides instead, counted in tiles plus one per band (one image of 55 x 55: 5 bands of 11 rows
// 10.4 us, 28 bands of 2 rows 7.5 us).  At larger batches even runs do not pay for tall bands: 1024 such images take 124 us in bands of 11
// rows (25 tiles per image), 159 us in bands of 17 (26).
int patch_set_batch(PatchPlan* plan, const ConvGeom& g0, int batch)
{
    if (plan->band_batch == batch) return 0;
    const ConvGeom g = patch_group_geom(g0);
    const int taps = g.kH * g.kW, Wp = plan->Wp;
    const long long ctas = plan->num_sms / plan->G > 0 ? plan->num_sms / plan->G : 1;
    int best_R = 0;
    for (int even = 0; even < 2; ++even) {
        long long best = 0;
        for (int R = 1; R <= g.oH; ++R) {
            if (R + (g.kH - 1) * g.dY > 256) break;
            if (patch_smem_bytes(taps, g.C, plan->BN, patch_alloc_bytes(g, Wp, R), P_BRING_MIN, 2, plan->proj_in ? patch_proj_alloc(g, Wp, R) : 0) > 226 * 1024) break;
            // streamed weights: every tile of a band accumulates while the taps pass, so a band has at most as many
            // tiles as there are accumulators
            const int tall = (R * Wp + PBM - 1) / PBM;
            if (plan->b_stream && tall > P_SLOTS) break;
            const int bands = (g.oH + R - 1) / R, rest = g.oH - (bands - 1) * R;
            const long long cost = even ? ((long long)batch * bands + ctas - 1) / ctas * (tall + 1)
                                        : (long long)(bands - 1) * tall + (rest * Wp + PBM - 1) / PBM;
            if (best == 0 || cost <= best) { best_R = R; best = cost; }
        }
        if (best_R == 0 || (long long)batch * ((g.oH + best_R - 1) / best_R) >= 2 * ctas) break;
    }
    if (best_R == 0) return -1;
    plan->band_batch = batch;
    if (best_R == plan->R) return 0;
    plan->R = best_R;
    plan->bands = (g.oH + best_R - 1) / best_R;
    const int box_rows = best_R + (g.kH - 1) * g.dY;
    plan->patch_bytes = box_rows * plan->Wp * g.C;
    plan->patch_alloc = patch_alloc_bytes(g, plan->Wp, best_R);
    plan->proj_alloc = plan->proj_in ? patch_proj_alloc(g, plan->Wp, best_R) : 0;
    plan->proj_bytes = plan->proj_in ? best_R * plan->Wp * g.C : 0;
    plan->bring = P_BRING_MIN;
    while (plan->b_stream && plan->bring < P_BRING_MAX
           && patch_smem_bytes(taps, g.C, plan->BN, plan->patch_alloc, plan->bring + 1) <= 226 * 1024)
        ++plan->bring;
    plan->nbuf = 2;
    while (plan->nbuf < P_BUFS_MAX
           && patch_smem_bytes(taps, g.C, plan->BN, plan->patch_alloc, plan->bring, plan->nbuf + 1, plan->proj_alloc) <= 226 * 1024)
        ++plan->nbuf;
    plan->smem_bytes = patch_smem_bytes(taps, g.C, plan->BN, plan->patch_alloc, plan->bring, plan->nbuf, plan->proj_alloc);
    // NHWC activations as (C, W, H, B); one box = a whole patch, zero-filled outside the image
    const CUtensorMapSwizzle swz = g.C == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                                              : (g.C == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    const int Ct = g0.C;
    const cuuint64_t dims[4] = {(cuuint64_t)Ct, (cuuint64_t)g.W, (cuuint64_t)g.H, (cuuint64_t)plan->max_batch};
    const cuuint64_t strides[3] = {(cuuint64_t)Ct, (cuuint64_t)Ct * g.W, (cuuint64_t)Ct * g.W * g.H};
    const cuuint32_t box[4] = {(cuuint32_t)g.C, (cuuint32_t)plan->Wp, (cuuint32_t)box_rows, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    if (plan->proj_in) {   // the projection's input: the output's extents, a box without border rows
        const cuuint64_t dims2[4] = {(cuuint64_t)g.C, (cuuint64_t)g.oW, (cuuint64_t)g.oH, (cuuint64_t)plan->max_batch};
        const cuuint64_t strides2[3] = {(cuuint64_t)g.C, (cuuint64_t)g.C * g.oW, (cuuint64_t)g.C * g.oW * g.oH};
        const cuuint32_t box2[4] = {(cuuint32_t)g.C, (cuuint32_t)plan->Wp, (cuuint32_t)best_R, 1};
        if (((EncodeTiledFn)plan->encode)(&plan->tmA2, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, (void*)plan->proj_in, dims2, strides2, box2, estr,
                                          CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return -1;
    }
    return ((EncodeTiledFn)plan->encode)(&plan->tmA, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, (void*)plan->in, dims, strides, box, estr,
                                         CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -1;
}

// A residual sum in this kernel's epilogue: 64 -> 64 channels, 3x3.  (At 128 channels the implicit-GEMM kernel is even.)
bool patch_takes_residual(const ConvGeom& g)
{
    return g.groups == 1 && g.C == 64 && g.O == 64 && g.kH == 3 && g.kW == 3 && !patch_streams(9, 64, 64) && patch_eligible(g);
}

cudaError_t launch_patch(const PatchPlan& plan, const ConvGeom& g0, int n_base, const Residual& r, const FastQuant& fast, void* out,
                         int* status_word, cudaStream_t s, const FastQuant* branch)
{
    // branch: the layer's own rescale where `fast` is that of the projection beside it (with the sum's), and r says how the branch's bytes are signed
    if ((branch != nullptr) != (plan.proj_in != nullptr)) return cudaErrorInvalidConfiguration;
    if (r.ptr && (!patch_takes_residual(g0) || !fast.fq2 || fast.dp4a)) return cudaErrorInvalidConfiguration;
    const ConvGeom g = patch_group_geom(g0);
    PatchArgs a;
    memset(&a, 0, sizeof(a));
    a.B = g.B; a.oH = g.oH; a.oW = g.oW; a.N = g.O; a.BN = plan.BN; a.C = g.C;
    a.G = plan.G; a.ldo = g0.O;
    if (a.B == 0) return cudaSuccess;
    a.taps_y = g.kH; a.taps_x = g.kW; a.dY = g.dY; a.dX = g.dX; a.pT = g.pT; a.pL = g.pL;
    a.Wp = plan.Wp; a.R = plan.R; a.bands = plan.bands;
    a.n_base = n_base;
    a.patch_bytes = plan.patch_bytes; a.patch_alloc = plan.patch_alloc;
    a.b_stream = plan.b_stream;
    a.late_weights = plan.late_weights;
    a.bring = plan.bring;
    a.nbuf = plan.nbuf;
    a.rcp_Wp = (unsigned)(((1ull << 32) + (unsigned)plan.Wp - 1) / (unsigned)plan.Wp);
    a.idesc = (2u << 4) | ((plan.in_unsigned ? 0u : 1u) << 7) | (1u << 10) | ((unsigned)(plan.BN >> 3) << 17)
            | ((unsigned)(PBM >> 4) << 24);
    a.tmem_cols = (unsigned)(P_SLOTS * plan.BN);   // 256 or 512: a power of two
    a.out = out;
    a.status = status_word;
    a.fq = fast.fq;
    a.cpad = fast.cpad;
    a.out_unsigned = fast.out_unsigned;
    a.res = (const uint8_t*)r.ptr;
    a.res_unsigned = r.is_unsigned;
    a.fq2 = fast.fq2;
    a.t_lo = fast.t_lo; a.t_hi = fast.t_hi;
    if (branch) {
        a.fq_branch = branch->fq;
        a.cpad_branch = branch->cpad;
        a.proj_alloc = plan.proj_alloc;
        a.proj_bytes = plan.proj_bytes;
        a.idesc_proj = (a.idesc & ~(1u << 7)) | ((plan.proj_unsigned ? 0u : 1u) << 7);
        a.tmem_cols = 512;
    }
    static const PatchKernel patch_int[2][6] = N2D2B_PATCH_KERNELS(0);
    static SmemLimitSet limits[3][2][6];
    // a multiple of the group count: CTA b works on group b % G
    const long long items = (long long)a.B * a.bands;
    const long long per_group = plan.num_sms / plan.G > 0 ? plan.num_sms / plan.G : 1;
    const int grid = (int)((items < per_group ? items : per_group) * plan.G);
    const int shape = branch ? 5 : r.ptr ? 4 : (g.kH == 3 && g.kW == 3 && !plan.b_stream) ? (g.C == 32 ? 1 : (g.C == 64 ? 2 : 3)) : 0;
    const int form = fast.form == EF_WIDE ? 2 : (fast.form == EF_FLOAT ? 1 : 0), clamped = fast.need_clamp || (branch && branch->need_clamp) ? 1 : 0;
    const PatchKernel kernel = (form == 2 ? patch_wide : (form == 1 ? patch_float : patch_int))[clamped][shape];
    if (cudaError_t e = raise_smem_limit(kernel, limits[form][clamped][shape])) return e;
    return launch_pdl(kernel, grid, r.ptr || branch ? P_THREADS_RES : P_THREADS, plan.smem_bytes, s, plan.tmA, plan.tmB, plan.tmA2, plan.tmB2, a);
}

}  // namespace n2d2b
