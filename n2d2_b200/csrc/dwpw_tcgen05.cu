// Host side of the depthwise + 1x1 kernel: which pairs of layers it takes, how a call is split, its launch.
#include <algorithm>
#include <string.h>
#include "dwpw_kernel.cuh"

namespace n2d2b {

static const int DP_SMEM_LIMIT = 226 * 1024;

// Bytes of a K block (and its swizzle span): the widest that divides the channels
static int block_channels(int C) { return C % 128 == 0 ? 128 : (C % 64 == 0 ? 64 : 32); }

// The 3x3 depthwise layer `d` with the 1x1 layer `p` behind it.  Up to 1024 channels in 16 blocks: a CTA's whole operand tile then has room
// beside its patches
bool dwpw_eligible(const ConvGeom& d, const ConvGeom& p)
{
    return d.kH == 3 && d.kW == 3 && d.dX == 1 && d.dY == 1 && d.sX == d.sY && (d.sX == 1 || d.sX == 2) && d.groups == d.C && d.O == d.C && d.Cg == 1
        && d.C % 32 == 0 && d.C <= 1024 && d.C / block_channels(d.C) <= DP_MAX_A && p.kH == 1 && p.kW == 1 && p.sX == 1 && p.sY == 1 && p.pT == 0 && p.pL == 0 && p.groups == 1 && p.C == d.C
        && p.H == d.oH && p.W == d.oW && p.oH == d.oH && p.oW == d.oW && p.O % 32 == 0 && p.O <= 2048;
}

// Whether one kernel is faster than two in calls of up to `batch` images.  Measured as pairs of 32 to 1024 channels, maps of 2 to 112 pixels a side, 0.5 to 4 times
// as many outputs, strides 1 and 2 and 1 to 256 images, in graphs of several passes; times as two kernels over times as one:
//   - 1500 output pixels and more of whole blocks of 128 channels (6200 of 64, 9000 of 32 channels, 6400 of three blocks), up to two blocks and twice as many outputs, or
//     up to four blocks and as many: shift scalings 0.96 to 1.28 (512 -> 512 at 14 x 14, 33 images: 21.2 us, 19.9), fixed-point ones 0.95 to 1.2.  Outside a
//     graph a hand-over costs about half a microsecond more than in one, so the lines lie a little below the points where the graphs are even
//   - one, two, four or eight blocks of 128 channels and few output rows (a third of the multiprocessors, fewer of more blocks; of one block and up to 128 outputs,
//     more of which several CTAs would share and compute the depthwise part again, up to half): 0.97 to 1.1 and a launch less, which bounds a pass of so few
//     pixels outside a graph (MobileNet, one image: 86.3 us with thirteen pairs, 90.3 with three; in a graph 81.1 and 79.0)
//   - in between (2 rows a CTA) 0.86 to 0.95
//   - more outputs, which take several passes over the operand, 0.78 to 1.05 (512 -> 1024, 14 x 14 to 7 x 7, 256 images: 34.7 us, 41.8)
//   - more blocks, whose patches and operands do not fit beside one another, 0.37 to 0.9 (960 channels at 7 x 7)
bool dwpw_faster(const ConvGeom& d, int N, int batch, int num_sms)
{
    const int bk = block_channels(d.C), blocks = d.C / bk;
    const long long rows = (long long)batch * d.oH, pixels = rows * d.oW;
    if (N > 2 * d.C) return false;
    if (bk == 128 && (blocks & (blocks - 1)) == 0 && rows <= num_sms / 3 && rows * blocks <= 64) return true;
    if (blocks == 1 && d.C > 32 && N <= 128 && rows <= num_sms / 2) return true;
    return blocks <= 4 && (blocks <= 2 || N <= d.C) && pixels >= (blocks == 3 ? 6400 : (d.C >= 128 ? 1500 : (d.C > 32 ? 6200 : 9000)));
}

size_t dwpw_depthwise_words(const ConvGeom& d) { return (size_t)3 * d.C; }

// [C][3][3] -> [3][C] words: bytes w(0, kx), w(1, kx), w(2, kx), 0
void dwpw_arrange_depthwise(const ConvGeom& d, const int8_t* w, uint32_t* dst)
{
    for (int c = 0; c < d.C; ++c)
        for (int kx = 0; kx < 3; ++kx) {
            uint32_t v = 0;
            for (int ky = 0; ky < 3; ++ky) v |= (uint32_t)(uint8_t)w[(size_t)c * 9 + 3 * ky + kx] << (8 * ky);
            dst[(size_t)kx * d.C + c] = v;
        }
}

// (the constants of a depthwise layer, see DPF_UNIT; of the 1x1 layer a unit multiplier saves nothing)
static int form_of(const FastQuant& f) { return f.form == EF_WIDE ? DPF_WIDE : (f.need_clamp ? DPF_CLAMP : DPF_INT); }

static const DwPwKernel* kernels_for(const FastQuant& dw, const FastQuant& pw)
{
    static const DwPwKernel plain[2] = {dwpw_i8_tcgen05_kernel<1, DPF_INT, DPF_INT>, dwpw_i8_tcgen05_kernel<2, DPF_INT, DPF_INT>};
    static const DwPwKernel unit[2] = {dwpw_i8_tcgen05_kernel<1, DPF_UNIT, DPF_INT>, dwpw_i8_tcgen05_kernel<2, DPF_UNIT, DPF_INT>};
    static const DwPwKernel clamped[2] = {dwpw_i8_tcgen05_kernel<1, DPF_CLAMP, DPF_CLAMP>, dwpw_i8_tcgen05_kernel<2, DPF_CLAMP, DPF_CLAMP>};
    if (dw.form == EF_FLOAT || pw.form == EF_FLOAT) return nullptr;   // slower than two kernels (MobileNet, 1 / 16 / 256 images: 82 / 144 / 813 us, as one 92 / 162 / 875)
    const int a = form_of(dw), b = form_of(pw);
    if ((a == DPF_WIDE && dw.need_clamp) || (b == DPF_WIDE && pw.need_clamp)) return nullptr;
    if (a == DPF_WIDE) return b == DPF_WIDE ? dwpw_wide : dwpw_wide_depthwise;
    if (b == DPF_WIDE) return dwpw_wide_1x1;
    if (a == DPF_INT && b == DPF_INT) return dw.unit_multiplier ? unit : plain;
    return clamped;     // (the clamp rows are valid where none is needed)
}

bool dwpw_takes_forms(const FastQuant& dw, const FastQuant& pw) { return dw.enabled && pw.enabled && dw.out_unsigned && kernels_for(dw, pw); }

// Patch rows of a tile of `rt` segments: every image it touches brings its own border rows
static int patch_rows(const ConvGeom& d, int segs_per_row, int rt)
{
    if (segs_per_row > 1) return 3;
    const int images = (rt + 2 * d.oH - 2) / d.oH;
    return rt * d.sX + (3 - d.sX) * images;
}

// Warps of the epilogue; the others of twenty do the depthwise part.  Layers of up to 64 columns have as few channels in: their 1x1 outputs are half the
// instructions (32 -> 64 channels of 112 x 112, 256 images: 150 us with eight)
static int dp_epilogue_warps(int bn) { return bn == 64 ? 12 : 8; }

// How a call of `batch` images is split.  A CTA's work is, in cycles, the issue slots of its depthwise outputs and of its 1x1 outputs (about 9.5 and
// 4 instructions each, four a cycle, three quarters of the slots used), its MMAs (full tiles of 128 rows whatever they hold) and the
// weights it streams (about 60 bytes a cycle).  It ranks the splits; launches take 1.2 to 2.4 times what it says (waits for operand slots).  Column ranges of a tile go to several CTAs, which then repeat the depthwise part, only where
// there are fewer row segments than multiprocessors.
int dwpw_set_batch(DwPwPlan* plan, int batch)
{
    if (plan->batch == batch) return 0;
    const ConvGeom& d = plan->d;
    const int C = d.C, N = plan->N, bk = block_channels(C), kch = C / bk, S = d.sX;
    plan->bk = bk;
    const int spr = (d.oW + 125) / 126, seg = (d.oW + spr - 1) / spr;
    int pitch_px = (seg - 1) * S + 3;
    while (pitch_px * bk % 128) ++pitch_px;
    const int pitch = pitch_px * bk;
    const long long units = (long long)batch * d.oH * spr;
    if (units >= (1ll << 30)) return -1;
    bool found = false;
    double best = 0;
    for (int ns = 1; ns == 1 || (ns <= 16 && N % (64 * ns) == 0); ns *= 2) {
        const int ncta = N / ns, bn = ncta % 256 == 0 ? 256 : (ncta > 64 ? 128 : 64), passes = (ncta + bn - 1) / bn;
        const int ctas = std::max(1, plan->num_sms / ns);
        const int groups = (int)std::min<long long>(units, ctas);
        const int per = (int)((units + groups - 1) / groups);
        int rt = 0, subs = 1, na = 0, np = 0, nb = 0, a_sub = 0, patch = 0, shared = 1;
        const int b_bytes = bn * bk, b_all = passes * kch * b_bytes;
        size_t bytes = 0;
        for (int most = spr > 1 ? 1 : std::max(1, 128 / seg); most >= 1; --most) {
            int tiles = (per + most - 1) / most;
            rt = (per + tiles - 1) / tiles;
            a_sub = (rt * seg + 7) / 8 * 8 * bk;
            nb = b_all <= 64 * 1024 ? 0 : 6;
            // A tile of few channels is little work between two barriers (112 pixels of 32 channels: 30 steps of one warp): several of them
            // share a patch then, which also brings fewer border rows
            subs = 1;
            while (!nb && spr == 1 && kch == 1 && d.sX == 1 && subs < 4 && 2 * subs * rt * seg * C <= 32768 && 2 * subs <= tiles) subs *= 2;
            const int blocks = (tiles + subs - 1) / subs;
            patch = patch_rows(d, spr, rt * subs) * pitch;
            const int na_min = passes > 1 ? kch : std::min(2, kch * blocks);
            // the most of everything first: operand blocks of two tiles, four patches, six weight slots; then less of what hurts least
            const int want_na = std::min(DP_MAX_A, std::max(na_min, std::min(kch * blocks, std::max(2 * kch, 4))));
            np = std::min(DP_MAX_PATCH, kch * blocks);
            na = want_na;
            shared = 1;
            auto total = [&] {
                return (size_t)1024 + (nb ? (size_t)nb * b_bytes : (size_t)b_all) + (size_t)na * a_sub * subs + std::max((size_t)np * patch, (size_t)128 * bk)
                     + (size_t)passes * DP_PARAM_BYTES + (shared ? (size_t)(3 + FAST_NP) * 4 * C : 0) + DP_BARS * 8 + 16;
            };
            while (total() > (size_t)DP_SMEM_LIMIT) {
                if (np > 3) --np;
                else if (na > kch + (kch + 1) / 2 && na > na_min) --na;
                else if (nb > 4) --nb;
                else if (np > 2) --np;
                else if (na > na_min) --na;
                else if (nb > 3) --nb;
                else if (kch > 4 && shared) shared = 0;
                else if (nb > 2) --nb;
                else break;
            }
            np = std::min(np, na);
            bytes = total();
            if (bytes <= (size_t)DP_SMEM_LIMIT) break;
            rt = 0;
        }
        if (!rt) continue;
        const int tiles = (per + rt - 1) / rt;
        const double px = (double)per * seg;
        const double issue = px * (C * (S == 1 ? 9.5 : 12.0) + (double)ncta * 4.0) / (32 * 4 * 0.75);
        const double mma = (double)tiles * passes * (C / 32) * (bn == 256 ? 128 : (bn == 128 ? 64 : 48));
        const double load = (nb ? (double)tiles : 1.0) * b_all / 60.0;
        const double cost = std::max(issue, std::max(mma, load)) + 0.25 * (issue + mma + load);
        if (found && cost > 0.95 * best) continue;
        found = true;
        best = cost;
        plan->nsplit = ns; plan->bn = bn; plan->passes = passes; plan->groups = groups; plan->rt = rt;
        plan->subs = subs; plan->a_sub = a_sub; plan->na = na; plan->dw_shared = shared; plan->patch_bytes = patch; plan->np = np; plan->b_bytes = b_bytes; plan->nb = nb;
        plan->smem_bytes = bytes;
        // Work items: as long as they keep the depthwise warps (eight or twelve) busy over the patches in flight (two columns of every item are read for
        // its neighbour).  Items of several lanes' groups start an odd number of pixels apart: in other banks
        const int groups_of_lanes = 32 / (bk / 4), flight = std::min(np, kch * ((tiles + subs - 1) / subs));
        int item = seg;
        for (int parts = 1; parts <= seg; ++parts) {
            item = (seg + parts - 1) / parts;
            if (item <= 4 || ((seg + item - 1) / item * rt * subs + groups_of_lanes - 1) / groups_of_lanes * flight >= DP_WARPS - dp_epilogue_warps(bn) + 2) break;
        }
        if (groups_of_lanes > 1) item |= 1;
        plan->item = item;
        plan->parts = (seg + item - 1) / item;
    }
    if (!found) return -1;
    plan->seg = seg; plan->segs_per_row = spr; plan->pitch = pitch; plan->units = (int)units;
    plan->batch = batch;
    return 0;
}

int dwpw_make_plan(DwPwPlan* plan, const void* in, const void* dw_words, const int8_t* w, const ConvGeom& d, int N, int max_batch, int num_sms, const char** why)
{
    static const char* kWhy = "";
    *why = kWhy;
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                               CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    cudaDriverEntryPointQueryResult qr;
    void* fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) != cudaSuccess || !fn) { *why = "cuTensorMapEncodeTiled is not available"; return -1; }
    const Encode encode = (Encode)fn;
    if (((uintptr_t)in & 15) || ((uintptr_t)w & 15) || ((uintptr_t)dw_words & 15)) { *why = "operands must be 16-byte aligned"; return -1; }
    memset(plan, 0, sizeof(*plan));
    plan->d = d;
    plan->N = N;
    plan->num_sms = num_sms;
    plan->dw_words = dw_words;
    if (dwpw_set_batch(plan, max_batch)) { *why = "no split of the layer fits shared memory"; return -1; }
    {
        const cuuint64_t dims[4] = {(cuuint64_t)d.C, (cuuint64_t)d.W, (cuuint64_t)d.H, (cuuint64_t)max_batch};
        const cuuint64_t strides[3] = {(cuuint64_t)d.C, (cuuint64_t)d.C * d.W, (cuuint64_t)d.C * d.W * d.H};
        const cuuint32_t box[4] = {(cuuint32_t)plan->bk, (cuuint32_t)(plan->pitch / plan->bk), 1, 1};
        const cuuint32_t estr[4] = {1, 1, 1, 1};
        if (encode(&plan->tmA, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, (void*)in, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) { *why = "no tensor map of the input"; return -1; }
    }
    {
        const cuuint64_t dims[2] = {(cuuint64_t)d.C, (cuuint64_t)N};
        const cuuint64_t strides[1] = {(cuuint64_t)d.C};
        const cuuint32_t box[2] = {(cuuint32_t)plan->bk, (cuuint32_t)DP_BOX_N};
        const cuuint32_t estr[2] = {1, 1};
        const CUtensorMapSwizzle swz = plan->bk == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (plan->bk == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
        if (encode(&plan->tmB, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)w, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) { *why = "no tensor map of the weights"; return -1; }
    }
    return 0;
}

cudaError_t launch_dwpw(const DwPwPlan& plan, int n_base, const FastQuant& dw, const FastQuant& pw, void* out, int* status_word, cudaStream_t s)
{
    const DwPwKernel* const table = kernels_for(dw, pw);
    if (!table || !plan.batch) return cudaErrorInvalidValue;
    const ConvGeom& d = plan.d;
    DwPwArgs a;
    memset(&a, 0, sizeof(a));
    a.C = d.C; a.N = plan.N; a.kchunks = d.C / plan.bk; a.oH = d.oH; a.oW = d.oW; a.pT = d.pT; a.pL = d.pL;
    a.seg = plan.seg; a.segs_per_row = plan.segs_per_row; a.rt = plan.rt;
    a.unit0 = n_base * d.oH * plan.segs_per_row; a.units = plan.units; a.groups = plan.groups; a.nsplit = plan.nsplit;
    a.bn = plan.bn; a.passes = plan.passes; a.acc_shift = plan.bn == 256 ? 1 : 2; a.epi_warps = dp_epilogue_warps(plan.bn); a.epi_groups = plan.bn == 256 ? 1 : a.epi_warps / 4;
    a.item = plan.item; a.parts = plan.parts; a.rcp_parts = 65536u / (unsigned)plan.parts + 1u;
    a.pitch = plan.pitch; a.patch_bytes = plan.patch_bytes; a.np = plan.np;
    a.subs = plan.subs; a.rcp_rt = 65536u / (unsigned)plan.rt + 1u; a.a_sub = plan.a_sub; a.a_bytes = plan.a_sub * plan.subs; a.na = plan.na; a.b_bytes = plan.b_bytes; a.nb = plan.nb;
    // D = s32, A = u8, B = s8, both K-major
    a.idesc = (2u << 4) | (1u << 10) | ((unsigned)(plan.bn >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
    a.tmem_cols = (unsigned)plan.bn << a.acc_shift;
    a.dw_w = (const int4*)plan.dw_words; a.dw_fq = dw.fq; a.dw_cpad = dw.cpad; a.dw_shared = plan.dw_shared;
    a.fq = pw.fq; a.cpad = pw.cpad; a.out_unsigned = pw.out_unsigned;
    a.out = (uint8_t*)out;
    a.status = status_word;
    static SmemLimitSet limits[6][2];
    const int v = dw.unit_multiplier && form_of(dw) == DPF_INT && form_of(pw) == DPF_INT ? 0
                : (form_of(dw) == DPF_INT && form_of(pw) == DPF_INT ? 1 : (table == dwpw_wide ? 2 : (table == dwpw_wide_1x1 ? 3 : (table == dwpw_wide_depthwise ? 4 : 5))));
    const DwPwKernel kernel = table[d.sX - 1];
    if (cudaError_t e = raise_smem_limit(kernel, limits[v][d.sX - 1])) return e;
    return launch_pdl(kernel, dim3((unsigned)(plan.groups * plan.nsplit)), DP_THREADS, plan.smem_bytes, s, plan.tmA, plan.tmB, a, plan.bk);
}

}  // namespace n2d2b
