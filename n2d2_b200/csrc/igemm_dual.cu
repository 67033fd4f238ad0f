// Host side of the kernel of a branch, its projection and their sum (and its kernels of the 32-bit rescale)
#include <algorithm>
#include <string.h>
#include "igemm_dual_kernel.cuh"

namespace n2d2b {

static size_t dual_smem_bytes(int stages, int slot_bytes, size_t resident)
{
    return 1024 + resident + (size_t)stages * slot_bytes + NUM_EPI_WARPS * REGION_BYTES * DUAL_REGIONS + (2 * stages + 2 * MAX_ACC + 2) * 8 + 32
         + DUAL_SETS * FAST_NP * 256 * 4 + 64;
}

static long long dual_tiles_per_cta(const ConvGeom& g, int bn, int num_sms)
{
    const long long tiles = ((long long)g.B * g.oH * g.oW + BM - 1) / BM * ((g.O + bn - 1) / bn);
    return (tiles + num_sms - 1) / num_sms;
}

// Whether the weights of a CTA's column block stay in shared memory: for a single tile they would all have to arrive before its first multiplication
static bool dual_resident(const ConvGeom* g, int bn, int num_sms)
{
    long long weights = 0;
    for (int s = 0; s < 2; ++s) weights += (long long)g[s].kH * g[s].kW * g[s].C * bn;
    return weights <= 96 * 1024 && dual_tiles_per_cta(g[1], bn, num_sms) > 1;
}

// Columns of a tile by an estimate in cycles like igemm_tile_columns', for two multiplications and both rescales.  Tiles of 128 columns keep two
// tiles' accumulators in TMEM: the longer of loads and epilogue, and 0.4 of the shorter.  Tiles of 256 keep one: each multiplication runs under the
// epilogue of the other one, 0.4 of it the branch's.  An activation block then serves twice the columns, which pays where the operand loads bound
// the tile: 256 + 512 channels into 1024 at 1024 images of 14 x 14 go from 220 us to 172, 512 + 1024 into 2048 at 7 x 7 from 183 to 136 (at 128 images
// from 31.3 to 26.9), but 64 + 64 into 256 at 55 x 55 and 128 images from 65.7 to 67.9.  Fitted to 33 calls of
// 4 to 1024 images.
static int dual_tile_columns(const ConvGeom* g, const int* bk, const bool* im2col, int num_sms)
{
    const long long m_tiles = ((long long)g[1].B * g[1].oH * g[1].oW + BM - 1) / BM;
    auto cost = [&](int bn) {
        const long long tiles = m_tiles * ((g[1].O + bn - 1) / bn), per_cta = dual_tiles_per_cta(g[1], bn, num_sms);
        const double rate = tiles < num_sms ? 114.0 - 43.0 * tiles / num_sms : 71.0;
        const bool resident = dual_resident(g, bn, num_sms);
        double k[2];
        for (int s = 0; s < 2; ++s) {
            const double blocks = (double)g[s].kH * g[s].kW * ((g[s].C + bk[s] - 1) / bk[s]);
            const double load = bk[s] * (BM / (im2col[s] ? std::min(rate, 34.0) : rate) + (resident ? 0 : bn) / rate);
            k[s] = blocks * std::max((bn == 64 ? 48.0 : 0.5 * bn) * bk[s] / 32, load);
        }
        const double epi = bn * (bn == 256 ? 23.0 : (bn == 128 ? 24.0 : 26.0)), sum = k[0] + k[1];
        const double tile = bn == 256 ? std::max(k[1], 0.4 * epi) + std::max(k[0], 0.6 * epi) : std::max(sum, epi) + 0.4 * std::min(sum, epi);
        return per_cta * (per_cta > 1 ? tile : sum) + epi * (bn == 256 ? 1.25 : 1.0);
    };
    if (g[1].O <= 64) return 64;
    const int bn = cost(64) < 0.93 * cost(128) ? 64 : 128;
    return g[1].O > 128 && cost(256) < 0.97 * cost(bn) ? 256 : bn;
}

// a: the branch, b: the projection, both with the output's extents and weights permuted in blocks of 32 channels
int dual_make_plan(DualPlan* plan, const void* in_a, const int8_t* w_a, const ConvGeom& ga, int a_unsigned, const void* in_b, const int8_t* w_b, const ConvGeom& gb,
                   int b_unsigned, const void* out, int num_sms, const char** why)
{
    static const char* kWhy = "";
    *why = kWhy;
    memset(plan, 0, sizeof(*plan));
    const ConvGeom g[2] = {ga, gb};
    if (ga.groups != 1 || gb.groups != 1 || ga.C % 16 || gb.C % 16 || ga.O != gb.O || ga.oH != gb.oH || ga.oW != gb.oW || gb.O % 32) { *why = "extents"; return -1; }
    int bk[2];
    bool im2col[2];
    for (int s = 0; s < 2; ++s) {
        bk[s] = g[s].C % 128 == 0 ? 128 : (g[s].C % 64 == 0 ? 64 : 32);
        im2col[s] = !(g[s].kH == 1 && g[s].kW == 1 && g[s].sX == 1 && g[s].sY == 1 && g[s].pT == 0 && g[s].pL == 0);
    }
    const int bn = dual_tile_columns(g, bk, im2col, num_sms);
    if (igemm_make_plan(&plan->a, in_a, w_a, out, nullptr, ga, a_unsigned, 0, bn, num_sms, why)) return -1;
    if (igemm_make_plan(&plan->b, in_b, w_b, out, nullptr, gb, b_unsigned, 0, bn, num_sms, why)) return -1;
    if (!plan->b.has_out_maps || plan->a.parts != plan->b.parts || bn / plan->b.parts < 32 || (gb.O + bn - 1) / bn > num_sms) { *why = "tiling"; return -1; }
    size_t weights = 0;
    int a_most = 0, slot = 0;
    for (int s = 0; s < 2; ++s) {
        const IgemmPlan& p = s ? plan->b : plan->a;
        weights += (size_t)p.taps * ((p.Cin + p.BK - 1) / p.BK) * p.BK * bn;
        a_most = std::max(a_most, BM * p.BK);
        slot = std::max(slot, (BM + bn) * p.BK);
    }
    plan->resident = dual_resident(g, bn, num_sms) ? 1 : 0;
    auto depth = [&] {
        int st = 8;
        while (st > 2 && dual_smem_bytes(st, plan->slot_bytes, plan->resident ? weights : 0) > 226 * 1024) --st;
        return st;
    };
    plan->slot_bytes = plan->resident ? a_most : slot;
    plan->stages = depth();
    if (plan->resident && plan->stages < 3) {
        plan->resident = 0;
        plan->slot_bytes = slot;
        plan->stages = depth();
    }
    plan->smem_bytes = dual_smem_bytes(plan->stages, plan->slot_bytes, plan->resident ? weights : 0);
    if (plan->smem_bytes > 226 * 1024) { *why = "the tile ring does not fit shared memory"; return -1; }
    return 0;
}

cudaError_t launch_dual(const DualPlan& plan, const ConvGeom& gb, const FastQuant& fa, const FastQuant& fb, int branch_unsigned, int m_base, int late_weights,
                        int* status_word, cudaStream_t s)
{
    const IgemmPlan* const p[2] = {&plan.a, &plan.b};
    const IgemmPlan& q = plan.b;
    const int M = gb.B * gb.oH * gb.oW;
    if (M == 0) return cudaSuccess;
    DualArgs d;
    memset(&d, 0, sizeof(d));
    IgemmArgs& a = d.g;
    a.m_base = m_base;
    a.M = M; a.N = q.N; a.BN = q.BN; a.stages = plan.stages; a.b_resident = plan.resident; a.late_weights = late_weights;
    a.oW = q.oW; a.oH = q.oH;
    a.num_m_tiles = (M + BM - 1) / BM;
    a.num_n_tiles = (q.N + q.BN - 1) / q.BN;
    a.parts = q.parts; a.groups = 4 / q.parts;
    int first = 0;
    for (int i = 0; i < 2; ++i) {
        DualSegment& g = d.seg[i];
        g.BK = p[i]->BK;
        g.kchunks = (p[i]->Cin + g.BK - 1) / g.BK;
        g.num_kb = p[i]->taps * g.kchunks;
        g.tail = p[i]->Cin - (g.kchunks - 1) * g.BK;
        g.im2col = p[i]->a_im2col; g.kW = p[i]->kW; g.sX = p[i]->sX; g.sY = p[i]->sY; g.pL = p[i]->pL; g.pT = p[i]->pT; g.dX = p[i]->dX; g.dY = p[i]->dY;
        g.a_bytes = BM * g.BK;
        g.b_bytes = q.BN * g.BK;
        g.tx = g.a_bytes + (plan.resident ? 0 : g.b_bytes);
        g.idesc = (2u << 4) | ((p[i]->a_unsigned ? 0u : 1u) << 7) | (1u << 10) | ((unsigned)(q.BN >> 3) << 17) | ((unsigned)(BM >> 4) << 24);
        g.b_first = first;
        first += g.num_kb * g.b_bytes;
    }
    d.slot_bytes = plan.slot_bytes;
    a.takers = (d.seg[0].num_kb + d.seg[1].num_kb) * 550 / (q.BN * 16) + 1;
    a.takers = std::min(a.takers, std::min(plan.stages, NUM_PRODUCERS));
    a.status = status_word;
    a.fq = fb.fq; a.fq2 = fb.fq2; a.cpad = fb.cpad; a.t_lo = fb.t_lo; a.t_hi = fb.t_hi;
    const bool t_unsigned = fb.dp4a ? fb.dp_t_unsigned : (fb.t_lo == 0);
    a.ef = (fb.out_unsigned ? EF_OUT_UNSIGNED : 0) | (branch_unsigned ? EF_RES_UNSIGNED : 0) | (t_unsigned ? EF_T_UNSIGNED : 0)
         | (fb.dp_a_signed ? EF_DP_A_SIGNED : 0) | fb.form;
    d.fq_a = fa.fq; d.cpad_a = fa.cpad; d.clamp_a = fa.need_clamp ? 1 : 0;
    d.ef_a = (fa.out_unsigned ? EF_OUT_UNSIGNED : 0) | fa.form;
    a.acc_shift = q.parts == 4 ? 1 : (q.parts == 2 ? 2 : 3);
    a.tmem_cols = (unsigned)q.BN << a.acc_shift;
    const int tiles = a.num_m_tiles * a.num_n_tiles;
    int grid = std::min(q.num_sms, tiles);
    if (tiles > grid && a.num_n_tiles > 1) grid -= grid % a.num_n_tiles;   // every CTA keeps its column block
    auto pixels = [&](long long m) {
        PixelStep t;
        t.x = (int)(m % a.oW);
        t.y = (int)(m / a.oW % a.oH);
        t.n = (int)(m / a.oW / a.oH);
        return t;
    };
    a.step_m = std::max(1, grid / a.num_n_tiles);
    a.adv_tiles = pixels((long long)a.step_m * BM);
    static const DualKernel dual_int[3] = {igemm_dual_tcgen05_kernel<2, DUAL_INT>, igemm_dual_tcgen05_kernel<4, DUAL_INT>, igemm_dual_tcgen05_kernel<5, DUAL_INT>};
    static SmemLimitSet limits[3][3];
    const int forms = !fb.form && !fa.form ? DUAL_INT : (fb.form == EF_FLOAT && fa.form == EF_FLOAT ? DUAL_FLOAT : DUAL_ANY);
    const int v = fb.need_clamp ? 0 : (fb.dp4a ? 2 : 1);
    const DualKernel kernel = (forms == DUAL_INT ? dual_int : (forms == DUAL_FLOAT ? dual_float : dual_any))[v];
    if (!kernel) return cudaErrorInvalidConfiguration;
    if (cudaError_t e = raise_smem_limit(kernel, limits[forms][v])) return e;
    return launch_pdl(kernel, grid, NUM_THREADS, plan.smem_bytes, s, plan.a.tmA, plan.a.tmB, plan.b.tmA, plan.b.tmB, plan.b.tmO, d);
}

}  // namespace n2d2b
