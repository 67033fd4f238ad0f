// Host side of the kernel of an expansion with its residual sum and the 1x1 layer behind it (and its kernels of the 32-bit rescale)
#include <algorithm>
#include <string.h>
#include "igemm_chain_kernel.cuh"

namespace n2d2b {

static size_t chain_smem_bytes(int C, int N2, int slots)
{
    return 1024 + (size_t)slots * CH_SLOT_BYTES + (size_t)CH_STAGES * BM * C + (size_t)CH_N * C + (size_t)4 * N2 * 64 + 3 * FAST_NP * 256 * 4 + CH_BARS * 8 + 32;
}

// The expansion `g` with its residual sum, and the layer `p` behind it
bool chain_eligible(const ConvGeom& g, const ConvGeom& p)
{
    auto plain = [](const ConvGeom& c) {
        return c.groups == 1 && c.kH == 1 && c.kW == 1 && c.sX == 1 && c.sY == 1 && c.pT == 0 && c.pL == 0 && c.oH == c.H && c.oW == c.W;
    };
    return plain(g) && plain(p) && g.O == CH_N && p.C == CH_N && (g.C == 64 || g.C == 128) && p.O % 32 == 0 && p.O <= 128 && p.H == g.oH && p.W == g.oW
        && chain_smem_bytes(g.C, p.O, 3) <= 226 * 1024;
}

int chain_make_plan(ChainPlan* plan, const void* in, const int8_t* w, const void* y, const void* res, const ConvGeom& g, int in_unsigned, const int8_t* w_next,
                    const ConvGeom& p, int y_unsigned, int num_sms, const char** why)
{
    static const char* kWhy = "";
    *why = kWhy;
    memset(plan, 0, sizeof(*plan));
    if (igemm_make_plan(&plan->a, in, w, y, res, g, in_unsigned, 0, 128, num_sms, why)) return -1;
    if (!plan->a.has_out_maps || plan->a.parts != 2 || plan->a.a_im2col || plan->a.BK != g.C || ((uintptr_t)w_next & 15)) { *why = "tiling"; return -1; }
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                               CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    cudaDriverEntryPointQueryResult qr;
    void* fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) != cudaSuccess || !fn) { *why = "cuTensorMapEncodeTiled is not available"; return -1; }
    const cuuint64_t dims[2] = {(cuuint64_t)CH_N, (cuuint64_t)p.O};
    const cuuint64_t strides[1] = {(cuuint64_t)CH_N};
    const cuuint32_t box[2] = {64, (cuuint32_t)p.O};
    const cuuint32_t estr[2] = {1, 1};
    if (((Encode)fn)(&plan->tmB2, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)w_next, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) { *why = "no tensor map of the weights"; return -1; }
    plan->C = g.C;
    plan->N2 = p.O;
    plan->y_unsigned = y_unsigned;
    plan->slots = chain_smem_bytes(g.C, p.O, 4) <= 226 * 1024 ? 4 : 3;
    plan->smem_bytes = chain_smem_bytes(g.C, p.O, plan->slots);
    return 0;
}

cudaError_t launch_chain(const ChainPlan& plan, int M, const FastQuant& fast, int res_unsigned, const FastQuant& next, void* out, int m_base, int* status_word,
                         cudaStream_t s)
{
    if (M == 0) return cudaSuccess;
    ChainArgs a;
    memset(&a, 0, sizeof(a));
    a.M = M; a.m_base = m_base; a.C = plan.C; a.N2 = plan.N2; a.slots = plan.slots;
    a.idesc1 = (2u << 4) | ((plan.a.a_unsigned ? 0u : 1u) << 7) | (1u << 10) | ((128u >> 3) << 17) | ((unsigned)(BM >> 4) << 24);
    a.idesc2 = (2u << 4) | ((plan.y_unsigned ? 0u : 1u) << 7) | (1u << 10) | ((unsigned)(plan.N2 >> 3) << 17) | ((unsigned)(BM >> 4) << 24);
    a.fq = fast.fq; a.fq2 = fast.fq2; a.cpad = fast.cpad;
    a.fq_next = next.fq; a.cpad_next = next.cpad;
    const bool t_unsigned = fast.dp4a ? fast.dp_t_unsigned : (fast.t_lo == 0);
    a.ef = (fast.out_unsigned ? EF_OUT_UNSIGNED : 0) | (res_unsigned ? EF_RES_UNSIGNED : 0) | (t_unsigned ? EF_T_UNSIGNED : 0)
         | (fast.dp_a_signed ? EF_DP_A_SIGNED : 0) | fast.form;
    a.t_lo = fast.t_lo; a.t_hi = fast.t_hi;
    a.ef_next = (next.out_unsigned ? EF_OUT_UNSIGNED : 0) | next.form;
    a.clamp_next = next.need_clamp ? 1 : 0;
    a.out = (uint8_t*)out;
    a.status = status_word;
    static const ChainKernel chain_int[3] = {igemm_chain_tcgen05_kernel<2, CHAIN_INT>, igemm_chain_tcgen05_kernel<4, CHAIN_INT>, igemm_chain_tcgen05_kernel<5, CHAIN_INT>};
    static SmemLimitSet limits[3][3];
    const int forms = !fast.form && !next.form ? CHAIN_INT : (fast.form == EF_FLOAT && next.form == EF_FLOAT ? CHAIN_FLOAT : CHAIN_ANY);
    const int v = fast.need_clamp ? 0 : (fast.dp4a ? 2 : 1);
    const ChainKernel kernel = (forms == CHAIN_INT ? chain_int : (forms == CHAIN_FLOAT ? chain_float : chain_any))[v];
    if (!kernel) return cudaErrorInvalidConfiguration;
    if (cudaError_t e = raise_smem_limit(kernel, limits[forms][v])) return e;
    const int tiles = (M + BM - 1) / BM;
    return launch_pdl(kernel, std::min(plan.a.num_sms, tiles), CH_THREADS, plan.smem_bytes, s, plan.a.tmA, plan.a.tmB, plan.tmB2, plan.a.tmO, plan.a.tmR, a);
}

}  // namespace n2d2b
