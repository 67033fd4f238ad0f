// Implicit GEMM: 256-row tiles, tiles shared by a cluster, and the host side (the main kernel: igemm_kernel.cuh)
#include <cstdio>
#include <cstring>
#include <algorithm>
#include "igemm_kernel.cuh"

namespace n2d2b {

// ----------------------------------------------------------------------------- 256-row tiles
// Large-K layers with 256 output channels per tile are bound by L2-to-shared bandwidth at 128 x 256 tiles
// (48 KB per K slab for 512 cycles of MMA).  This variant gives a CTA two 128-row tiles that share every
// weight slab: 64 KB per slab for 1024 cycles of MMA.  Both TMEM accumulators belong to the pair, so the
// epilogue of a pair does not overlap the MMAs of the next one - affordable when K is large.  No residual, the
// 32-bit epilogue only; the staging regions are 1 KB (32 rows x 32 columns, two passes per warp) to make
// room for three 64 KB stages.
static constexpr int PAIR_STAGES = 3;
static_assert(NUM_PRODUCERS <= PAIR_STAGES, "a producer may be at most one ring ahead of the issuer (see the producers above)");
static constexpr int PAIR_REGION = 1024;

template <bool CLAMP>
__global__ void __launch_bounds__(NUM_THREADS, 1)
igemm_pair_i8_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                             const __grid_constant__ CUtensorMap tmO32, const IgemmArgs a)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int A_BYTES = BM * 128, B_BYTES = 256 * 128, STAGE_BYTES = 2 * A_BYTES + B_BYTES;
    unsigned char* tiles = smem;
    unsigned char* stage_out = tiles + (size_t)PAIR_STAGES * STAGE_BYTES;
    unsigned long long* bars = (unsigned long long*)(stage_out + NUM_EPI_WARPS * PAIR_REGION);
    // bars: full[3], empty[3], tmem_full[2], tmem_empty[2], params_ready
    const unsigned full0 = smem_u32(bars);
    const unsigned empty0 = full0 + 8u * PAIR_STAGES;
    const unsigned tfull0 = empty0 + 8u * PAIR_STAGES;
    const unsigned tempty0 = tfull0 + 16u;
    const unsigned pready = tempty0 + 16u;
    unsigned* tmem_slot = (unsigned*)(bars + 2 * PAIR_STAGES + 6);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    int* par = (int*)(((uintptr_t)(tmem_slot + 4) + 15) & ~(uintptr_t)15);   // [FAST_NP][256]

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    const int producer = warp == 0 ? 0 : (warp >= EPI_WARP0 + NUM_EPI_WARPS ? warp - (EPI_WARP0 + NUM_EPI_WARPS) + 1 : -1);
    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < PAIR_STAGES; ++s) {
            mbar_init(full0 + 8u * s, 1);
            mbar_init(empty0 + 8u * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(tfull0 + 8u * s, 1);
            mbar_init(tempty0 + 8u * s, NUM_EPI_WARPS);
        }
        mbar_init(pready, NUM_EPI_WARPS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = *tmem_slot;
    const int num_pairs = (a.num_m_tiles + 1) / 2;
    const int num_pt = num_pairs * a.num_n_tiles;          // pair tiles, column block fastest
    const int kchunks = a.Cin / 128;
    const int num_kb = a.taps * kchunks;
    const int m_end = a.m_base + a.M;

    if (producer >= 0) {
        // ------------------------------------------------------------------ TMA producers (as in the kernel above)
        bool ok = true;
        int m_pair = (int)blockIdx.x / a.num_n_tiles, n_tile = (int)blockIdx.x - m_pair * a.num_n_tiles;
        int m0 = a.m_base + 2 * m_pair * BM, n0 = n_tile * 256;
        PixelPos px;
        px.start(a, m0);
        const unsigned tiles_s = smem_u32(tiles);
        unsigned pre = 0;
        if (a.late_weights) pdl_wait();
        if ((int)blockIdx.x < num_pt) {
            pre = (unsigned)(num_kb < PAIR_STAGES ? num_kb : PAIR_STAGES);
            if (elect_one()) {
                if (producer == 0) {
                    prefetch_tensor_map(&tmA);
                    prefetch_tensor_map(&tmO32);
                }
                int kc = 0, kcoord = 0, turn = producer;
                for (unsigned i = 0; i < pre; ++i) {
                    if (turn == 0) {
                        turn = NUM_PRODUCERS;
                        mbar_expect_tx(full0 + 8u * i, (unsigned)STAGE_BYTES);
                        tma_load_2d(tiles_s + i * (unsigned)STAGE_BYTES + 2u * A_BYTES, &tmB, full0 + 8u * i, kcoord, n0);
                    }
                    --turn;
                    if (++kc == kchunks) {
                        kc = 0;
                        kcoord += a.Cin - (kchunks - 1) * 128;
                    } else {
                        kcoord += 128;
                    }
                }
            }
            __syncwarp();
        }
        pdl_wait();
        const bool im2col = a.a_im2col != 0;
        unsigned bar = full0, dst = tiles_s, ph = 1u, it = 0;
        int turn = producer;
        for (int pt = blockIdx.x; pt < num_pt && ok; pt += gridDim.x) {
            PixelPos p2 = px;
            p2.advance(a, a.adv_one);
            const int iw0 = px.ox * a.sX - a.pL, ih0 = px.oy * a.sY - a.pT, in0 = px.n;
            const int iw1 = p2.ox * a.sX - a.pL, ih1 = p2.oy * a.sY - a.pT, in1 = p2.n;
            int kx = 0, ky = 0, kc = 0, kcoord = 0;
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                if (turn == 0) {
                    turn = NUM_PRODUCERS;
                    if (!mbar_wait_issuer(bar + 8u * PAIR_STAGES, ph, abort_flag, a.status, 1)) { ok = false; break; }
                    if (elect_one()) {
                        const bool weights = it >= pre;
                        if (weights) mbar_expect_tx(bar, (unsigned)STAGE_BYTES);
                        if (im2col) {
                            const unsigned short ox = (unsigned short)(kx * a.dX), oy = (unsigned short)(ky * a.dY);
                            tma_load_im2col_4d(dst, &tmA, bar, kc * 128, iw0, ih0, in0, ox, oy);
                            tma_load_im2col_4d(dst + A_BYTES, &tmA, bar, kc * 128, iw1, ih1, in1, ox, oy);
                        } else {
                            tma_load_2d(dst, &tmA, bar, kcoord, m0);
                            tma_load_2d(dst + A_BYTES, &tmA, bar, kcoord, m0 + BM);
                        }
                        if (weights) tma_load_2d(dst + 2 * A_BYTES, &tmB, bar, kcoord, n0);
                    }
                    __syncwarp();
                }
                --turn;
                bar += 8u;
                dst += (unsigned)STAGE_BYTES;
                if (bar == full0 + 8u * PAIR_STAGES) { bar = full0; dst = tiles_s; ph ^= 1u; }
                if (++kc == kchunks) {
                    kc = 0;
                    kcoord += a.Cin - (kchunks - 1) * 128;
                    if (++kx == a.kW) { kx = 0; ++ky; }
                } else {
                    kcoord += 128;
                }
            }
            m_pair += a.step_m;
            n_tile += a.step_n;
            px.advance(a, a.adv_tiles);
            if (n_tile >= a.num_n_tiles) {
                n_tile -= a.num_n_tiles;
                ++m_pair;
                px.advance(a, a.adv_one);
                px.advance(a, a.adv_one);
            }
            m0 = a.m_base + 2 * m_pair * BM;
            n0 = n_tile * 256;
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const unsigned desc_hi = (unsigned)(make_smem_desc(0u, 128) >> 32);
        const unsigned t_lo0 = (smem_u32(tiles) & 0x3ffffu) >> 4;
        const unsigned stage16 = (unsigned)(STAGE_BYTES >> 4), a16 = (unsigned)(A_BYTES >> 4);
        int s = 0;
        unsigned ph = 0, pit = 0, a_lo = t_lo0;
        bool ok = true;
        for (int pt = blockIdx.x; pt < num_pt && ok; pt += gridDim.x, ++pit) {
            const unsigned aph = pit & 1u;
            if (!mbar_wait_issuer(tempty0, aph ^ 1u, abort_flag, a.status, 2)) { ok = false; break; }
            if (!mbar_wait_issuer(tempty0 + 8u, aph ^ 1u, abort_flag, a.status, 2)) { ok = false; break; }
            for (int kb = 0; kb < num_kb; ++kb) {
                if (!mbar_wait_issuer(full0 + 8u * s, ph, abort_flag, a.status, 3)) { ok = false; break; }
                tc_fence_after();
                const unsigned al0 = a_lo, b_lo = a_lo + 2u * a16;
                const unsigned acc = kb ? 1u : 0u, ebar = empty0 + 8u * s;
                a_lo += stage16;
                if (++s == PAIR_STAGES) { s = 0; ph ^= 1u; a_lo = t_lo0; }
                if (elect_one()) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const unsigned d_tmem = tmem_base + (unsigned)(h * 256);
                        const unsigned al = al0 + (unsigned)h * a16;
                        tc_mma_i8_lohi(d_tmem, al, b_lo, desc_hi, a.idesc, acc);
                        tc_mma_i8_lohi(d_tmem, al + 2u, b_lo + 2u, desc_hi, a.idesc, 1u);
                        tc_mma_i8_lohi(d_tmem, al + 4u, b_lo + 4u, desc_hi, a.idesc, 1u);
                        tc_mma_i8_lohi(d_tmem, al + 6u, b_lo + 6u, desc_hi, a.idesc, 1u);
                    }
                    tc_commit(ebar);
                    if (kb + 1 == num_kb) {
                        tc_commit(tfull0);
                        tc_commit(tfull0 + 8u);
                    }
                }
                __syncwarp();
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue warps
        const int ew = warp - EPI_WARP0;
        const int quad = warp & 3;
        const int part = ew >> 2;                        // a quarter of the 256 columns
        const int cbase = part * 64;
        const unsigned par_off = (unsigned)((unsigned char*)par - smem_raw);
        const unsigned region_off = (unsigned)(stage_out - smem_raw) + (unsigned)(ew * PAIR_REGION);
        const unsigned region = smem_u32(stage_out + (size_t)ew * PAIR_REGION);
        unsigned rb[4];
        perm_rowbase(rb, 32, lane, 4);
        // the launch keeps every CTA on one column block: its constants are staged once
        const int n0 = ((int)blockIdx.x % a.num_n_tiles) * 256;
        for (int i = ew * 32 + lane; i < FAST_NP * 256; i += 32 * NUM_EPI_WARPS) {
            const int prm = i >> 8, c = i & 255;
            par[i] = (n0 + c < a.cpad) ? __ldg(a.fq + (size_t)prm * a.cpad + n0 + c) : 0;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(pready);
        bool ok = mbar_wait_warp(pready, 0, abort_flag, a.status, 5);
        pdl_wait();
        unsigned pit = 0;
        int m_pair = (int)blockIdx.x / a.num_n_tiles;
        const int gx = n0 + cbase;
        for (int pt = blockIdx.x; pt < num_pt && ok; pt += gridDim.x, ++pit) {
            const int pair_now = m_pair;
            {
                // same stepping as the producer; the column block stays
                const int n_tile = (int)blockIdx.x % a.num_n_tiles;
                m_pair += a.step_m + ((n_tile + a.step_n >= a.num_n_tiles) ? 1 : 0);
            }
#pragma unroll 1
            for (int h = 0; h < 2 && ok; ++h) {
                const int gy = a.m_base + (2 * pair_now + h) * BM + quad * 32;
                const bool active = gx < a.N && gy < m_end;
                if (!mbar_wait_warp(tfull0 + 8u * h, pit & 1u, abort_flag, a.status, 4)) { ok = false; break; }
                tc_fence_after();
                const unsigned tbase = tmem_base + ((unsigned)(quad * 32) << 16) + (unsigned)(h * 256 + cbase);
#pragma unroll 1
                for (int pass = 0; pass < 2; ++pass) {
                    if (lane == 0) bulk_wait_read_all();   // the previous store has finished reading the region
                    __syncwarp();
                    if (active) {
                        unsigned va[16], vb[16];
                        tc_ld_2x16x256b_x4_wait(tbase + (unsigned)(32 * pass), va, vb);
                        const int pc = cbase + 32 * pass;
                        switch (a.ef & (EF_OUT_UNSIGNED | EF_WIDE | EF_FLOAT)) {
                        case 0: perm_block<4, false, CLAMP, false, EF_PERM>(va, vb, par_off, pc, region_off, rb, 0, lane, 0, 0); break;
                        case EF_OUT_UNSIGNED:
                            perm_block<4, false, CLAMP, false, EF_OUT_UNSIGNED | EF_PERM>(va, vb, par_off, pc, region_off, rb, 0, lane, 0, 0);
                            break;
                        case EF_WIDE: perm_block<4, false, CLAMP, false, EF_WIDE | EF_PERM>(va, vb, par_off, pc, region_off, rb, 0, lane, 0, 0); break;
                        case EF_WIDE | EF_OUT_UNSIGNED:
                            perm_block<4, false, CLAMP, false, EF_WIDE | EF_OUT_UNSIGNED | EF_PERM>(va, vb, par_off, pc, region_off, rb, 0, lane, 0, 0);
                            break;
                        case EF_FLOAT: perm_block<4, false, CLAMP, false, EF_FLOAT | EF_PERM>(va, vb, par_off, pc, region_off, rb, 0, lane, 0, 0); break;
                        default:
                            perm_block<4, false, CLAMP, false, EF_FLOAT | EF_OUT_UNSIGNED | EF_PERM>(va, vb, par_off, pc, region_off, rb, 0, lane, 0, 0);
                            break;
                        }
                    }
                    if (pass == 1) {
                        // the accumulator is drained: hand it back before the store goes out
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(tempty0 + 8u * h);
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0 && active) {
                        tma_store_2d(&tmO32, region, gx + 32 * pass, gy);
                        bulk_commit();
                    }
                }
            }
        }
        if (lane == 0) bulk_wait_read_all();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// ----------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*EncodeIm2colFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const int*, const int*, cuuint32_t, cuuint32_t,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn g_encode_tiled = nullptr;
static EncodeIm2colFn g_encode_im2col = nullptr;

static int load_driver_entry_points(const char** why)
{
    if (g_encode_tiled && g_encode_im2col) return 0;
    cudaDriverEntryPointQueryResult qr;
    void* fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) != cudaSuccess || !fn) {
        *why = "cuTensorMapEncodeTiled is not available from the CUDA driver";
        return -1;
    }
    g_encode_tiled = (EncodeTiledFn)fn;
    fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &fn, cudaEnableDefault, &qr) != cudaSuccess || !fn) {
        *why = "cuTensorMapEncodeIm2col is not available from the CUDA driver";
        return -1;
    }
    g_encode_im2col = (EncodeIm2colFn)fn;
    return 0;
}

static CUtensorMapSwizzle swizzle_for(int bk)
{
    return bk == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
         : (bk == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : (bk == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE));
}

// resident_b = bytes of the weight block kept in shared memory for the whole launch (0: weights ride the ring)
// regions = staging regions per epilogue warp (1; 2 or 4 with a fused residual)
// w4: a stage also holds the packed form of its weight block, and one more barrier
static size_t igemm_smem_bytes(int stages, int BK, int BN, int regions, size_t resident_b, int w4 = 0)
{
    return 1024 /*alignment slack*/ + resident_b + (size_t)stages * ((BM + (resident_b ? 0 : BN)) * BK + (w4 ? BN * BK / 2 : 0))
         + NUM_EPI_WARPS * REGION_BYTES * regions
         + (2 * stages + 2 * MAX_ACC + 4 + 4 * NUM_EPI_WARPS + (w4 ? stages : 0)) * 8 + 32 + 2 * 2 * FAST_NP * 256 * 4 + 64;
}

// Channels per block-diagonal group of a depthwise layer this kernel takes (0: not such a layer): groups of 64
// channels = one 64-column tile each, or a single group of 32
int igemm_dw_group(const ConvGeom& g)
{
    if (g.groups <= 1 || g.groups != g.C || g.O != g.C || g.Cg != 1 || g.Og != 1) return 0;
    if (g.C % 64 == 0) return 64;
    if (g.C == 32) return 32;
    return 0;
}

size_t igemm_dw_weight_bytes(const ConvGeom& g) { return (size_t)g.C * g.kH * g.kW * igemm_dw_group(g); }

// Depthwise weights [C][taps] as the block-diagonal matrix [C][taps][group channels] (real channel order)
void igemm_dw_arrange_weights(const ConvGeom& g, const int8_t* w_ct, int8_t* dst)
{
    const int cg = igemm_dw_group(g), taps = g.kH * g.kW;
    const size_t row_bytes = (size_t)taps * cg;
    memset(dst, 0, (size_t)g.C * row_bytes);
    for (int o = 0; o < g.C; ++o)
        for (int t = 0; t < taps; ++t) dst[(size_t)o * row_bytes + (size_t)t * cg + (o % cg)] = w_ct[(size_t)o * taps + t];
}

// Columns of a tile: 256, 128 or 64, whichever finishes the busiest CTA first by an estimate in cycles.  A K block costs its MMAs
// (128 x 256 x 32 128 cycles, x 128 64, x 64 48) or, where that is longer, its loads (71 bytes per clock and SM with
// all of them loading, 40 through an im2col map; resident weights are loaded once), a tile its K blocks or its epilogue (a cycle count per column that is
// smaller where two or four groups of warps drain a tile each), a CTA its tiles and one epilogue nothing covers.  Wide tiles
// load the least per value; narrow ones fill the chip when there are few rows, or its second wave.  With a residual sum 256
// columns never pay (conv5.2 of ResNet-50 at 1024 images 90 us against 74 with two tiles in the epilogue at once).
// ResNet-50 at 33 images 481 -> 464 us against a rule that only filled the chip, ResNet-18 at 64 images 310 -> 291.
static int igemm_tile_columns(const ConvGeom& g, int BK, bool im2col, bool res, int w4, int num_sms, int force_pair)
{
    const int widest = g.O >= 256 && !res ? 256 : (g.O > 64 ? 128 : 64);
    if (force_pair) return widest;
    const long long m_tiles = ((long long)g.B * g.oH * g.oW + BM - 1) / BM;
    const int num_kb = g.kH * g.kW * ((g.C + BK - 1) / BK);
    int best_bn = widest;
    double best = 0;
    for (int bn = widest; bn >= 64; bn >>= 1) {
        const long long n_tiles = (g.O + bn - 1) / bn, tiles = m_tiles * n_tiles, per_cta = (tiles + num_sms - 1) / num_sms;
        const bool resident = !w4 && (long long)num_kb * BK * bn <= 96 * 1024 && (n_tiles == 1 || num_sms > n_tiles);
        const double mma = (bn == 256 ? 128.0 : (bn == 128 ? 64.0 : 48.0)) * BK / 32;
        const double rate = tiles < num_sms ? 114.0 - 43.0 * tiles / num_sms : 71.0;
        const double load = BK * (BM / (im2col ? std::min(rate, 40.0) : rate) + (resident && per_cta > 1 ? 0 : bn) / rate);
        const double epi = bn * (bn == 256 ? 10.0 : (bn == 128 ? 11.0 : 15.0)) * (res ? 1.9 : 1.0);
        const double cost = per_cta * std::max(num_kb * std::max(mma, load), per_cta > 1 ? epi : 0.0) + epi;
        if (best == 0 || cost < 0.93 * best) { best = cost; best_bn = bn; }
    }
    return best_bn;
}

// The map of the activations: `g.B` images at `in`, Ct channels per pixel (g: one group of a layer of several)
static int encode_activations(IgemmPlan* plan, const void* in, const ConvGeom& g, int Ct, const char** why)
{
    const CUtensorMapSwizzle swz = swizzle_for(plan->BK);
    CUresult rc;
    if (!plan->a_im2col) {
        const cuuint64_t dims[2] = {(cuuint64_t)g.C, (cuuint64_t)g.B * g.oH * g.oW};
        const cuuint64_t strides[1] = {(cuuint64_t)g.C};
        const cuuint32_t box[2] = {(cuuint32_t)plan->BK, (cuuint32_t)BM};
        const cuuint32_t estr[2] = {1, 1};
        rc = g_encode_tiled(&plan->tmA, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)in, dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (rc != CUDA_SUCCESS) { *why = "cuTensorMapEncodeTiled failed for the activation matrix"; return -1; }
    } else {
        // NHWC activations as a (C, W, H, N) tensor; the base pixel of output (ox, oy) is
        // (ox*sX - pL, oy*sY - pT) and the filter tap is passed as an offset per load.
        const cuuint64_t dims[4] = {(cuuint64_t)Ct, (cuuint64_t)g.W, (cuuint64_t)g.H, (cuuint64_t)g.B};
        const cuuint64_t strides[3] = {(cuuint64_t)Ct, (cuuint64_t)Ct * g.W, (cuuint64_t)Ct * g.W * g.H};
        const int lower[2] = {-g.pL, -g.pT};
        // last base pixel = (oW-1)*sX - pL  ->  upper corner relative to the tensor edge
        const int upper[2] = {(g.oW - 1) * g.sX - g.pL - (g.W - 1), (g.oH - 1) * g.sY - g.pT - (g.H - 1)};
        const cuuint32_t estr[4] = {1, (cuuint32_t)g.sX, (cuuint32_t)g.sY, 1};
        rc = g_encode_im2col(&plan->tmA, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, (void*)in, dims, strides, lower, upper,
                             (cuuint32_t)plan->BK, (cuuint32_t)BM, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (rc != CUDA_SUCCESS) { *why = "cuTensorMapEncodeIm2col failed for the activation tensor"; return -1; }
        // Drivers up to CUDA 13.1 encode im2col maps of tensors smaller than 128 KiB with a flag
        // (bit 21 of the second 64-bit word) that makes the load misbehave; clearing it is the
        // documented remedy used by NVIDIA's own open-source templates.
        int drv = 0;
        if (cudaDriverGetVersion(&drv) == cudaSuccess && drv <= 13010) {
            const size_t bytes = (size_t)Ct * g.W * g.H * g.B;
            if (bytes < 131072) reinterpret_cast<unsigned long long*>(&plan->tmA)[1] &= ~(1ull << 21);
        }
    }
    return 0;
}

// The map of the residual operand: `rows` pixels at `res`
static int encode_residual(IgemmPlan* plan, const void* res, long long rows, const char** why)
{
    const int wb = plan->BN / plan->parts;   // an epilogue warp's columns: 64, or 32 or 16 with four warps on a narrow tile
    const cuuint64_t dims[2] = {(cuuint64_t)plan->N, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)plan->N};
    const cuuint32_t box[2] = {(cuuint32_t)wb, 32};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult rc = g_encode_tiled(&plan->tmR, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)res, dims, strides, box, estr,
                                       CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(wb), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) { *why = "cuTensorMapEncodeTiled failed for the residual matrix"; return -1; }
    return 0;
}

int igemm_bind_buffers(IgemmPlan* plan, const void* in, const void* res, const ConvGeom& g0, const char** why)
{
    if (((uintptr_t)in & 15) || ((uintptr_t)res & 15)) { *why = "operands must be 16-byte aligned"; return -1; }
    ConvGeom g = g0;
    if (const int cg = igemm_dw_group(g0)) g.C = cg;
    if (in && encode_activations(plan, in, g, g0.C, why)) return -1;
    return res && plan->has_out_maps ? encode_residual(plan, res, (long long)g.B * g.oH * g.oW, why) : 0;
}

int igemm_make_plan(IgemmPlan* plan, const void* in, const int8_t* w, const void* out, const void* res,
                    const ConvGeom& g0, int in_unsigned, int force_im2col, int force_bn, int num_sms, const char** why,
                    int force_pair, int w4)
{
    static const char* kWhy = "";
    *why = kWhy;
    if (load_driver_entry_points(why)) return -1;
    // A depthwise layer runs as block-diagonal groups: per 64-column tile a dense layer over the tile's own 64 input
    // channels (weights [C][taps * 64], zeros off the diagonal); the activation loads take the group's channel slice.
    ConvGeom g = g0;
    const int Ct = g0.C;          // channels per pixel of the input tensor
    int grouped = 0;
    if (const int cg = igemm_dw_group(g0)) {
        if (w4 || res) { *why = "block-diagonal groups take neither packed weights nor a residual"; return -1; }
        g.C = cg; g.groups = 1; g.Cg = cg; g.Og = g0.O;
        grouped = Ct > cg ? 1 : 0;
        force_im2col = 1;
        force_bn = 64;
        force_pair = 0;
    }
    if (g.groups != 1) { *why = "grouped convolution is not a dense contraction"; return -1; }
    if (g.C % 16 != 0) { *why = "input channels must be a multiple of 16 for the TMA path"; return -1; }
    if (((uintptr_t)in & 15) || ((uintptr_t)w & 15)) { *why = "operands must be 16-byte aligned"; return -1; }
    memset(plan, 0, sizeof(*plan));
    const bool plain = (g.kH == 1 && g.kW == 1 && g.sY == 1 && g.sX == 1 && g.pT == 0 && g.pL == 0
                        && g.oH == g.H && g.oW == g.W);
    plan->a_im2col = (plain && !force_im2col) ? 0 : 1;
    plan->M = g.B * g.oH * g.oW;
    plan->N = g.O;
    plan->Cin = g.C;
    plan->taps = g.kH * g.kW;
    // widest K slab (= swizzle span) that divides the channel count; a channel count that is only a
    // multiple of 16 uses 32-byte slabs whose tail the TMA unit zero-fills
    plan->BK = (g.C % 128 == 0) ? 128 : (g.C % 64 == 0 ? 64 : 32);
    int bn = force_bn;
    if (bn == 0) {
        bn = igemm_tile_columns(g, plan->BK, plan->a_im2col != 0, res != nullptr, w4, num_sms, force_pair);
    }
    plan->BN = bn;
    plan->grouped = grouped;
    // groups of epilogue warps on different tiles need a CTA whose column block never changes
    plan->parts = (g.O + bn - 1) / bn < num_sms ? (bn >= 256 ? 4 : (bn >= 128 ? 2 : 1)) : 4;
    // one tile per CTA: two warps per quadrant share a narrow one (ResNet-50 at one image 263 us against 259; four warps 262)
    if (((long long)g.B * g.oH * g.oW + BM - 1) / BM * ((g.O + bn - 1) / bn) <= num_sms) plan->parts = std::max(plan->parts, 2);
    plan->w4 = w4 ? 1 : 0;
    plan->num_sms = num_sms;
    plan->a_unsigned = in_unsigned;
    plan->oW = g.oW; plan->oH = g.oH; plan->kW = g.kW;
    plan->sX = g.sX; plan->sY = g.sY; plan->pL = g.pL; plan->pT = g.pT; plan->dX = g.dX; plan->dY = g.dY;
    // pipeline depth: fill up to ~200 KB of shared memory, at most 8 stages
    const int with_res = res ? 1 : 0;
    const int num_m_tiles = (plan->M + BM - 1) / BM;
    const int num_n_tiles = (plan->N + plan->BN - 1) / plan->BN;
    const long long tiles = (long long)num_m_tiles * num_n_tiles;
    plan->grid = (int)(tiles < num_sms ? tiles : num_sms);
    if (plan->grid < 1) plan->grid = 1;
    // A CTA whose column block never changes keeps that block's weights in shared memory: the loads of
    // a small-K layer are then activations only.
    const size_t wblock = (size_t)plan->taps * ((g.C + plan->BK - 1) / plan->BK) * plan->BK * plan->BN;
    plan->b_resident = (!w4 && wblock <= 96 * 1024 && (num_n_tiles == 1 || num_sms > num_n_tiles)) ? 1 : 0;
    const int num_kb = plan->taps * ((g.C + plan->BK - 1) / plan->BK);
    auto depth = [&](int regions, size_t resident) {
        int st = 8;
        while (st > 2 && igemm_smem_bytes(st, plan->BK, plan->BN, regions, resident, w4) > 226 * 1024) --st;
        return st;
    };
    auto fits = [&](int st, int regions, size_t resident) {
        return igemm_smem_bytes(st, plan->BK, plan->BN, regions, resident, w4) <= 226 * 1024;
    };
    // A residual cell stages the residual of up to three tiles ahead when that leaves the ring deep enough
    // (four regions per epilogue warp instead of two): its loads then have two tile times to arrive.
    int regions = with_res ? 4 : 1;
    size_t resident = plan->b_resident ? wblock : 0;
    int stages = depth(regions, resident);
    const int want = num_kb + 1 < 4 ? num_kb + 1 : 4;
    if (with_res && (!fits(stages, regions, resident) || stages < want)) {
        regions = 2;
        stages = depth(regions, resident);
    }
    if (plan->b_resident && !fits(stages, regions, resident)) {
        plan->b_resident = 0;
        resident = 0;
        stages = depth(regions, 0);
    }
    plan->stages = stages;
    plan->res_slots = with_res ? regions : 0;
    plan->smem_bytes = igemm_smem_bytes(stages, plan->BK, plan->BN, regions, resident, w4);
    if (!fits(stages, regions, resident)) { *why = "the tile ring does not fit shared memory"; return -1; }

    const CUtensorMapSwizzle swz = swizzle_for(plan->BK);
    CUresult rc;
    // B: weights [N][Ktot], K fastest; packed 4-bit weights: [N][Ktot / 2] bytes, loaded unswizzled (the expansion
    // warps write the swizzled tile)
    {
        const cuuint64_t kbytes = (cuuint64_t)plan->taps * g.C / (w4 ? 2 : 1);
        const cuuint64_t dims[2] = {kbytes, (cuuint64_t)g.O};
        const cuuint64_t strides[1] = {kbytes};
        const cuuint32_t box[2] = {(cuuint32_t)(plan->BK / (w4 ? 2 : 1)), (cuuint32_t)plan->BN};
        const cuuint32_t estr[2] = {1, 1};
        rc = g_encode_tiled(&plan->tmB, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)w, dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, w4 ? CU_TENSOR_MAP_SWIZZLE_NONE : swz,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (rc != CUDA_SUCCESS) { *why = "cuTensorMapEncodeTiled failed for the weight matrix"; return -1; }
    }
    if (encode_activations(plan, in, g, Ct, why)) return -1;
    // output (and residual) as [M][N] bytes, one box = an epilogue warp's 32 rows and columns
    plan->has_out_maps = 0;
    if (out && g.O % 16 == 0 && !((uintptr_t)out & 15) && !((uintptr_t)res & 15)) {
        const int wb = plan->BN / plan->parts;   // an epilogue warp's columns: 64, or 32 or 16 with four warps on a narrow tile
        const cuuint64_t dims[2] = {(cuuint64_t)g.O, (cuuint64_t)plan->M};
        const cuuint64_t strides[1] = {(cuuint64_t)g.O};
        const cuuint32_t box[2] = {(cuuint32_t)wb, 32};
        const cuuint32_t estr[2] = {1, 1};
        rc = g_encode_tiled(&plan->tmO, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)out, dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(wb), CU_TENSOR_MAP_L2_PROMOTION_NONE,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (rc != CUDA_SUCCESS) { *why = "cuTensorMapEncodeTiled failed for the output matrix"; return -1; }
        plan->tmR = plan->tmO;
        if (res && encode_residual(plan, res, plan->M, why)) return -1;
        plan->has_out_maps = 1;
        // 256-row variant: 256-column tiles, 128-byte K slabs, no residual, weights not resident, and enough
        // work per CTA that halving the weight traffic pays for the un-overlapped epilogue
        const int num_kb = plan->taps * (g.C / 128);
        if (plan->BN == 256 && plan->BK == 128 && !res && !plan->b_resident && !w4 && g.O % 32 == 0
            && (force_pair || (num_kb >= 8 && (long long)num_m_tiles * num_n_tiles >= 4ll * num_sms))) {
            const cuuint32_t box32[2] = {32, 32};
            rc = g_encode_tiled(&plan->tmO32, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)out, dims, strides, box32, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (rc == CUDA_SUCCESS) {
                plan->pair = 1;
                plan->pair_smem_bytes = 1024 + (size_t)PAIR_STAGES * (2 * BM * 128 + 256 * 128) + NUM_EPI_WARPS * PAIR_REGION
                                      + (2 * PAIR_STAGES + 6) * 8 + 32 + FAST_NP * 256 * 4 + 64;
            }
        }
    }
    return 0;
}

// ----------------------------------------------------------------------------- few tiles, long K: a cluster per tile
// A late layer at a small batch has a handful of 128 x 64 tiles and up to 36 K blocks, each of which costs one CTA about 400
// cycles of waits, loads and MMAs while most of the chip idles (ResNet-50's 3x3 layers of 7 x 7 maps, one image: 8 tiles).  Here the S = 8
// CTAs of a cluster share a tile: CTA s multiplies its part of K (at most SPLIT_STAGES blocks, each with a stage of its own, so
// nothing ever waits for a slot), sends the 64 / S columns that CTA t finishes to t's shared memory, and finishes its own
// columns from the S partial sums.  Sums of 32-bit integers: the same bits in any order.  A 7 x 7 x 512 3x3
// layer at one image: 16.4 us -> 12.3, ResNet-18 155 us -> 141.
static constexpr int SPLIT = 8;               // CTAs of a cluster
static constexpr int SPLIT_STAGES = 7;
static constexpr int SPLIT_EPI_WARPS = 8;
static constexpr int SPLIT_THREADS = 32 * (EPI_WARP0 + SPLIT_EPI_WARPS);
static constexpr int SPLIT_BN = 64;

struct SplitArgs {
    IgemmArgs g;
    int per;            // K blocks per CTA
    int perm_ng;        // permutation of the stored weight rows (perm_block / 8)
    int form, need_clamp, dp, ef;
};

static size_t split_smem_bytes(int per, int BK)
{
    return 1024 + (size_t)per * (BM + SPLIT_BN) * BK + (size_t)BM * SPLIT_BN * 4 + 2 * FAST_NP * SPLIT_BN * 4 + (SPLIT_STAGES + 1) * 8 + 32;
}

__device__ __forceinline__ int split_rescale(int x, int form, bool clamp, const int* c, int stride)
{
    if (form == EF_FLOAT) {
        return clamp ? rescale<true, EF_FLOAT>(x, c[0], c[stride], c[2 * stride], c[3 * stride], c[4 * stride])
                     : rescale<false, EF_FLOAT>(x, 0, 0, c[2 * stride], c[3 * stride], c[4 * stride]);
    }
    if (form == EF_WIDE)
        return clamp ? rescale<true, EF_WIDE>(x, c[0], c[stride], c[2 * stride], c[3 * stride], c[4 * stride])
                     : rescale<false, EF_WIDE>(x, c[0], 0, c[2 * stride], c[3 * stride], c[4 * stride]);
    return clamp ? rescale<true, 0>(x, c[0], c[stride], c[2 * stride], c[3 * stride], c[4 * stride])
                 : rescale<false, 0>(x, 0, 0, c[2 * stride], c[3 * stride], c[4 * stride]);
}

__global__ void __launch_bounds__(SPLIT_THREADS, 1)
igemm_split_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const SplitArgs sa)
{
    const IgemmArgs& a = sa.g;
    constexpr int S = SPLIT, COLS = SPLIT_BN / S, PAIRS = COLS / 2, CHUNKS = COLS / 4;   // columns, column pairs and 16-byte chunks a CTA finishes
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int a_bytes = BM * a.BK, stage_bytes = a_bytes + SPLIT_BN * a.BK;
    unsigned char* sums = smem + (size_t)sa.per * stage_bytes;       // [S][128][COLS] int32, chunks of a row swizzled
    int* cst = (int*)(sums + BM * SPLIT_BN * 4);                     // [2][FAST_NP][COLS], stored column order
    unsigned long long* bars = (unsigned long long*)(cst + 2 * FAST_NP * SPLIT_BN);
    const unsigned full0 = smem_u32(bars), tfull = full0 + 8u * SPLIT_STAGES;
    unsigned* tmem_slot = (unsigned*)(bars + SPLIT_STAGES + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    pdl_launch_dependents();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // (waited for before the first remote store)

    const int tile = (int)blockIdx.x / S, rank = (int)blockIdx.x % S;   // clusters are S consecutive CTAs
    const int m_tile = tile / a.num_n_tiles, n_tile = tile - m_tile * a.num_n_tiles;
    const int m0 = a.m_base + m_tile * BM, n0 = n_tile * SPLIT_BN, part0 = rank * COLS;
    const int kchunks = (a.Cin + a.BK - 1) / a.BK, num_kb = a.taps * kchunks;
    const int kb0 = rank * sa.per, nkb = max(0, min(sa.per, num_kb - kb0));
    if (warp == 0) {
        if (lane <= SPLIT_STAGES) mbar_init(full0 + 8u * lane, 1);
        if (lane == 0) {
            *abort_flag = 0;
            prefetch_tensor_map(&tmA);
            prefetch_tensor_map(&tmB);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(64u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = threadIdx.x; i < (a.fq2 ? 2 : 1) * FAST_NP * COLS; i += SPLIT_THREADS) {
        const int set = i / (FAST_NP * COLS), j = i - set * FAST_NP * COLS, prm = j / COLS, c = j - prm * COLS;
        cst[(set * FAST_NP + prm) * COLS + c] = __ldg((set ? a.fq2 : a.fq) + (size_t)prm * a.cpad + n0 + perm_real_channel(part0 + c, sa.perm_ng));
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = *tmem_slot, tiles_s = smem_u32(smem);

    // epilogue threads: this thread's column pairs of the tile, u = pair index + PAIRS * row
    constexpr int UNITS = BM * PAIRS / (32 * SPLIT_EPI_WARPS);
    const int et = (int)threadIdx.x - 32 * EPI_WARP0;
    unsigned short res[UNITS];
    bool ok = true;
    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        PixelPos px;
        px.start(a, m0);
        const int iw0 = px.ox * a.sX - a.pL, ih0 = px.oy * a.sY - a.pT;
        const int tap0 = kb0 / kchunks, kc0 = kb0 - tap0 * kchunks;
        const int ky0 = tap0 / a.kW, kx0 = tap0 - ky0 * a.kW;
        if (a.late_weights) pdl_wait();
        if (elect_one()) {
            int kc = kc0, kcoord = tap0 * a.Cin + kc0 * a.BK;
            for (int i = 0; i < nkb; ++i) {
                mbar_expect_tx(full0 + 8u * i, (unsigned)stage_bytes);
                tma_load_2d(tiles_s + (unsigned)(i * stage_bytes + a_bytes), &tmB, full0 + 8u * i, kcoord, n0);
                if (++kc == kchunks) { kc = 0; kcoord += a.Cin - (kchunks - 1) * a.BK; }
                else kcoord += a.BK;
            }
        }
        __syncwarp();
        pdl_wait();   // weights are constants; the activations are the previous kernel's output
        if (elect_one()) {
            int kc = kc0, kx = kx0, ky = ky0, kcoord = tap0 * a.Cin + kc0 * a.BK;
            for (int i = 0; i < nkb; ++i) {
                const unsigned dst = tiles_s + (unsigned)(i * stage_bytes);
                if (a.a_im2col) tma_load_im2col_4d(dst, &tmA, full0 + 8u * i, kc * a.BK, iw0, ih0, px.n, (unsigned short)(kx * a.dX), (unsigned short)(ky * a.dY));
                else tma_load_2d(dst, &tmA, full0 + 8u * i, kcoord, m0);
                if (++kc == kchunks) {
                    kc = 0;
                    kcoord += a.Cin - (kchunks - 1) * a.BK;
                    if (++kx == a.kW) { kx = 0; ++ky; }
                } else {
                    kcoord += a.BK;
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const unsigned desc_hi = (unsigned)(make_smem_desc(0u, a.BK) >> 32);
        unsigned a_lo = (tiles_s & 0x3ffffu) >> 4;
        const unsigned stage16 = (unsigned)(stage_bytes >> 4), a16 = (unsigned)(a_bytes >> 4);
        for (int i = 0; i < nkb; ++i, a_lo += stage16) {
            if (!mbar_wait_issuer(full0 + 8u * i, 0, abort_flag, a.status, 3)) { ok = false; break; }
            tc_fence_after();
            if (elect_one()) {
                const unsigned b_lo = a_lo + a16;
                tc_mma_i8_lohi(tmem_base, a_lo, b_lo, desc_hi, a.idesc, i > 0 ? 1u : 0u);
                if (a.BK >= 64) tc_mma_i8_lohi(tmem_base, a_lo + 2u, b_lo + 2u, desc_hi, a.idesc, 1u);
                if (a.BK == 128) {
                    tc_mma_i8_lohi(tmem_base, a_lo + 4u, b_lo + 4u, desc_hi, a.idesc, 1u);
                    tc_mma_i8_lohi(tmem_base, a_lo + 6u, b_lo + 6u, desc_hi, a.idesc, 1u);
                }
                if (i + 1 == nkb) tc_commit(tfull);
            }
            __syncwarp();
        }
    } else {
        pdl_wait();   // the residual is an earlier kernel's output; the output may still be read by one
        if (a.r.ptr) {
#pragma unroll
            for (int k = 0; k < UNITS; ++k) {
                const int u = et + k * 32 * SPLIT_EPI_WARPS, row = u / PAIRS, p = u - row * PAIRS, m = m0 + row;
                const int ch = n0 + perm_real_channel(part0 + 2 * p, sa.perm_ng);
                res[k] = m < a.m_base + a.M && ch < a.N ? *(const unsigned short*)((const uint8_t*)a.r.ptr + (size_t)m * a.N + ch) : (unsigned short)0;
            }
        }
    }
    __syncwarp();
    // every CTA of the cluster runs: its shared memory may be written
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp >= EPI_WARP0) {
        const int quad = warp & 3, half = (warp - EPI_WARP0) >> 2, row = quad * 32 + lane;
        unsigned v[32];
        if (nkb > 0) {
            ok = mbar_wait_warp(tfull, 0, abort_flag, a.status, 4);
            tc_fence_after();
            if (ok) {
                tc_ld32(tmem_base + ((unsigned)(quad * 32) << 16) + 32u * half, v);
                tc_wait_ld_into(v);
            }
        }
        if (nkb == 0 || !ok) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0u;
        }
        const unsigned swz = (unsigned)(row / (8 / CHUNKS)) & (CHUNKS - 1);
        const unsigned mine = smem_u32(sums) + (unsigned)((rank * BM + row) * COLS * 4);
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const unsigned col = 32u * half + (unsigned)j, target = col / COLS, chunk = (col % COLS) / 4;
            unsigned addr;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(mine + ((chunk ^ swz) << 4)), "r"(target));
            asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[j]), "r"(v[j + 1]), "r"(v[j + 2]), "r"(v[j + 3]) : "memory");
        }
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp >= EPI_WARP0) {
#pragma unroll
        for (int k = 0; k < UNITS; ++k) {
            const int u = et + k * 32 * SPLIT_EPI_WARPS, row = u / PAIRS, p = u - row * PAIRS, m = m0 + row;
            const unsigned swz = (unsigned)(row / (8 / CHUNKS)) & (CHUNKS - 1);
            const unsigned char* at = sums + (size_t)row * COLS * 4 + ((((unsigned)p >> 1) ^ swz) << 4) + (p & 1) * 8;
            int x0 = 0, x1 = 0;
#pragma unroll
            for (int src = 0; src < S; ++src) {
                const int2 w = *(const int2*)(at + (size_t)src * BM * COLS * 4);
                x0 += w.x;
                x1 += w.y;
            }
            const int* c = cst + 2 * p;
            int y0 = split_rescale(x0, sa.form, sa.need_clamp != 0, c, COLS), y1 = split_rescale(x1, sa.form, sa.need_clamp != 0, c + 1, COLS);
            if (a.r.ptr) {
                const int* c2 = c + FAST_NP * COLS;
                const unsigned rw = res[k];
                if (sa.dp) {
                    unsigned a4;
                    if (sa.ef & EF_T_UNSIGNED) asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(a4) : "r"(y1), "r"(y0), "r"(rw));
                    else asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(a4) : "r"(y1), "r"(y0), "r"(rw));
                    // row 0 of the residual set holds the column-selecting multiplier words (see perm_block)
                    if (sa.ef & EF_DP_A_SIGNED) {
                        asm("dp4a.s32.u32 %0, %1, %2, %3;" : "=r"(y0) : "r"(a4), "r"(c2[0]), "r"(c2[3 * COLS]));
                        asm("dp4a.s32.u32 %0, %1, %2, %3;" : "=r"(y1) : "r"(a4), "r"(c2[1]), "r"(c2[3 * COLS + 1]));
                    } else {
                        asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(y0) : "r"(a4), "r"(c2[0]), "r"(c2[3 * COLS]));
                        asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(y1) : "r"(a4), "r"(c2[1]), "r"(c2[3 * COLS + 1]));
                    }
                    y0 >>= c2[4 * COLS];
                    y1 >>= c2[4 * COLS + 1];
                } else {
                    const bool ru = (sa.ef & EF_RES_UNSIGNED) != 0;
                    const int form2 = sa.form == EF_WIDE ? 0 : sa.form;   // the second stage of a wide cell is the 32-bit one
                    y0 = split_rescale(min(max(y0, a.t_lo), a.t_hi) + byte_extend(rw, 0, ru), form2, sa.need_clamp != 0, c2, COLS);
                    y1 = split_rescale(min(max(y1, a.t_lo), a.t_hi) + byte_extend(rw, 1, ru), form2, sa.need_clamp != 0, c2 + 1, COLS);
                }
            }
            const unsigned w = pack4_sat(y0, y1, 0, 0, a.out_unsigned != 0);
            const int ch = n0 + perm_real_channel(part0 + 2 * p, sa.perm_ng);
            if (m < a.m_base + a.M && ch < a.N) *(unsigned short*)((uint8_t*)a.out + (size_t)m * a.N + ch) = (unsigned short)w;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(64u) : "memory");
    }
}

// Whether the CTAs of a cluster share a tile: from 24 K blocks on and up to half the chip.  Measured with one image: at 36 blocks a
// layer goes from 16.4 us to 12.3; at 16 and 18 it gains nothing and takes the idle SMs that the next kernel's prologue would run on
// (ResNet-50 274 us with 36-block layers split, 286 with all from 12 on, 289 with none), as do 128 CTAs at four images.
static bool igemm_split(long long tiles, int num_kb, int num_sms)
{
    return num_kb >= 24 && num_kb <= SPLIT * SPLIT_STAGES && tiles * SPLIT <= num_sms / 2;
}

// Eight weights per thread; at most a few megabytes that stay in L2.  All cells of a pass in one launch: with one launch each a ResNet-18 of packed weights
// spent twenty hand-overs on them.
static constexpr int WIDEN_JOBS = 32;
struct WidenTable {
    WidenJob job[WIDEN_JOBS];
    unsigned first[WIDEN_JOBS + 1];   // destination words before each job
    int count;
};

__global__ void __launch_bounds__(256) widen_int4_kernel(const __grid_constant__ WidenTable t)
{
    pdl_launch_dependents();
    pdl_wait();   // the destination may still be read by the previous kernel
    int j = 0;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < t.first[t.count]; i += gridDim.x * blockDim.x) {
        while (i >= t.first[j + 1]) ++j;   // (i only grows)
        const WidenJob& job = t.job[j];
        const unsigned at = i - t.first[j], n = at / job.words, w = at - n * job.words;
        const int real = perm_real_channel((int)n, job.ng_dst);
        uint2 o = make_uint2(0u, 0u);
        if (real < job.rows_src) {
            int src = real;
            if (job.ng_src) {   // where the packed rows hold this channel (the inverse of perm_real_channel)
                const int k = real % (8 * job.ng_src), q = k / (2 * job.ng_src), r = k - q * 2 * job.ng_src;
                src = real - k + 8 * (r >> 1) + 2 * q + (r & 1);
            }
            unsigned lo, hi;
            expand_int4_x16(__ldg((const unsigned*)job.packed + (size_t)src * job.words + w), lo, hi);
            auto down = [](unsigned x) {   // 16 x the value in every byte -> the value
                const unsigned t = (x >> 4) & 0x0f0f0f0fu;
                return t | ((t & 0x08080808u) * 0x1eu);
            };
            o = make_uint2(down(lo), down(hi));
        }
        ((uint2*)job.dst)[at] = o;
    }
}

cudaError_t launch_widen_int4(const WidenJob* jobs, int count, cudaStream_t s)
{
    for (int done = 0; done < count;) {
        WidenTable t;
        memset(&t, 0, sizeof(t));
        unsigned long long total = 0;
        for (; done < count && t.count < WIDEN_JOBS; ++done) {
            const unsigned long long words = (unsigned long long)jobs[done].rows * jobs[done].words;
            if (words >= (1ull << 31)) return cudaErrorInvalidValue;
            if (words == 0) continue;
            if (total + words >= (1ull << 31)) break;
            t.job[t.count] = jobs[done];
            t.first[t.count++] = (unsigned)total;
            total += words;
            t.first[t.count] = (unsigned)total;
        }
        if (t.count == 0) break;
        const unsigned long long blocks = (total + 255) / 256, most = 8ull * current_sms();
        if (cudaError_t e = launch_pdl(widen_int4_kernel, (int)(blocks < most ? blocks : most), 256, 0, s, t)) return e;
    }
    return cudaSuccess;
}

bool igemm_uses_fast_epilogue(const IgemmPlan& plan, const FastQuant& fast, bool has_residual, int out_dtype)
{
    return fast.enabled && out_dtype == DT_I8 && (plan.N % 32 == 0) && (!has_residual || fast.fq2) && plan.has_out_maps;
}

int igemm_perm_block(const IgemmPlan& plan) { return plan.BN / plan.parts >= 32 ? 32 : 16; }

void igemm_permute_weights(const int8_t* w, int8_t* dst, int N, size_t row_bytes, int perm_block)
{
    const int ng = perm_block / 8;
    for (int n = 0; n < N; ++n) memcpy(dst + (size_t)n * row_bytes, w + (size_t)perm_real_channel(n, ng) * row_bytes, row_bytes);
}

// Tiles of a launch, and its CTAs: a multiple of the number of column blocks keeps every CTA on one, whose constants are staged once
static void igemm_grid(const IgemmPlan& plan, int* tiles, int* grid)
{
    const int num_n_tiles = (plan.N + plan.BN - 1) / plan.BN;
    *tiles = (plan.M + BM - 1) / BM * num_n_tiles;
    *grid = std::min(plan.grid, *tiles);
    if (*tiles > *grid && num_n_tiles > 1 && *grid > num_n_tiles) *grid -= *grid % num_n_tiles;
}

// A launch of up to two tiles per CTA has the variant that stores from the registers (see DRY)
static bool igemm_short(int tiles, int grid) { return tiles <= 2 * grid; }

// (of a cell with the 32-bit epilogue)
bool igemm_takes_clusters(const IgemmPlan& plan)
{
    int tiles, grid;
    igemm_grid(plan, &tiles, &grid);
    return !plan.w4 && !plan.grouped && plan.BN == SPLIT_BN && igemm_split(tiles, plan.taps * ((plan.Cin + plan.BK - 1) / plan.BK), plan.num_sms);
}

bool igemm_writes_rows(const IgemmPlan& plan, int columns)
{
    int tiles, grid;
    igemm_grid(plan, &tiles, &grid);
    return plan.perm && !plan.w4 && !plan.grouped && !plan.pair && plan.BN / plan.parts >= 32 && columns % 8 == 0 && igemm_short(tiles, grid)
        && !igemm_takes_clusters(plan);
}

cudaError_t launch_igemm(const IgemmPlan& plan, const QuantDev& q, const Residual& r, const FastQuant& fast, void* out,
                         int out_dtype, int m_base, int* status_word, cudaStream_t s, void* rows, int columns)
{
    if (plan.M == 0 || plan.N == 0) return cudaSuccess;
    if (rows && (r.ptr || !igemm_writes_rows(plan, columns))) return cudaErrorInvalidConfiguration;
    IgemmArgs a;
    memset(&a, 0, sizeof(a));
    a.m_base = m_base;
    a.M = plan.M; a.N = plan.N; a.Cin = plan.Cin; a.taps = plan.taps; a.BK = plan.BK; a.BN = plan.BN;
    a.b_resident = plan.b_resident;
    a.late_weights = plan.late_weights;
    // As many producers as keep up (about 550 cycles a fill each) with a tile's epilogue, about 8 cycles per column: idle ones wait at the
    // CTA's last barrier and poll nothing
    a.takers = (plan.taps * ((plan.Cin + plan.BK - 1) / plan.BK) * 550 + plan.BN * 8 - 1) / (plan.BN * 8);
    a.takers = std::min(a.takers, std::min(plan.stages, NUM_PRODUCERS));
    a.stages = plan.stages; a.a_im2col = plan.a_im2col;
    a.grouped = plan.grouped;
    a.res_slots = plan.res_slots ? plan.res_slots : 2;
    a.oW = plan.oW; a.oH = plan.oH; a.kW = plan.kW; a.sX = plan.sX; a.sY = plan.sY;
    a.pL = plan.pL; a.pT = plan.pT; a.dX = plan.dX; a.dY = plan.dY;
    a.num_m_tiles = (plan.M + BM - 1) / BM;
    a.num_n_tiles = (plan.N + plan.BN - 1) / plan.BN;
    // instruction descriptor: D = s32, A = u8/s8, B = s8, both K-major, N and M extents
    a.idesc = (2u << 4) | ((plan.a_unsigned ? 0u : 1u) << 7) | (1u << 10) | ((unsigned)(plan.BN >> 3) << 17)
            | ((unsigned)(BM >> 4) << 24);
    a.parts = plan.parts;
    a.groups = 4 / plan.parts;
    a.out_dtype = out_dtype;
    a.out = out;
    a.ldo = plan.N;
    a.status = status_word;
    a.q = q;
    a.r = r;
    a.fq = fast.fq; a.fq2 = fast.fq2; a.cpad = fast.cpad; a.t_lo = fast.t_lo; a.t_hi = fast.t_hi;
    a.out_unsigned = fast.out_unsigned;
    a.dp_a_signed = fast.dp_a_signed;
    const bool t_unsigned = fast.dp4a ? fast.dp_t_unsigned : (fast.t_lo == 0);
    a.ef = (fast.out_unsigned ? EF_OUT_UNSIGNED : 0) | (r.is_unsigned ? EF_RES_UNSIGNED : 0)
         | (t_unsigned ? EF_T_UNSIGNED : 0) | (fast.dp_a_signed ? EF_DP_A_SIGNED : 0) | fast.form;
    const bool use_fast = igemm_uses_fast_epilogue(plan, fast, r.ptr != nullptr, out_dtype);
    // the weights of a cell on the 32-bit epilogue are stored permuted (and only those)
    if (use_fast != (plan.perm != 0)) return cudaErrorInvalidConfiguration;
    // two accumulators per group of epilogue warps (two in all for the exact epilogue)
    a.acc_shift = use_fast ? (plan.parts == 4 ? 1 : (plan.parts == 2 ? 2 : 3)) : 1;
    a.tmem_cols = (unsigned)plan.BN << a.acc_shift;
    const int mode = !use_fast ? 0 : (r.ptr ? (fast.need_clamp ? 2 : (fast.dp4a ? 5 : 4)) : (fast.need_clamp ? 1 : 3));
    static const IgemmKernel kernels[2][6] = {
        {igemm_i8_tcgen05_kernel<0, false, false>, igemm_i8_tcgen05_kernel<1, false, false>, igemm_i8_tcgen05_kernel<2, false, false>,
         igemm_i8_tcgen05_kernel<3, false, false>, igemm_i8_tcgen05_kernel<4, false, false>, igemm_i8_tcgen05_kernel<5, false, false>},
        {igemm_i8_tcgen05_kernel<0, false, false>, igemm_i8_tcgen05_kernel<1, false, true>, igemm_i8_tcgen05_kernel<2, false, true>,
         igemm_i8_tcgen05_kernel<3, false, true>, igemm_i8_tcgen05_kernel<4, false, true>, igemm_i8_tcgen05_kernel<5, false, true>}};
    static SmemLimitSet limits[3][6];
    int tiles, grid;
    igemm_grid(plan, &tiles, &grid);
    // Few tiles, long K: a cluster of CTAs per tile
    const int num_kb = plan.taps * ((plan.Cin + plan.BK - 1) / plan.BK);
    if (use_fast && igemm_takes_clusters(plan)) {
        static SmemLimitSet split_limit;
        if (cudaError_t e = raise_smem_limit(igemm_split_tcgen05_kernel, split_limit)) return e;
        SplitArgs sa;
        sa.g = a;
        sa.per = (num_kb + SPLIT - 1) / SPLIT;
        sa.perm_ng = plan.perm / 8;
        sa.form = fast.form;
        sa.need_clamp = fast.need_clamp ? 1 : 0;
        sa.dp = r.ptr && fast.dp4a && !fast.need_clamp ? 1 : 0;
        sa.ef = a.ef;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(tiles * SPLIT));
        cfg.blockDim = dim3(SPLIT_THREADS);
        cfg.dynamicSmemBytes = split_smem_bytes(sa.per, plan.BK);
        cfg.stream = s;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = SPLIT;
        attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        return cudaLaunchKernelEx(&cfg, igemm_split_tcgen05_kernel, plan.tmA, plan.tmB, sa);
    }
    // resident weights rely on a column block that does not change (or on one tile per CTA)
    if (a.b_resident && tiles > grid && a.num_n_tiles > 1 && grid % a.num_n_tiles != 0) return cudaErrorInvalidConfiguration;
    auto pixels = [&](long long m) {
        PixelStep d;
        d.x = (int)(m % a.oW);
        d.y = (int)(m / a.oW % a.oH);
        d.n = (int)(m / a.oW / a.oH);
        return d;
    };
    a.step_m = grid / a.num_n_tiles;
    a.step_n = grid % a.num_n_tiles;
    a.adv_tiles = pixels((long long)a.step_m * BM);
    a.adv_one = pixels(BM);
    if (plan.pair && use_fast && !r.ptr) {
        typedef void (*PairKernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const IgemmArgs);
        static const PairKernel pair_kernels[2] = {igemm_pair_i8_tcgen05_kernel<false>, igemm_pair_i8_tcgen05_kernel<true>};
        static SmemLimitSet pair_limits[2];
        const int pair_tiles = ((a.num_m_tiles + 1) / 2) * a.num_n_tiles;
        int pgrid = plan.grid < pair_tiles ? plan.grid : pair_tiles;
        if (pair_tiles > pgrid && a.num_n_tiles > 1 && pgrid > a.num_n_tiles) pgrid -= pgrid % a.num_n_tiles;
        if (pair_tiles <= pgrid || a.num_n_tiles == 1 || pgrid % a.num_n_tiles == 0) {
            a.step_m = pgrid / a.num_n_tiles;
            a.step_n = pgrid % a.num_n_tiles;
            a.adv_tiles = pixels(2ll * a.step_m * BM);
            const int v = fast.need_clamp ? 1 : 0;
            if (cudaError_t e = raise_smem_limit(pair_kernels[v], pair_limits[v])) return e;
            return launch_pdl(pair_kernels[v], pgrid, NUM_THREADS, plan.pair_smem_bytes, s, plan.tmA,
                              plan.tmB, plan.tmO32, a);
        }
    }
    const int table = plan.w4 ? 2 : (igemm_short(tiles, grid) ? 1 : 0);
    if (rows) {
        a.N = a.ldo = columns;
        a.out = rows;
    }
    const IgemmKernel kernel = plan.w4 ? igemm_w4_kernels[mode] : kernels[table][mode];
    if (cudaError_t e = raise_smem_limit(kernel, limits[table][mode])) return e;
    return launch_pdl(kernel, grid, NUM_THREADS + (plan.w4 ? 32 * W4_UNPACK_WARPS : 0), plan.smem_bytes, s,
                      plan.tmA, plan.tmB, plan.tmO, plan.tmR, a);
}

}  // namespace n2d2b
