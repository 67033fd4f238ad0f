// A 1x1 expansion with its residual sum and the 1x1 layer behind it as one kernel (the seam between two units of a residual network's first stage).
//
//   y   = rescale_sum(rescale(A * B1^T) + residual)     256 channels, stored: the next sum and others read it
//   out = rescale(y * B2^T)                             up to 128 channels
//
// The implicit-GEMM kernel (igemm_kernel.cuh) with both column blocks of a 128-row tile in one CTA.  The bytes of y that its epilogue warps leave in the
// staging regions, rows of 64 swizzled for the store, are the operand of the second multiplication as they stand: four K blocks of 64.  By itself the second
// layer read y from HBM again (ResNet-50 at 1024 images 793 MB) and added a hand-over between kernels.
//
// Warp 0 loads, warp 1 issues, two groups of eight warps drain a column block of 128 each, and of the second multiplication a block of 32 columns per warp
// quadruple, one tile behind.  A region is free again when the second accumulator of its tile has been seen complete (its operands have been read) and
// its store has finished reading; residual loads therefore run two tiles ahead in four regions.
//
// What bounds it: the epilogue's issue slots and shared-memory wavefronts, as in the residual cells of the implicit GEMM.
#pragma once
#include "igemm_kernel.cuh"

namespace n2d2b {

static constexpr int CH_N = 256;                 // channels of y
static constexpr int CH_STAGES = 4;              // activation tiles
static constexpr int CH_SLOTS_MAX = 4;
static constexpr int CH_SLOT_BYTES = 128 * CH_N; // a tile of y
static constexpr int CH_THREADS = 32 * (EPI_WARP0 + NUM_EPI_WARPS);
// full[stages], empty[stages], t1full[2], t1empty[2], yfull[slots], t2full[2], t2empty[2], weights, constants, residual[slots * epilogue warps]
static constexpr int CH_BARS = 2 * CH_STAGES + 4 + CH_SLOTS_MAX + 4 + 2 + CH_SLOTS_MAX * NUM_EPI_WARPS;

struct ChainArgs {
    int M, m_base, C, N2, slots;
    unsigned idesc1, idesc2;
    const int *fq, *fq2, *fq_next;   // the expansion's rescale, the sum's, the next layer's
    int cpad, cpad_next;
    int ef, t_lo, t_hi;
    int ef_next, clamp_next;
    uint8_t* out;
    int* status;
};

// The forms of the rescale that a kernel knows.  Loading a kernel loads the module it is in, so each set is a module of its own
// (igemm_chain.cu, igemm_chain_float.cu, igemm_chain_any.cu) and a network loads the forms it has.
static constexpr int CHAIN_INT = 0, CHAIN_FLOAT = 1, CHAIN_ANY = 2;

template <bool CLAMP, int FORM>
__device__ __forceinline__ void chain_drain_sum_form(const EpiTile& e, unsigned tbase, int cbase, unsigned region_off, const unsigned* rb, int lane, int ef)
{
    switch (ef & (EF_OUT_UNSIGNED | EF_RES_UNSIGNED)) {
    case 0: epi_drain<true, CLAMP, false, FORM | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
    case EF_OUT_UNSIGNED: epi_drain<true, CLAMP, false, FORM | EF_OUT_UNSIGNED | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
    case EF_RES_UNSIGNED: epi_drain<true, CLAMP, false, FORM | EF_RES_UNSIGNED | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
    default: epi_drain<true, CLAMP, false, FORM | EF_OUT_UNSIGNED | EF_RES_UNSIGNED | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
    }
}

template <int MODE, int FORMS>
__device__ __forceinline__ void chain_drain_sum(const EpiTile& e, unsigned tbase, int cbase, unsigned region_off, const unsigned* rb, int lane, int ef)
{
    constexpr bool CLAMP = MODE == 2, DP = MODE == 5;
    if (DP) {
        switch (ef & (EF_OUT_UNSIGNED | EF_T_UNSIGNED | EF_DP_A_SIGNED)) {
        case 0: epi_drain<true, CLAMP, DP, 0 | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
        case 1: epi_drain<true, CLAMP, DP, 1 | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
        case 4: epi_drain<true, CLAMP, DP, 4 | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
        case 5: epi_drain<true, CLAMP, DP, 5 | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
        case 8: epi_drain<true, CLAMP, DP, 8 | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
        case 9: epi_drain<true, CLAMP, DP, 9 | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
        case 12: epi_drain<true, CLAMP, DP, 12 | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
        default: epi_drain<true, CLAMP, DP, 13 | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
        }
        return;
    }
    const int form = FORMS == CHAIN_INT ? 0 : (FORMS == CHAIN_FLOAT ? EF_FLOAT : ef & (EF_WIDE | EF_FLOAT));
    if (FORMS != CHAIN_INT && form == EF_FLOAT) chain_drain_sum_form<CLAMP, EF_FLOAT>(e, tbase, cbase, region_off, rb, lane, ef);
    else if (FORMS == CHAIN_ANY && form == EF_WIDE) chain_drain_sum_form<CLAMP, EF_WIDE>(e, tbase, cbase, region_off, rb, lane, ef);
    else if (FORMS != CHAIN_FLOAT) chain_drain_sum_form<CLAMP, 0>(e, tbase, cbase, region_off, rb, lane, ef);
}

template <bool CLAMP, int FORM>
__device__ __forceinline__ void chain_drain_next_form(const unsigned* va, const unsigned* vb, unsigned par_off, int col, uint8_t* out, const unsigned (&rowoff)[4], unsigned rowok, int lane, int ef)
{
    if (ef & EF_OUT_UNSIGNED) perm_block_global<CLAMP, FORM | EF_OUT_UNSIGNED>(va, vb, par_off, col, out, rowoff, rowok, lane);
    else perm_block_global<CLAMP, FORM>(va, vb, par_off, col, out, rowoff, rowok, lane);
}

template <bool CLAMP, int FORMS>
__device__ __forceinline__ void chain_drain_next(const unsigned* va, const unsigned* vb, unsigned par_off, int col, uint8_t* out, const unsigned (&rowoff)[4], unsigned rowok, int lane, int ef)
{
    const int form = FORMS == CHAIN_INT ? 0 : (FORMS == CHAIN_FLOAT ? EF_FLOAT : ef & (EF_WIDE | EF_FLOAT));
    if (FORMS != CHAIN_INT && form == EF_FLOAT) chain_drain_next_form<CLAMP, EF_FLOAT>(va, vb, par_off, col, out, rowoff, rowok, lane, ef);
    else if (FORMS == CHAIN_ANY && form == EF_WIDE) chain_drain_next_form<CLAMP, EF_WIDE>(va, vb, par_off, col, out, rowoff, rowok, lane, ef);
    else if (FORMS != CHAIN_FLOAT) chain_drain_next_form<CLAMP, 0>(va, vb, par_off, col, out, rowoff, rowok, lane, ef);
}

template <int MODE, int FORMS>
__global__ void __launch_bounds__(CH_THREADS, 1)
igemm_chain_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ CUtensorMap tmB2,
                           const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmR, const ChainArgs a)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int a_bytes = BM * a.C, b1_bytes = CH_N * a.C, b2_block = a.N2 * 64;
    unsigned char* const regions = smem;                                        // [slots][4 column blocks of 64][4 quadrants][32 rows][64]
    unsigned char* const tiles = regions + a.slots * CH_SLOT_BYTES;
    unsigned char* const b1 = tiles + CH_STAGES * a_bytes;
    unsigned char* const b2 = b1 + b1_bytes;                                    // [4][N2][64]
    int* const par = (int*)(b2 + 4 * b2_block);                                 // [expansion, sum, next][FAST_NP][256]
    unsigned long long* const bars = (unsigned long long*)(par + 3 * FAST_NP * 256);
    const unsigned full0 = smem_u32(bars), empty0 = full0 + 8u * CH_STAGES, t1full0 = empty0 + 8u * CH_STAGES, t1empty0 = t1full0 + 16u;
    const unsigned yfull0 = t1empty0 + 16u, t2full0 = yfull0 + 8u * CH_SLOTS_MAX, t2empty0 = t2full0 + 16u, bfull = t2empty0 + 16u, cready = bfull + 8u;
    const unsigned rbar0 = cready + 8u;
    unsigned* const tmem_slot = (unsigned*)(bars + CH_BARS);
    volatile int* const abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    pdl_launch_dependents();

    if (warp == 0) {
        for (int i = lane; i < CH_BARS; i += 32) {
            const int j = i - 2 * CH_STAGES;
            unsigned n = 1;
            if (j >= 2 && j < 4) n = NUM_EPI_WARPS / 2;                                                  // t1empty
            else if (j >= 4 && j < 4 + CH_SLOTS_MAX) n = NUM_EPI_WARPS;                                  // yfull
            else if (j >= 6 + CH_SLOTS_MAX && j < 8 + CH_SLOTS_MAX) n = NUM_EPI_WARPS;                   // t2empty
            else if (j == 9 + CH_SLOTS_MAX) n = NUM_EPI_WARPS;                                           // constants
            mbar_init(full0 + 8u * i, n);
        }
        if (lane == 0) {
            *abort_flag = 0;
            prefetch_tensor_map(&tmA);
            prefetch_tensor_map(&tmB1);
            prefetch_tensor_map(&tmB2);
            prefetch_tensor_map(&tmO);
            prefetch_tensor_map(&tmR);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = *tmem_slot, tmem_next = tmem_base + 256u;   // accumulators: two column blocks of y, then two of the next layer
    const int num_tiles = (a.M + BM - 1) / BM, m_end = a.m_base + a.M;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if ((int)blockIdx.x < num_tiles) {
            if (elect_one()) {
                mbar_expect_tx(bfull, (unsigned)(b1_bytes + 4 * b2_block));
                for (int n = 0; n < 2; ++n) tma_load_2d(smem_u32(b1) + (unsigned)(n * 128 * a.C), &tmB1, bfull, 0, 128 * n);
                for (int k = 0; k < 4; ++k) tma_load_2d(smem_u32(b2) + (unsigned)(k * b2_block), &tmB2, bfull, 64 * k, 0);
            }
            __syncwarp();
        }
        pdl_wait();
        int s = 0;
        unsigned ph = 1u;
        for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
            if (!mbar_wait_issuer(empty0 + 8u * s, ph, abort_flag, a.status, 61)) break;
            if (elect_one()) {
                mbar_expect_tx(full0 + 8u * s, (unsigned)a_bytes);
                tma_load_2d(smem_u32(tiles) + (unsigned)(s * a_bytes), &tmA, full0 + 8u * s, 0, a.m_base + tile * BM);
            }
            __syncwarp();
            if (++s == CH_STAGES) { s = 0; ph ^= 1u; }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        bool ok = true;
        if ((int)blockIdx.x < num_tiles) ok = mbar_wait_issuer(bfull, 0, abort_flag, a.status, 62);
        const unsigned desc1 = (unsigned)(make_smem_desc(0u, a.C) >> 32), desc2 = (unsigned)(make_smem_desc(0u, 64) >> 32);
        const unsigned a_lo0 = (smem_u32(tiles) & 0x3ffffu) >> 4, b1_lo = (smem_u32(b1) & 0x3ffffu) >> 4, b2_lo = (smem_u32(b2) & 0x3ffffu) >> 4;
        const unsigned y_lo0 = (smem_u32(regions) & 0x3ffffu) >> 4;
        const int ksteps = a.C / 32;
        int s = 0, ys = 0;
        unsigned ph = 0, yph = 0, it = 0;
        // the second multiplication of tile `t`: its bytes are in region ys
        auto next_layer = [&](unsigned t) -> bool {
            if (!mbar_wait_issuer(yfull0 + 8u * ys, yph, abort_flag, a.status, 63)) return false;
            if (!mbar_wait_issuer(t2empty0 + 8u * (t & 1u), ((t >> 1) & 1u) ^ 1u, abort_flag, a.status, 64)) return false;
            tc_fence_after();
            if (elect_one()) {
                const unsigned d2 = tmem_next + (t & 1u) * 128u;
                unsigned y = y_lo0 + (unsigned)(ys * (CH_SLOT_BYTES >> 4)), b = b2_lo;
                for (int k = 0; k < 4; ++k, y += (BM * 64) >> 4, b += (unsigned)(b2_block >> 4)) {
                    tc_mma_i8_lohi(d2, y, b, desc2, a.idesc2, k ? 1u : 0u);
                    tc_mma_i8_lohi(d2, y + 2u, b + 2u, desc2, a.idesc2, 1u);
                }
                tc_commit(t2full0 + 8u * (t & 1u));
            }
            __syncwarp();
            if (++ys == a.slots) { ys = 0; yph ^= 1u; }
            return true;
        };
        for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++it) {
            if (!mbar_wait_issuer(full0 + 8u * s, ph, abort_flag, a.status, 65)) { ok = false; break; }
            for (int n = 0; n < 2; ++n) {
                if (!mbar_wait_issuer(t1empty0 + 8u * n, (it & 1u) ^ 1u, abort_flag, a.status, 66)) { ok = false; break; }
                tc_fence_after();
                if (elect_one()) {
                    const unsigned al = a_lo0 + (unsigned)(s * (a_bytes >> 4)), bl = b1_lo + (unsigned)(n * ((128 * a.C) >> 4));
                    for (int k = 0; k < ksteps; ++k) tc_mma_i8_lohi(tmem_base + 128u * n, al + 2u * k, bl + 2u * k, desc1, a.idesc1, k ? 1u : 0u);
                    tc_commit(t1full0 + 8u * n);
                    if (n) tc_commit(empty0 + 8u * s);
                }
                __syncwarp();
            }
            if (!ok) break;
            if (++s == CH_STAGES) { s = 0; ph ^= 1u; }
            if (it > 0) ok = next_layer(it - 1);
        }
        if (ok && it > 0) next_layer(it - 1);
    } else {
        // ------------------------------------------------------------------ epilogue warps
        const int quad = warp & 3, part4 = (warp - EPI_WARP0) >> 2, n = part4 >> 1, cbase = (part4 & 1) * 64;   // columns 64 part4 .. of y
        bool ok = true;
        for (int i = (warp - EPI_WARP0) * 32 + lane; i < 3 * FAST_NP * 256; i += 32 * NUM_EPI_WARPS) {
            const int set = i / (FAST_NP * 256), prm = (i >> 8) - set * FAST_NP, c = i & 255;
            if (set < 2) par[i] = __ldg((set ? a.fq2 : a.fq) + (size_t)prm * a.cpad + c);
            else par[i] = __ldg(a.fq_next + (size_t)prm * a.cpad_next + c);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(cready);
        ok = mbar_wait_warp(cready, 0, abort_flag, a.status, 67);
        pdl_wait();   // residual loads and output stores touch tensors the previous kernel reads or writes
        unsigned rb[4], rowoff[4];
        perm_rowbase(rb, 64, lane, 4);
#pragma unroll
        for (int k = 0; k < 4; ++k) rowoff[k] = (unsigned)((lane >> 2) + 8 * k) * (unsigned)a.N2;
        EpiTile e;
        e.BN = 128; e.N = CH_N; e.M = m_end; e.wp = 64;
        // constants by column of y: a block of 128 columns is drained as columns cbase.. of its accumulator
        e.par_off = (unsigned)((unsigned char*)par - smem_raw) + (unsigned)(n * 128 * 4);
        e.t_lo = a.t_lo; e.t_hi = a.t_hi;
        const unsigned next_off = (unsigned)((unsigned char*)par - smem_raw) + 2u * FAST_NP * 1024u;
        const unsigned my_region = (unsigned)(regions - smem_raw) + (unsigned)(part4 * (BM * 64) + quad * REGION_BYTES);
        const unsigned my_rbar = rbar0 + 8u * CH_SLOTS_MAX * (unsigned)(warp - EPI_WARP0);
        const bool has_next = 32 * part4 < a.N2;
        const unsigned tq = (unsigned)(quad * 32) << 16;
        // residual loads: tile pf goes into region pf mod slots, slots - 2 tiles ahead
        int pf_tile = blockIdx.x, pf_slot = 0;
        unsigned pf = 0;
        auto next_tile = [&](unsigned t, int tile) -> bool {   // the next layer's block of 32 columns of tile `tile`, the CTA's t-th
            if (!mbar_wait_warp(t2full0 + 8u * (t & 1u), (t >> 1) & 1u, abort_flag, a.status, 68)) return false;
            tc_fence_after();
            const int gy = a.m_base + tile * BM + quad * 32;
            if (has_next && gy < m_end) {
                unsigned rowok = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (gy + (lane >> 2) + 8 * k < m_end) rowok |= 1u << k;
                unsigned va[16], vb[16];
                tc_ld_2x16x256b_x4_wait(tmem_next + (t & 1u) * 128u + tq + 32u * part4, va, vb);
                uint8_t* const out = a.out + (size_t)gy * a.N2 + 32 * part4;
                if (a.clamp_next) chain_drain_next<true, FORMS>(va, vb, next_off, 32 * part4, out, rowoff, rowok, lane, a.ef_next);
                else chain_drain_next<false, FORMS>(va, vb, next_off, 32 * part4, out, rowoff, rowok, lane, a.ef_next);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(t2empty0 + 8u * (t & 1u));
            return true;
        };
        unsigned it = 0, rph = 0;
        int slot = 0, last = -1;
        for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++it) {
            const int gx = 64 * part4, gy = a.m_base + tile * BM + quad * 32;
            const bool active = gy < m_end;
            if (lane == 0) {
                // the region of the tile two back: its next layer has been drained (last step), its store is not the latest
                bulk_wait_read_1();
                while (pf < it + (unsigned)(a.slots - 1) && pf_tile < num_tiles) {
                    epi_issue_residual(&tmR, my_region, CH_SLOT_BYTES, my_rbar, (unsigned)pf_slot, gx, a.m_base + pf_tile * BM + quad * 32, CH_N, m_end, 64);
                    ++pf;
                    pf_tile += gridDim.x;
                    if (++pf_slot == a.slots) pf_slot = 0;
                }
            }
            __syncwarp();
            const unsigned region_off = my_region + (unsigned)(slot * CH_SLOT_BYTES);
            if (!mbar_wait_warp(t1full0 + 8u * n, it & 1u, abort_flag, a.status, 69)) { ok = false; break; }
            if (!mbar_wait_warp(my_rbar + 8u * slot, rph, abort_flag, a.status, 70)) { ok = false; break; }
            tc_fence_after();
            if (active) chain_drain_sum<MODE, FORMS>(e, tmem_base + 128u * n + tq + (unsigned)cbase, cbase, region_off, rb, lane, a.ef);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(t1empty0 + 8u * n);
            fence_async_smem();   // the bytes are read by the store and by the tensor core through the async proxy
            __syncwarp();
            if (lane == 0) {
                if (active) tma_store_2d(&tmO, smem_u32(dyn_smem() + region_off), gx, gy);
                bulk_commit();
                mbar_arrive(yfull0 + 8u * slot);
            }
            if (++slot == a.slots) { slot = 0; rph ^= 1u; }
            if (it > 0 && !next_tile(it - 1, last)) { ok = false; break; }
            last = tile;
        }
        if (ok && it > 0) next_tile(it - 1, last);
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

// By the expansion's epilogue: with clamps, without, dot-product sum
typedef void (*ChainKernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const ChainArgs);
extern const ChainKernel chain_float[3], chain_any[3];

}  // namespace n2d2b
