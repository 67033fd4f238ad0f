// Two convolutions and the sum of their outputs as one kernel: the branch and the projection of a residual block's first unit.
//
//   t = rescale_a(A_a * B_a^T)          the branch (any filter), kept in shared memory as bytes
//   y = rescale_sum(rescale_b(A_b * B_b^T) + t)     the 1x1 projection and the sum
//
// The implicit-GEMM kernel (igemm_kernel.cuh) with two multiplications per output tile: the producers bring the K blocks of the branch and then
// those of the projection through the same ring, the issuer gives each its own accumulator, and an epilogue warp requantises the first
// one into its staging region, exactly where the residual operand of the second one would otherwise arrive from HBM.  The branch's output is
// never stored: by themselves the two layers write and read it once (ResNet-50's first block at 1024 images 793 MB each way) and hand
// over between two kernels.
//
// Roles, waits and the launch are those of the implicit-GEMM kernel.  What bounds it: the epilogue's issue slots (both rescales and
// the sum per output value) on layers of few channels, the operand loads on deep ones (three ring slots beside tiles of 256 columns).
#pragma once
#include "igemm_kernel.cuh"

namespace n2d2b {

struct DualSegment {
    int BK, kchunks, num_kb, tail;   // bytes of a K block, blocks per tap, in all; step of the weight coordinate behind a tap's last block
    int im2col, kW, sX, sY, pL, pT, dX, dY;
    int a_bytes, b_bytes, tx;        // of a ring slot: activations, weights, what TMA brings
    unsigned idesc;
    int b_first;                     // resident weights: byte offset of the segment's blocks
};

struct DualArgs {
    IgemmArgs g;                     // the projection: extents, tiling, its rescale and the sum's (no residual operand)
    DualSegment seg[2];
    int slot_bytes;
    const int* fq_a;                 // the branch's rescale
    int cpad_a, ef_a, clamp_a;
};

static constexpr int DUAL_REGIONS = 2;   // staging regions per epilogue warp: the store of one tile reads the one while the next fills the other
static constexpr int DUAL_SETS = 3;      // constants: branch, projection, sum

// The forms of the rescale that a kernel knows.  Loading a kernel loads the module it is in, so each set is a module of its own
// (igemm_dual.cu, igemm_dual_float.cu, igemm_dual_any.cu) and a network loads the forms it has.
static constexpr int DUAL_INT = 0, DUAL_FLOAT = 1, DUAL_ANY = 2;

template <bool CLAMP, int FORM>
__device__ __forceinline__ void dual_drain_branch_form(const EpiTile& e, unsigned tbase, int cbase, unsigned region_off, const unsigned* rb, int lane, int ef)
{
    if (ef & EF_OUT_UNSIGNED) epi_drain<false, CLAMP, false, FORM | EF_OUT_UNSIGNED | EF_PERM>(e, tbase, cbase, region_off, rb, lane);
    else epi_drain<false, CLAMP, false, FORM | EF_PERM>(e, tbase, cbase, region_off, rb, lane);
}

template <bool CLAMP, int FORMS>
__device__ __forceinline__ void dual_drain_branch(const EpiTile& e, unsigned tbase, int cbase, unsigned region_off, const unsigned* rb, int lane, int ef)
{
    const int form = FORMS == DUAL_INT ? 0 : (FORMS == DUAL_FLOAT ? EF_FLOAT : ef & (EF_WIDE | EF_FLOAT));
    if (FORMS != DUAL_INT && form == EF_FLOAT) dual_drain_branch_form<CLAMP, EF_FLOAT>(e, tbase, cbase, region_off, rb, lane, ef);
    else if (FORMS == DUAL_ANY && form == EF_WIDE) dual_drain_branch_form<CLAMP, EF_WIDE>(e, tbase, cbase, region_off, rb, lane, ef);
    else if (FORMS != DUAL_FLOAT) dual_drain_branch_form<CLAMP, 0>(e, tbase, cbase, region_off, rb, lane, ef);
}

template <bool CLAMP, int FORM>
__device__ __forceinline__ void dual_drain_sum_form(const EpiTile& e, unsigned tbase, int cbase, unsigned region_off, const unsigned* rb, int lane, int ef)
{
    switch (ef & (EF_OUT_UNSIGNED | EF_RES_UNSIGNED)) {
    case 0: epi_drain<true, CLAMP, false, FORM | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
    case EF_OUT_UNSIGNED: epi_drain<true, CLAMP, false, FORM | EF_OUT_UNSIGNED | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
    case EF_RES_UNSIGNED: epi_drain<true, CLAMP, false, FORM | EF_RES_UNSIGNED | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
    default: epi_drain<true, CLAMP, false, FORM | EF_OUT_UNSIGNED | EF_RES_UNSIGNED | EF_PERM>(e, tbase, cbase, region_off, rb, lane); break;
    }
}

// The projection's accumulator and the sum, in place of the branch's bytes
template <int MODE, int FORMS>
__device__ __forceinline__ void dual_drain_sum(const EpiTile& e, unsigned tbase, int cbase, unsigned region_off, const unsigned* rb, int lane, int ef)
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
    const int form = FORMS == DUAL_INT ? 0 : (FORMS == DUAL_FLOAT ? EF_FLOAT : ef & (EF_WIDE | EF_FLOAT));
    if (FORMS != DUAL_INT && form == EF_FLOAT) dual_drain_sum_form<CLAMP, EF_FLOAT>(e, tbase, cbase, region_off, rb, lane, ef);
    else if (FORMS == DUAL_ANY && form == EF_WIDE) dual_drain_sum_form<CLAMP, EF_WIDE>(e, tbase, cbase, region_off, rb, lane, ef);
    else if (FORMS != DUAL_FLOAT) dual_drain_sum_form<CLAMP, 0>(e, tbase, cbase, region_off, rb, lane, ef);
}

template <int MODE, int FORMS>
__global__ void __launch_bounds__(NUM_THREADS, 1)
igemm_dual_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmB0, const __grid_constant__ CUtensorMap tmA1,
                          const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ CUtensorMap tmO, const DualArgs d)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const IgemmArgs& a = d.g;
    const int resident = a.b_resident ? d.seg[1].b_first + d.seg[1].num_kb * d.seg[1].b_bytes : 0;
    unsigned char* const tiles = smem + resident;
    unsigned char* const stage_out = tiles + (size_t)a.stages * d.slot_bytes;
    unsigned long long* const bars = (unsigned long long*)(stage_out + NUM_EPI_WARPS * REGION_BYTES * DUAL_REGIONS);
    // bars: full[stages], empty[stages], tmem_full[8], tmem_empty[8], constants, resident weights
    const unsigned full0 = smem_u32(bars), empty0 = full0 + 8u * a.stages, tfull0 = empty0 + 8u * a.stages, tempty0 = tfull0 + 8u * MAX_ACC;
    const unsigned pready = tempty0 + 8u * MAX_ACC, bfull = pready + 8u;
    unsigned* const tmem_slot = (unsigned*)(bars + 2 * a.stages + 2 * MAX_ACC + 2);
    volatile int* const abort_flag = (volatile int*)(tmem_slot + 1);
    int* const par = (int*)(((uintptr_t)(tmem_slot + 4) + 15) & ~(uintptr_t)15);   // [sets][FAST_NP][256]
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    constexpr int LAST_PRODUCERS = EPI_WARP0 + NUM_EPI_WARPS;
    const int producer = warp == 0 ? 0 : (warp >= LAST_PRODUCERS ? warp - LAST_PRODUCERS + 1 : -1);
    pdl_launch_dependents();

    if (warp == 0) {
        const int nb = 2 * a.stages + 2 * MAX_ACC + 2;
        for (int i = lane; i < nb; i += 32) {
            const int j = i - (2 * a.stages + MAX_ACC);
            unsigned n = 1;
            if (j >= 0 && j < MAX_ACC) n = 4u * a.parts;
            else if (i == nb - 2) n = NUM_EPI_WARPS;
            else if (i == nb - 1) n = NUM_PRODUCERS;
            mbar_init(full0 + 8u * i, n);
        }
        if (lane == 0) {
            *abort_flag = 0;
            prefetch_tensor_map(&tmA0);
            prefetch_tensor_map(&tmB0);
            prefetch_tensor_map(&tmA1);
            prefetch_tensor_map(&tmB1);
            prefetch_tensor_map(&tmO);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = *tmem_slot;
    const unsigned tiles_s = smem_u32(tiles), res_b_s = smem_u32(smem);
    const int num_tiles = a.num_m_tiles * a.num_n_tiles;
    const int first = (int)blockIdx.x;
    const int n0 = (first % a.num_n_tiles) * a.BN;   // a CTA keeps its column block (the launcher sees to it)

    if (producer >= 0) {
        // ------------------------------------------------------------------ TMA producers (see igemm_kernel.cuh)
        bool ok = true;
        int m_tile = first / a.num_n_tiles;
        PixelPos px;
        px.start(a, a.m_base + m_tile * BM);
        const int takers = a.takers, my_turn = producer < takers ? producer : 0x40000000;
        const int all_kb = d.seg[0].num_kb + d.seg[1].num_kb;
        unsigned pre = 0;   // ring fills whose weights are issued before the wait
        if (a.late_weights) pdl_wait();
        if (first < num_tiles) {
            if (!a.b_resident) pre = (unsigned)min(all_kb, a.stages);
            const int nload = a.b_resident ? all_kb : (int)pre;
            if (elect_one()) {
                int own = 0, turn = my_turn;
                if (a.b_resident) {
                    for (int i = my_turn; i < all_kb; i += takers) own += i < d.seg[0].num_kb ? d.seg[0].b_bytes : d.seg[1].b_bytes;
                    mbar_expect_tx(bfull, (unsigned)own);
                }
                int kb = 0, kc = 0, kcoord = 0;
                bool second = false;
                for (int i = 0; i < nload; ++i) {
                    if (kb == d.seg[0].num_kb && !second) { second = true; kb = kc = kcoord = 0; }
                    const DualSegment& s = d.seg[second ? 1 : 0];
                    if (turn == 0) {
                        turn = takers;
                        const CUtensorMap* const tm = second ? &tmB1 : &tmB0;
                        if (a.b_resident) {
                            tma_load_2d(res_b_s + (unsigned)(s.b_first + kb * s.b_bytes), tm, bfull, kcoord, n0);
                        } else {
                            const unsigned bar = full0 + 8u * i;
                            mbar_expect_tx(bar, (unsigned)s.tx);
                            tma_load_2d(tiles_s + (unsigned)(i * d.slot_bytes + s.a_bytes), tm, bar, kcoord, n0);
                        }
                    }
                    --turn;
                    ++kb;
                    if (++kc == s.kchunks) { kc = 0; kcoord += s.tail; } else kcoord += s.BK;
                }
            }
            __syncwarp();
        }
        bool waited = false;
        const unsigned ring_end = full0 + 8u * a.stages, to_empty = 8u * a.stages;
        unsigned bar = full0, dst = tiles_s, ph = 1u, it = 0;
        int turn = my_turn;
        for (int tile = first; tile < num_tiles && ok; tile += gridDim.x) {
            const int m0 = a.m_base + m_tile * BM;
#pragma unroll
            for (int sg = 0; sg < 2; ++sg) {
                const DualSegment& s = d.seg[sg];
                const CUtensorMap *const ta = sg ? &tmA1 : &tmA0, *const tb = sg ? &tmB1 : &tmB0;
                const int iw0 = px.ox * s.sX - s.pL, ih0 = px.oy * s.sY - s.pT;
                int kx = 0, ky = 0, kc = 0, kcoord = 0;
                for (int kb = 0; kb < s.num_kb && ok; ++kb, ++it) {
                    if (turn == 0) {
                        turn = takers;
                        if (!mbar_wait_issuer(bar + to_empty, ph, abort_flag, a.status, 41)) { ok = false; break; }
                        if (!waited) {   // weights are constants; the activations are the previous kernel's output
                            pdl_wait();
                            waited = true;
                        }
                        if (elect_one()) {
                            const bool weights = it >= pre;   // else they are on their way
                            if (weights) mbar_expect_tx(bar, (unsigned)s.tx);
                            if (s.im2col) tma_load_im2col_4d(dst, ta, bar, kc * s.BK, iw0, ih0, px.n, (unsigned short)(kx * s.dX), (unsigned short)(ky * s.dY));
                            else tma_load_2d(dst, ta, bar, kcoord, m0);
                            if (weights && !a.b_resident) tma_load_2d(dst + (unsigned)s.a_bytes, tb, bar, kcoord, n0);
                        }
                        __syncwarp();
                    }
                    --turn;
                    bar += 8u;
                    dst += (unsigned)d.slot_bytes;
                    if (bar == ring_end) { bar = full0; dst = tiles_s; ph ^= 1u; }
                    if (++kc == s.kchunks) {
                        kc = 0;
                        kcoord += s.tail;
                        if (++kx == s.kW) { kx = 0; ++ky; }
                    } else {
                        kcoord += s.BK;
                    }
                }
            }
            m_tile += a.step_m;
            px.advance(a, a.adv_tiles);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer: two accumulators per tile
        unsigned acc_it = 0;
        bool ok = true;
        if (a.b_resident && first < num_tiles) ok = mbar_wait_issuer(bfull, 0, abort_flag, a.status, 42);
        int s = 0;
        unsigned ph = 0;
        const unsigned a_lo0 = (tiles_s & 0x3ffffu) >> 4, slot16 = (unsigned)(d.slot_bytes >> 4);
        unsigned a_lo = a_lo0;
        for (int tile = first; tile < num_tiles && ok; tile += gridDim.x) {
#pragma unroll
            for (int sg = 0; sg < 2; ++sg, ++acc_it) {
                if (!ok) break;
                const DualSegment& g = d.seg[sg];
                const unsigned as = acc_it & ((1u << a.acc_shift) - 1u), aph = (acc_it >> a.acc_shift) & 1u;
                if (!mbar_wait_issuer(tempty0 + 8u * as, aph ^ 1u, abort_flag, a.status, 43)) { ok = false; break; }
                const unsigned d_tmem = tmem_base + as * (unsigned)a.BN;
                const unsigned desc_hi = (unsigned)(make_smem_desc(0u, g.BK) >> 32), a16 = (unsigned)(g.a_bytes >> 4), b16 = (unsigned)(g.b_bytes >> 4);
                unsigned b_res = ((res_b_s + (unsigned)g.b_first) & 0x3ffffu) >> 4;
                for (int kb = 0; kb < g.num_kb; ++kb) {
                    if (!mbar_wait_issuer(full0 + 8u * s, ph, abort_flag, a.status, 44)) { ok = false; break; }
                    tc_fence_after();
                    const unsigned al = a_lo, bl = a.b_resident ? b_res : a_lo + a16, ebar = empty0 + 8u * s;
                    a_lo += slot16;
                    b_res += b16;
                    if (++s == a.stages) { s = 0; ph ^= 1u; a_lo = a_lo0; }
                    if (elect_one()) {
                        tc_mma_i8_lohi(d_tmem, al, bl, desc_hi, g.idesc, kb > 0 ? 1u : 0u);
                        if (g.BK >= 64) tc_mma_i8_lohi(d_tmem, al + 2u, bl + 2u, desc_hi, g.idesc, 1u);
                        if (g.BK == 128) {
                            tc_mma_i8_lohi(d_tmem, al + 4u, bl + 4u, desc_hi, g.idesc, 1u);
                            tc_mma_i8_lohi(d_tmem, al + 6u, bl + 6u, desc_hi, g.idesc, 1u);
                        }
                        tc_commit(ebar);
                        if (kb + 1 == g.num_kb) tc_commit(tfull0 + 8u * as);
                    }
                    __syncwarp();
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue warps
        const int quad = warp & 3, part4 = (warp - EPI_WARP0) >> 2;
        const int part = part4 & (a.parts - 1), group = part4 / a.parts;
        const int wp = a.BN / a.parts, cbase = part * wp, bn_shift = 31 - __clz(a.BN);
        unsigned rb[4];
        perm_rowbase(rb, wp, lane, wp >= 32 ? 4 : 2);
        bool ok = true;
        if (first < num_tiles) {
            const int per_set = FAST_NP << bn_shift;
            for (int i = (warp - EPI_WARP0) * 32 + lane; i < DUAL_SETS * per_set; i += 32 * NUM_EPI_WARPS) {
                const int set = i / per_set, prm = (i - set * per_set) >> bn_shift, c = i & (a.BN - 1);
                const int* const src = set == 0 ? d.fq_a + (size_t)prm * d.cpad_a : (set == 1 ? a.fq : a.fq2) + (size_t)prm * a.cpad;
                par[(set * FAST_NP + prm) * 256 + c] = __ldg(src + n0 + c);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(pready);
            ok = mbar_wait_warp(pready, 0, abort_flag, a.status, 45);
        }
        pdl_wait();   // output stores touch a tensor that the previous kernel may read or write
        EpiTile e;
        e.BN = a.BN; e.N = a.N; e.M = a.m_base + a.M; e.n0 = n0; e.wp = wp;
        e.t_lo = a.t_lo; e.t_hi = a.t_hi;
        const unsigned par_off = (unsigned)((unsigned char*)par - smem_raw);
        const unsigned my_regions = (unsigned)(stage_out - smem_raw) + (unsigned)((warp - EPI_WARP0) * REGION_BYTES * DUAL_REGIONS);
        unsigned acc_it = 2u * (unsigned)group, mine = 0;
        int m0 = a.m_base + (first / a.num_n_tiles + group * a.step_m) * BM;
        for (int tile = first + group * (int)gridDim.x; tile < num_tiles && ok; tile += a.groups * (int)gridDim.x, acc_it += 2u * (unsigned)a.groups, ++mine) {
            const int gx = n0 + cbase, gy = m0 + quad * 32;
            const bool active = gx < a.N && gy < e.M;
            const unsigned region_off = my_regions + (mine & 1u) * REGION_BYTES;
            if (lane == 0) bulk_wait_read_1();   // the store before the last one has left this region
            __syncwarp();
            for (unsigned sg = 0; sg < 2; ++sg) {
                const unsigned as = (acc_it + sg) & ((1u << a.acc_shift) - 1u), aph = ((acc_it + sg) >> a.acc_shift) & 1u;
                if (!mbar_wait_warp(tfull0 + 8u * as, aph, abort_flag, a.status, 46)) { ok = false; break; }
                tc_fence_after();
                if (active) {
                    const unsigned tbase = tmem_base + as * (unsigned)a.BN + ((unsigned)(quad * 32) << 16) + (unsigned)cbase;
                    e.par_off = par_off + sg * (FAST_NP * 1024u);
                    if (sg) dual_drain_sum<MODE, FORMS>(e, tbase, cbase, region_off, rb, lane, a.ef);
                    else if (d.clamp_a) dual_drain_branch<true, FORMS>(e, tbase, cbase, region_off, rb, lane, d.ef_a);
                    else dual_drain_branch<false, FORMS>(e, tbase, cbase, region_off, rb, lane, d.ef_a);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty0 + 8u * as);
            }
            if (!ok) break;
            fence_async_smem();
            __syncwarp();
            if (lane == 0 && active) {
                tma_store_2d(&tmO, smem_u32(dyn_smem() + region_off), gx, gy);
                bulk_commit();
            }
            m0 += a.groups * a.step_m * BM;
        }
        if (lane == 0) bulk_wait_read_all();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(a.tmem_cols) : "memory");
    }
}

// By the projection's epilogue: with clamps, without, dot-product sum
typedef void (*DualKernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const DualArgs);
extern const DualKernel dual_float[3], dual_any[3];

}  // namespace n2d2b
