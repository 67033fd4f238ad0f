// Stride-1 convolution with a small channel count (32, 64 or 128) on the tensor cores, fed from an input
// patch that is loaded once: the 3x3 layers of the first ResNet stage, where the implicit-GEMM kernel
// would fetch every input pixel nine times through im2col loads and wait on a barrier per filter tap.
//
// A CTA works on a band of R output rows of one image.  One TMA load brings the (R + halo) x (oW + halo)
// x C input patch, zero-filled outside the image, into shared memory as rows of one pixel each (C bytes,
// swizzled by C).  Seen as a list of pixels p = y * Wp + x, the patch is its own im2col matrix: the operand
// of filter tap (ky, kx) for the 128 consecutive positions p0 .. p0+127 is the 128 patch rows that start
// at p0 + ky*dY*Wp + kx*dX.  So every tap is one shared-memory descriptor with a different start row,
// no data moves, and the MMAs of a tile (taps x C/32 of them) are issued back to back.  Positions in the
// halo columns (x >= oW) compute values nobody stores.  The weights of all taps stay resident.
//
// Depthwise layers of many pixels take the same route as block-diagonal groups: the channels are cut into groups of 64 (32), a
// CTA works on one group for its whole life (CTA b on group b mod G, so the group's weight block - its own taps on
// the diagonal, zeros elsewhere - stays resident), the patch load takes the group's channel slice of the NHWC tensor
// and the output rows are written into that slice.  The tensor core multiplies 64 times more than the layer needs.
// With 3x3 filters that is level with the dot-product kernel on the CUDA cores (conv_depthwise3x3_kernel) on large maps of few channels
// and behind it elsewhere (see dw3x3_faster); wider filters run 2 to 4 times faster than on their CUDA-core kernel (5x5 on 64 x 56 x 56,
// 64 images: 37 us against 137).
//
// Warp 0 loads (weights once, patches into two to four buffers), warps 1-4 issue tcgen05.mma kind::i8 for alternate
// tiles into a ring of four TMEM accumulators, and four groups of four epilogue warps (one warp per TMEM lane quadrant) each
// drain every fourth tile: 32-bit requantisation in the fragment layout, the bytes going from the registers straight to
// the NHWC output (eight consecutive channels per lane).  Every wait is bounded.
#pragma once
#include "kernels.h"
#include "tc_common.cuh"

namespace n2d2b {

static constexpr int PBM = 128;
static constexpr int P_EPI_WARPS = 16;
static constexpr int P_SLOTS = 4;            // TMEM accumulators = epilogue groups
static constexpr int P_ISSUERS = 4;           // MMA-issuing warps: tiles alternate between them
static constexpr int P_EPI_WARP0 = 1 + P_ISSUERS;
static constexpr int P_THREADS = 32 * (P_EPI_WARP0 + P_EPI_WARPS);
static constexpr int P_ISSUERS_RES = 2;       // with a residual sum: fewer warps, more registers for each
static constexpr int P_THREADS_RES = 32 * (1 + P_ISSUERS_RES + P_EPI_WARPS);
static constexpr int P_BRING_MIN = 4;         // weight ring slots (one filter tap each) when the weights stream:
static constexpr int P_BRING_MAX = 8;         // as many as shared memory holds between these two
static constexpr int P_BUFS_MAX = 4;          // patch buffers: small patches are consumed faster than two loads arrive

struct PatchArgs {
    int B, oH, oW, N, BN, C;   // N, C: output and input channels of one group (= of the layer when G == 1)
    int G;                  // channel groups (block-diagonal layers); CTA b works on group b % G
    int ldo;                // output channels per pixel of the whole tensor
    int taps_y, taps_x, dY, dX, pT, pL;
    int Wp;                 // patch width in pixels: oW + (kW-1)*dX
    int R;                  // output rows per band
    int bands;              // bands per image
    int n_base;             // first image of this call within the tensors (batch slices)
    int patch_bytes;        // bytes one patch load delivers (the full TMA box)
    int patch_alloc;        // bytes reserved per patch buffer (box + the rows a last tile may read past it)
    int nbuf;               // patch buffers
    int late_weights;       // weights only after the dependency wait
    int b_stream;           // weights too large to stay resident: their tap blocks stream through a ring
    int bring;              // slots of that ring
    unsigned rcp_Wp;        // ceil(2^32 / Wp)
    unsigned idesc, idesc_proj, tmem_cols;
    void* out;
    int* status;
    const int* fq;
    int cpad;
    int out_unsigned;
    // RES: residual tensor (the output's geometry), constants of the sum, range the cell's own output saturates to
    const uint8_t* res;
    int res_unsigned;
    const int* fq2;
    int t_lo, t_hi;
    // RES_DUAL: the layer is the branch of a sum whose other operand, a 1x1 projection of a second tensor, is computed beside it
    const int* fq_branch;   // the branch's rescale (fq: the projection's)
    int cpad_branch, proj_alloc, proj_bytes;
};

// What the epilogue adds: nothing, a residual tensor, or the branch (the patch) to a projection
static constexpr int RES_NONE = 0, RES_TENSOR = 1, RES_DUAL = 2;

// The MMAs of one tile with compile-time tap counts: a straight run of address adds and MMAs.  The issuing
// thread pays the latency of every instruction it executes, so loop control and address arithmetic around a
// short MMA (one of 128 x 64 x 32 takes about 60 cycles of the tensor pipe) would cost more than the MMA.
template <int KH, int KW, int KS>
__device__ __forceinline__ void issue_tile(unsigned d_tmem, unsigned a_lo, unsigned b_lo, unsigned desc_hi, unsigned idesc,
                                           unsigned row_step, unsigned col_step, unsigned btap)
{
#pragma unroll
    for (int ky = 0; ky < KH; ++ky)
#pragma unroll
        for (int kx = 0; kx < KW; ++kx)
#pragma unroll
            for (int k = 0; k < KS; ++k)
                tc_mma_i8_lohi(d_tmem, a_lo + ky * row_step + kx * col_step + 2u * k, b_lo + (ky * KW + kx) * btap + 2u * k,
                               desc_hi, idesc, (ky | kx | k) ? 1u : 0u);
}

// The MMAs of one filter tap of one tile (C / 32 K steps), unrolled for the channel counts the kernel takes
template <int KS>
__device__ __forceinline__ void issue_tap_n(unsigned d_tmem, unsigned a_lo, unsigned b_lo, unsigned desc_hi, unsigned idesc, unsigned first)
{
    tc_mma_i8_lohi(d_tmem, a_lo, b_lo, desc_hi, idesc, first);
#pragma unroll
    for (int k = 1; k < KS; ++k) tc_mma_i8_lohi(d_tmem, a_lo + 2u * k, b_lo + 2u * k, desc_hi, idesc, 1u);
}
__device__ __forceinline__ void issue_tap(int ksteps, unsigned d_tmem, unsigned a_lo, unsigned b_lo, unsigned desc_hi, unsigned idesc,
                                          unsigned first)
{
    if (ksteps == 4) issue_tap_n<4>(d_tmem, a_lo, b_lo, desc_hi, idesc, first);
    else if (ksteps == 2) issue_tap_n<2>(d_tmem, a_lo, b_lo, desc_hi, idesc, first);
    else issue_tap_n<1>(d_tmem, a_lo, b_lo, desc_hi, idesc, first);
}

// SHAPE: 0 = any filter (loops), 1 / 2 / 3 = 3x3 filter with 32 / 64 / 128 channels (unrolled issue).  FORM: EF_WIDE or
// EF_FLOAT, the form of the rescale (0: 32-bit); a template because a choice per 32-column block inside the epilogue
// cost 2 % of a MobileNet.  RES: a residual sum in the epilogue (64 -> 64 channels); the bytes are loaded before the wait for the
// accumulator.  2.2_3x3_2 of ResNet-18 at 2048 images, clamped: 596 us on the implicit-GEMM kernel, 412 here
// RES_DUAL: a residual block's first unit, 64 -> 64 channels 3x3 beside a 64 -> 64 channel projection of the block's input, whose band arrives as a patch of its
// own without a border: one more tap into an accumulator of its own.  The branch's bytes stay in registers.  conv2.1 of ResNet-18 at 128 images 28.4 and 28.8 us
// by themselves, 40.8 here; 2048 images 603 / 469
template <bool CLAMP, int SHAPE, int FORM, int RES>
__global__ void __launch_bounds__(RES ? P_THREADS_RES : P_THREADS, 1)
patch_conv_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmA2,
                          const __grid_constant__ CUtensorMap tmB2, const PatchArgs a)
{
    constexpr int ISSUERS = RES ? P_ISSUERS_RES : P_ISSUERS, EPI_WARP0 = 1 + ISSUERS, THREADS = RES ? P_THREADS_RES : P_THREADS;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int taps = a.taps_y * a.taps_x;
    const int b_tap_bytes = a.BN * a.C;
    unsigned char* res_b = smem;                                              // [taps][BN][C], or a ring of a.bring taps
    unsigned char* patch0 = smem + (((size_t)(a.b_stream ? a.bring : taps + (RES == RES_DUAL ? 1 : 0)) * b_tap_bytes + 1023) & ~(size_t)1023);
    unsigned char* proj0 = patch0 + (size_t)a.nbuf * a.patch_alloc;            // RES_DUAL: the projection's bands
    unsigned long long* bars = (unsigned long long*)(proj0 + (RES == RES_DUAL ? (size_t)a.nbuf * a.proj_alloc : 0));
    // bars: patch_full[4], patch_empty[4], tmem_full[4], tmem_empty[4], weights, (spare), ring_full[8], ring_empty[8]
    const unsigned pfull0 = smem_u32(bars);
    const unsigned pempty0 = pfull0 + 8u * P_BUFS_MAX;
    const unsigned tfull0 = pempty0 + 8u * P_BUFS_MAX;
    const unsigned tempty0 = tfull0 + 8u * P_SLOTS;
    const unsigned bfull = tempty0 + 8u * P_SLOTS;
    const unsigned rfull0 = bfull + 16u;
    const unsigned rempty0 = rfull0 + 8u * P_BRING_MAX;
    unsigned* tmem_slot = (unsigned*)(bars + 2 * P_BUFS_MAX + 2 * P_SLOTS + 2 + 2 * P_BRING_MAX);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    int* par = (int*)(((uintptr_t)(tmem_slot + 4) + 15) & ~(uintptr_t)15);   // [FAST_NP][256]

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    pdl_launch_dependents();

    if (threadIdx.x == 0) {
        for (int s = 0; s < P_BUFS_MAX; ++s) {
            mbar_init(pfull0 + 8u * s, 1);
            mbar_init(pempty0 + 8u * s, ISSUERS);
        }
        for (int s = 0; s < P_SLOTS; ++s) {
            mbar_init(tfull0 + 8u * s, 1);
            mbar_init(tempty0 + 8u * s, 4);
        }
        mbar_init(bfull, 1);
        for (int r = 0; r < P_BRING_MAX; ++r) {
            mbar_init(rfull0 + 8u * r, 1);
            mbar_init(rempty0 + 8u * r, ISSUERS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // this CTA's channel group, and its place among the CTAs of that group
    const int grp = (int)blockIdx.x % a.G, cta = (int)blockIdx.x / a.G, nctas = (int)gridDim.x / a.G;
    const int ch0 = grp * a.N;                       // first output channel (= first input channel) of the group
    for (int i = threadIdx.x; i < FAST_NP * 256; i += THREADS) {
        const int prm = i >> 8, c = i & 255;
        if (RES == RES_DUAL && c >= 64 && c < 128) par[i] = __ldg(a.fq_branch + (size_t)prm * a.cpad_branch + c - 64);
        else if (RES && c >= 128) par[i] = __ldg(a.fq2 + (size_t)prm * a.cpad + c - 128);
        else par[i] = (ch0 + c < a.cpad) ? __ldg(a.fq + (size_t)prm * a.cpad + ch0 + c) : 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = *tmem_slot;
    const int items = a.B * a.bands;
    // rows and 128-position tiles of band `band` (the last band of an image may be shorter)
    auto band_rows = [&](int band) { const int r = a.oH - band * a.R; return r < a.R ? r : a.R; };
    auto band_tiles = [&](int band) { return (band_rows(band) * a.Wp + PBM - 1) / PBM; };

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0 && cta < items) {
            prefetch_tensor_map(&tmA);
            prefetch_tensor_map(&tmB);
            unsigned pre = 0, wt = 0;   // ring fills issued before the wait, ring fills so far
            if (a.late_weights) pdl_wait();
            if (a.b_stream) {
                pre = (unsigned)(taps < a.bring ? taps : a.bring);
                for (unsigned t = 0; t < pre; ++t) {
                    mbar_expect_tx(rfull0 + 8u * t, (unsigned)b_tap_bytes);
                    tma_load_2d(smem_u32(res_b + (size_t)t * b_tap_bytes), &tmB, rfull0 + 8u * t, (int)t * a.C, ch0);
                }
            } else {
                mbar_expect_tx(bfull, (unsigned)((taps + (RES == RES_DUAL ? 1 : 0)) * b_tap_bytes));
                if (RES == RES_DUAL) tma_load_2d(smem_u32(res_b + (size_t)taps * b_tap_bytes), &tmB2, bfull, 0, 0);
                for (int t = 0; t < taps; ++t)
                    tma_load_2d(smem_u32(res_b + (size_t)t * b_tap_bytes), &tmB, bfull, t * a.C, ch0);
            }
            pdl_wait();   // weights are constants; the activations are the previous kernel's output
            unsigned pb = 0, ph = 0;   // patch buffer and its phase
            int rs = 0;              // weight ring slot and its phase
            unsigned rph = 0;
            bool ok = true;
            int n = cta / a.bands, band = cta % a.bands;
            const int step_n = nctas / a.bands, step_b = nctas % a.bands;
            for (int item = cta; item < items; item += nctas) {
                if (!mbar_wait(pempty0 + 8u * pb, ph ^ 1u, abort_flag, a.status, 1)) break;
                mbar_expect_tx(pfull0 + 8u * pb, (unsigned)(a.patch_bytes + (RES == RES_DUAL ? a.proj_bytes : 0)));
                if (RES == RES_DUAL)
                    tma_load_4d(smem_u32(proj0 + (size_t)pb * a.proj_alloc), &tmA2, pfull0 + 8u * pb, 0, 0, band * a.R, a.n_base + n);
                tma_load_4d(smem_u32(patch0 + (size_t)pb * a.patch_alloc), &tmA, pfull0 + 8u * pb, grp * a.C, -a.pL,
                            band * a.R - a.pT, a.n_base + n);
                if (a.b_stream) {
                    // every item walks all taps once: its weights follow the patch through the ring
                    for (int t = 0; t < taps && ok; ++t, ++wt) {
                        if (wt < pre) {
                            if (++rs == a.bring) { rs = 0; rph ^= 1u; }
                            continue;
                        }
                        if (!mbar_wait(rempty0 + 8u * rs, rph ^ 1u, abort_flag, a.status, 5)) { ok = false; break; }
                        mbar_expect_tx(rfull0 + 8u * rs, (unsigned)b_tap_bytes);
                        tma_load_2d(smem_u32(res_b + (size_t)rs * b_tap_bytes), &tmB, rfull0 + 8u * rs, t * a.C, ch0);
                        if (++rs == a.bring) { rs = 0; rph ^= 1u; }
                    }
                    if (!ok) break;
                }
                if (++pb == (unsigned)a.nbuf) { pb = 0; ph ^= 1u; }
                n += step_n;
                band += step_b;
                if (band >= a.bands) { band -= a.bands; ++n; }
            }
        }
    } else if (warp < EPI_WARP0) {
        // ------------------------------------------------------------------ MMA issuers
        // An MMA of 128 x 64 x 32 costs its issuing warp about 48 cycles and the tensor pipe 50, but waits, commits and address updates
        // come on top: four warps (two beside a residual sum) take alternate tiles, whose accumulators are independent.
        // every lane of the warp runs the loop, an elected one issues (see elect_one)
        const unsigned me = (unsigned)__shfl_sync(0xffffffffu, warp - 1, 0);
        if (cta < items) {
            bool ok = a.b_stream ? true : mbar_wait_uniform(bfull, 0, abort_flag, a.status, 8);
            const unsigned desc_hi = (unsigned)(make_smem_desc(0u, a.C) >> 32);
            const unsigned res_b_lo = (smem_u32(res_b) & 0x3ffffu) >> 4, patch_lo = (smem_u32(patch0) & 0x3ffffu) >> 4;
            const int ksteps = a.C / 32;
            const unsigned row_step = (unsigned)((a.dY * a.Wp * a.C) >> 4), col_step = (unsigned)((a.dX * a.C) >> 4);
            const unsigned btap = (unsigned)(b_tap_bytes >> 4);
            unsigned pb = 0, ph = 0, seq = 0;
            int band = cta % a.bands;
            const int step_b = nctas % a.bands;
            const unsigned tile_step = (unsigned)((PBM * a.C) >> 4);
            int rs = 0;              // weight ring slot and its phase (streamed weights)
            unsigned rph = 0;
            for (int item = cta; item < items && ok; item += nctas) {
                const int T = band_tiles(band);
                if (!mbar_wait_uniform(pfull0 + 8u * pb, ph, abort_flag, a.status, 3)) { ok = false; break; }
                tc_fence_after();
                unsigned a_lo = patch_lo + pb * (unsigned)(a.patch_alloc >> 4);
                unsigned proj_lo = ((smem_u32(proj0) & 0x3ffffu) >> 4) + pb * (unsigned)(a.proj_alloc >> 4);
                if (a.b_stream) {
                    // At most P_SLOTS tiles per item, each with its own accumulator: this thread owns tiles `me` and
                    // `me + P_ISSUERS` and walks the taps as their weights arrive, so one pass of the weights serves
                    // the whole band; a thread without a tile still releases every ring slot.
                    const bool mine0 = (int)me < T, mine1 = (int)me + ISSUERS < T;
                    const unsigned seq0 = seq + me, seq1 = seq0 + ISSUERS;
                    const unsigned slot0 = seq0 & (P_SLOTS - 1), slot1 = seq1 & (P_SLOTS - 1);
                    if (mine0 && !mbar_wait_uniform(tempty0 + 8u * slot0, ((seq0 / P_SLOTS) & 1u) ^ 1u, abort_flag, a.status, 2)) { ok = false; break; }
                    if (mine1 && !mbar_wait_uniform(tempty0 + 8u * slot1, ((seq1 / P_SLOTS) & 1u) ^ 1u, abort_flag, a.status, 2)) { ok = false; break; }
                    tc_fence_after();
                    const unsigned d0 = tmem_base + slot0 * (unsigned)a.BN, d1 = tmem_base + slot1 * (unsigned)a.BN;
                    const unsigned tile2 = (unsigned)ISSUERS * tile_step;
                    unsigned ar = a_lo + me * tile_step, first = 0;
                    for (int ky = 0; ky < a.taps_y && ok; ++ky, ar += row_step) {
                        unsigned ac = ar;
                        for (int kx = 0; kx < a.taps_x; ++kx, ac += col_step) {
                            if (!mbar_wait_uniform(rfull0 + 8u * rs, rph, abort_flag, a.status, 6)) { ok = false; break; }
                            tc_fence_after();
                            const unsigned bt = res_b_lo + (unsigned)rs * btap;
                            if (elect_one()) {
                                if (mine0) issue_tap(ksteps, d0, ac, bt, desc_hi, a.idesc, first);
                                if (mine1) issue_tap(ksteps, d1, ac + tile2, bt, desc_hi, a.idesc, first);
                                tc_commit(rempty0 + 8u * rs);
                            }
                            __syncwarp();
                            first = 1u;
                            if (++rs == a.bring) { rs = 0; rph ^= 1u; }
                        }
                    }
                    if (!ok) break;
                    if (elect_one()) {
                        if (mine0) tc_commit(tfull0 + 8u * slot0);
                        if (mine1) tc_commit(tfull0 + 8u * slot1);
                        tc_commit(pempty0 + 8u * pb);
                    }
                    __syncwarp();
                    seq += (unsigned)T;
                    if (++pb == (unsigned)a.nbuf) { pb = 0; ph ^= 1u; }
                    band += step_b;
                    if (band >= a.bands) band -= a.bands;
                    continue;
                }
                for (int t = 0; t < T; ++t, ++seq, a_lo += tile_step, proj_lo += tile_step) {
                    if ((seq & (ISSUERS - 1)) != me) continue;
                    const unsigned slot = seq & (P_SLOTS - 1), sph = (seq / P_SLOTS) & 1u;
                    if (!mbar_wait_uniform(tempty0 + 8u * slot, sph ^ 1u, abort_flag, a.status, 2)) { ok = false; break; }
                    tc_fence_after();
                    const unsigned d_tmem = tmem_base + slot * (unsigned)a.BN;
                    // The operand of a tap starts at an arbitrary pixel row.  The swizzle is a function of the
                    // absolute shared-memory address, so the descriptor needs nothing but that address
                    // (measured: with the base-offset field left 0 every start row gives exact results).
                    if (elect_one()) {
                        if (SHAPE == 1) issue_tile<3, 3, 1>(d_tmem, a_lo, res_b_lo, desc_hi, a.idesc, row_step, col_step, btap);
                        else if (SHAPE == 2) issue_tile<3, 3, 2>(d_tmem, a_lo, res_b_lo, desc_hi, a.idesc, row_step, col_step, btap);
                        else if (SHAPE == 3) issue_tile<3, 3, 4>(d_tmem, a_lo, res_b_lo, desc_hi, a.idesc, row_step, col_step, btap);
                        else {
                            unsigned ar = a_lo, bt = res_b_lo, first = 0;
                            for (int ky = 0; ky < a.taps_y; ++ky, ar += row_step) {
                                unsigned ac = ar;
                                for (int kx = 0; kx < a.taps_x; ++kx, ac += col_step, bt += btap)
                                    for (int k = 0; k < ksteps; ++k) {
                                        tc_mma_i8_lohi(d_tmem, ac + 2u * k, bt + 2u * k, desc_hi, a.idesc, first);
                                        first = 1u;
                                    }
                            }
                        }
                        if (RES == RES_DUAL) issue_tap_n<2>(d_tmem + P_SLOTS * 64u, proj_lo, res_b_lo + (unsigned)taps * btap, desc_hi, a.idesc_proj, 0u);
                        tc_commit(tfull0 + 8u * slot);
                    }
                    __syncwarp();
                }
                if (ok && elect_one()) tc_commit(pempty0 + 8u * pb);   // the patch is free once every issuer's MMAs have read it
                __syncwarp();
                if (++pb == (unsigned)a.nbuf) { pb = 0; ph ^= 1u; }
                band += step_b;
                if (band >= a.bands) band -= a.bands;
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue warps
        pdl_wait();   // the output buffer may still be read by the previous kernel
        const int ew = warp - EPI_WARP0;
        const int quad = warp & 3;          // TMEM lane quadrant this warp may read
        const int group = ew >> 2;          // drains the tiles whose sequence number is `group` modulo 4
        const unsigned par_off = (unsigned)((unsigned char*)par - smem_raw);
        unsigned seq = 0;
        int n = cta / a.bands, band = cta % a.bands;
        const int step_n = nctas / a.bands, step_b = nctas % a.bands;
        bool ok = true;
        for (int item = cta; item < items && ok; item += nctas) {
            const int rows = band_rows(band);
            const int T = band_tiles(band);
            uint8_t* const band_out = (uint8_t*)a.out + ((size_t)(a.n_base + n) * a.oH + (size_t)(band * a.R)) * a.oW * a.ldo + ch0;
            for (int t = 0; t < T; ++t, ++seq) {
                if ((int)(seq & (P_SLOTS - 1)) != group) continue;
                const unsigned sph = (seq / P_SLOTS) & 1u;
                // This lane's four rows of the fragment (positions of the band's raster) and where they go: the bytes leave
                // the registers for global memory directly, eight channels per lane, a 32-byte sector per four lanes
                unsigned rowoff[4];   // byte offsets within the band: below 2^32
                unsigned rowok = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const unsigned p = (unsigned)(t * PBM + quad * 32 + (lane >> 2) + 8 * k);
                    const unsigned yy = __umulhi(p, a.rcp_Wp);
                    const unsigned x = p - yy * (unsigned)a.Wp;
                    if (x < (unsigned)a.oW && yy < (unsigned)rows) rowok |= 1u << k;
                    rowoff[k] = (yy * (unsigned)a.oW + x) * (unsigned)a.ldo;
                }
                uint2 res[4];
                const uint8_t* const rp = a.res + (band_out - (uint8_t*)a.out) + 8 * (lane & 3);
                if (RES == RES_TENSOR) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) res[k] = (rowok >> k) & 1u ? __ldg((const uint2*)(rp + rowoff[k])) : make_uint2(0u, 0u);
                }
                if (!mbar_wait_warp(tfull0 + 8u * group, sph, abort_flag, a.status, 4)) { ok = false; break; }
                tc_fence_after();
                const unsigned tbase = tmem_base + ((unsigned)(quad * 32) << 16) + (unsigned)(group * a.BN);
                if (RES) {
#pragma unroll 1
                    for (int cb = 0; cb < 64; cb += 32) {
                        unsigned va[16], vb[16];
                        if (RES == RES_DUAL) {
                            tc_ld_2x16x256b_x4_wait(tbase + (unsigned)cb, va, vb);
                            if (a.res_unsigned) perm_block_words<CLAMP, FORM | EF_OUT_UNSIGNED>(va, vb, par_off, 64 + cb, res, lane);
                            else perm_block_words<CLAMP, FORM>(va, vb, par_off, 64 + cb, res, lane);
                        }
                        tc_ld_2x16x256b_x4_wait(tbase + (RES == RES_DUAL ? P_SLOTS * 64u : 0u) + (unsigned)cb, va, vb);
                        switch ((a.out_unsigned ? EF_OUT_UNSIGNED : 0) | (a.res_unsigned ? EF_RES_UNSIGNED : 0)) {
                        case 0: perm_block_global<CLAMP, FORM, RES != RES_NONE>(va, vb, par_off, cb, band_out + cb, rowoff, rowok, lane, res, a.t_lo, a.t_hi); break;
                        case EF_OUT_UNSIGNED: perm_block_global<CLAMP, FORM | EF_OUT_UNSIGNED, RES != RES_NONE>(va, vb, par_off, cb, band_out + cb, rowoff, rowok, lane, res, a.t_lo, a.t_hi); break;
                        case EF_RES_UNSIGNED: perm_block_global<CLAMP, FORM | EF_RES_UNSIGNED, RES != RES_NONE>(va, vb, par_off, cb, band_out + cb, rowoff, rowok, lane, res, a.t_lo, a.t_hi); break;
                        default: perm_block_global<CLAMP, FORM | EF_OUT_UNSIGNED | EF_RES_UNSIGNED, RES != RES_NONE>(va, vb, par_off, cb, band_out + cb, rowoff, rowok, lane, res, a.t_lo, a.t_hi); break;
                        }
                        if (RES == RES_TENSOR && cb == 0) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) res[k] = (rowok >> k) & 1u ? __ldg((const uint2*)(rp + rowoff[k] + 32)) : make_uint2(0u, 0u);
                        }
                    }
                } else {
#pragma unroll 1
                    for (int cb = 0; cb < a.N; cb += 32) {
                        unsigned va[16], vb[16];
                        tc_ld_2x16x256b_x4_wait(tbase + (unsigned)cb, va, vb);
                        if (a.out_unsigned) perm_block_global<CLAMP, FORM | EF_OUT_UNSIGNED>(va, vb, par_off, cb, band_out + cb, rowoff, rowok, lane);
                        else perm_block_global<CLAMP, FORM>(va, vb, par_off, cb, band_out + cb, rowoff, rowok, lane);
                    }
                }
                // the accumulator is drained: hand it back
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty0 + 8u * group);
            }
            n += step_n;
            band += step_b;
            if (band >= a.bands) { band -= a.bands; ++n; }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(a.tmem_cols) : "memory");
    }
}

// The kernels by [clamped][filter shape; with a residual sum; with a projection], one module for each form of the rescale (patch_tcgen05.cu, patch_float.cu,
// patch_wide.cu): loading a kernel loads the module it is in, and a network rarely has two forms
typedef void (*PatchKernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const PatchArgs);
extern const PatchKernel patch_float[2][6], patch_wide[2][6];
#define N2D2B_PATCH(C, F) {patch_conv_tcgen05_kernel<C, 0, F, RES_NONE>, patch_conv_tcgen05_kernel<C, 1, F, RES_NONE>, patch_conv_tcgen05_kernel<C, 2, F, RES_NONE>, \
                           patch_conv_tcgen05_kernel<C, 3, F, RES_NONE>, patch_conv_tcgen05_kernel<C, 2, F, RES_TENSOR>, patch_conv_tcgen05_kernel<C, 2, F, RES_DUAL>}
#define N2D2B_PATCH_KERNELS(F) {N2D2B_PATCH(false, F), N2D2B_PATCH(true, F)}

}  // namespace n2d2b
