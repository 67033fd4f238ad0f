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
#include <cstring>
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

// ----------------------------------------------------------------------------- host side
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
    typedef void (*PatchKernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const PatchArgs);
#define N2D2B_PATCH(C, F) patch_conv_tcgen05_kernel<C, 0, F, RES_NONE>, patch_conv_tcgen05_kernel<C, 1, F, RES_NONE>, patch_conv_tcgen05_kernel<C, 2, F, RES_NONE>, \
                          patch_conv_tcgen05_kernel<C, 3, F, RES_NONE>, patch_conv_tcgen05_kernel<C, 2, F, RES_TENSOR>, patch_conv_tcgen05_kernel<C, 2, F, RES_DUAL>
    static const PatchKernel variants[36] = {N2D2B_PATCH(false, 0), N2D2B_PATCH(true, 0), N2D2B_PATCH(false, EF_FLOAT),
                                             N2D2B_PATCH(true, EF_FLOAT), N2D2B_PATCH(false, EF_WIDE), N2D2B_PATCH(true, EF_WIDE)};
#undef N2D2B_PATCH
    static SmemLimitSet limits[36];
    // a multiple of the group count: CTA b works on group b % G
    const long long items = (long long)a.B * a.bands;
    const long long per_group = plan.num_sms / plan.G > 0 ? plan.num_sms / plan.G : 1;
    const int grid = (int)((items < per_group ? items : per_group) * plan.G);
    const int shape = branch ? 5 : r.ptr ? 4 : (g.kH == 3 && g.kW == 3 && !plan.b_stream) ? (g.C == 32 ? 1 : (g.C == 64 ? 2 : 3)) : 0;
    const int v = (fast.form == EF_WIDE ? 24 : (fast.form == EF_FLOAT ? 12 : 0)) + (fast.need_clamp || (branch && branch->need_clamp) ? 6 : 0) + shape;
    if (cudaError_t e = raise_smem_limit(variants[v], limits[v])) return e;
    return launch_pdl(variants[v], grid, r.ptr || branch ? P_THREADS_RES : P_THREADS, plan.smem_bytes, s, plan.tmA, plan.tmB, plan.tmA2, plan.tmB2, a);
}

}  // namespace n2d2b
