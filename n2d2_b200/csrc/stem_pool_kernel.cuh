// First layer with stride 2 and 64 output channels whose only reader is an unpadded 3x3 / 2 max pooling (the head of the ResNets),
// as one kernel on the tensor cores: the convolution's own output, the largest tensor of such a network, never exists.
//
// As two kernels the pair is bound by the requantisation of 64 x 12544 values per image and by writing and reading them again
// (ResNet-50 at 1024 images: 430 us with the re-layout of the image, 270 us for the pooling).  Rescaling with
// a multiplier that is not negative, rounding and saturation never decrease, so the maximum may be taken first: this kernel pools
// the 32-bit accumulators and requantises a quarter of the values.
//
// The matrices are turned around to make that cheap.  Weights are the M operand: 128 rows = 64 channels x two adjacent
// convolution rows (the second row's filter is the first one's, one image row further down, so the K extent grows by one filter
// row); positions are the N operand.  The image is re-laid as in the space-to-depth kernel (16-byte pixels of a
// 2 x 2 block x 4 channels), and its bytes in shared memory are the operand: row n of the matrix starts at byte 16 n and is
// 32 bytes long.  One row pair takes (KH + 1) * KWp / 2 MMAs of 128 x N x 32, N = the row's positions rounded up to 16: for a
// 7x7 filter on 224 x 224 ten of 128 x 112 x 32, no halo columns.
//
// An accumulator lane then holds one channel of one convolution row, its columns the positions: the horizontal maximum of three
// stays in the thread.  The M rows are ordered so that lanes l and l + 16 of a quadrant are the same channel of the two rows; one shuffle
// per two values exchanges halves (lanes below 16 finish the left half of a warp's pooled columns, the others the right
// half), and the third row of a window is the first row of the next pair, which the same warp drains.  No barrier joins
// the epilogue warps, four of which (16 channels each) share a quarter of the columns.
//
// Warp 0 loads pairs of image rows through a ring, warps 1 and 18 issue the MMAs into four accumulators, warps 2-17 are the
// epilogue.  A work item is a band of pooled rows of one image; bands are as tall as the batch allows, each
// computes one row pair more than it has pooled rows.  Every wait is bounded.
#pragma once
#include "kernels.h"
#include "tc_common.cuh"

namespace n2d2b {

static constexpr int SP_SLOTS = 4;            // TMEM accumulators of 128 columns
static constexpr int SP_EPI_WARP0 = 2;
static constexpr int SP_GROUPS = 4;           // epilogue warps per TMEM lane quadrant, a quarter of the pooled columns each
static constexpr int SP_EPI_WARPS = 4 * SP_GROUPS;
static constexpr int SP_ISSUERS = 2;           // MMA-issuing warps (warp 1 and the last one): row pairs alternate between them
static constexpr int SP_WRITERS = 4;           // warps that re-lay the image where it does not come re-laid (warp 0 and the last three)
static constexpr int SP_THREADS = 32 * (SP_EPI_WARP0 + SP_EPI_WARPS + SP_ISSUERS - 1);
static constexpr int SP_THREADS_RAW = SP_THREADS + 32 * (SP_WRITERS - 1);
static constexpr int SP_RING = 16;            // pairs of re-laid image rows in flight (a power of two)
static constexpr int SP_CHANNELS = 64;

struct StemPoolArgs {
    int items, bands, P;    // bands of P pooled rows
    int poH, poW;
    int KH, KWp;            // filter rows and (even) filter columns after space-to-depth
    int Wp;                 // pixels per row of the re-laid image
    int n_base;             // first image of this call within the re-laid buffer
    const uint8_t* raw;     // RAW: the image itself, three channels, rows of whole words
    int H, W, shift;        // RAW: its size; what the re-laid image is moved by (even)
    int groups_per_row;     // RAW: groups of four input pixels behind a row of the re-laid image
    int chunk_alloc;        // bytes between ring slots
    int w_bytes;
    unsigned idesc;
    const int8_t* w;
    uint8_t* out;
    int* status;
    const int* fq;
    int cpad;
    int out_lo, out_hi;
};

__device__ __forceinline__ unsigned sp_desc_lo(unsigned addr, unsigned k_step) { return ((addr & 0x3ffffu) >> 4) | ((k_step >> 4) << 16); }
__device__ __forceinline__ unsigned sp_desc_hi(unsigned row_group_step) { return (row_group_step >> 4) | (1u << 14); }

__device__ __forceinline__ void sp_mma(unsigned d_tmem, unsigned a_lo, unsigned a_hi, unsigned b_lo, unsigned b_hi, unsigned idesc, unsigned accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %5, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}

// The MMAs of a row pair; the filter extents are constants where they can be (a 7x7 and a 3x3 filter): with run-time loops the
// issuing lane spent 220 cycles on each MMA of 56, computing and moving its operands
template <int KH, int KP>
__device__ __forceinline__ void sp_issue_pair(unsigned d, const unsigned (&x)[5], unsigned Wp, unsigned x_hi, unsigned w_lo, unsigned w_hi,
                                              unsigned idesc)
{
#pragma unroll
    for (int ky = 0; ky <= KH; ++ky)
#pragma unroll
        for (int j = 0; j < KP; ++j)
            sp_mma(d, w_lo + (unsigned)(ky * 128 * 2 * KP + 16 * j), w_hi, x[ky >> 1] + ((ky & 1) ? Wp : 0u) + 2u * j, x_hi, idesc, (ky | j) ? 1u : 0u);
}

__device__ __forceinline__ unsigned sp_pack2(int y0, int y1, bool out_unsigned)
{
    unsigned w;
    if (out_unsigned) asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(y1), "r"(y0), "r"(0));
    else asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(y1), "r"(y0), "r"(0));
    return w;
}

// HP: pooled columns per lane and row (eight times as many per row and CTA)
// SHAPE: 1 = 4 x 4 filter after space-to-depth (a 7x7/2 or 8x8/2 filter), 2 = 2 x 2 (a 3x3/2 filter), 0 = any
// RAW: the image comes as it is, [H][W][3] bytes; four warps write the re-laid rows into the ring.  A lane takes four adjacent pixels of
// two image rows, 12 bytes of each as words, and writes the two 16-byte pixels they make (the separate re-layout wrote and read
// 216 KB per 224 x 224 image; conv1 + pool1 of ResNet-50 at 1024 images went from 300 us to 270)
template <int HP, int SHAPE, bool CLAMP, int FORM, bool RAW>
__global__ void __launch_bounds__(RAW ? SP_THREADS_RAW : SP_THREADS, 1)
stem_pool_tcgen05_kernel(const __grid_constant__ CUtensorMap tmX, const StemPoolArgs a)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* ring = smem + (((size_t)a.w_bytes + 1023) & ~(size_t)1023);
    // a row's last positions, rounded up to 16, read up to 256 bytes past its slot: values nobody uses
    unsigned long long* bars = (unsigned long long*)(ring + (size_t)SP_RING * a.chunk_alloc + 1024);
    const unsigned full0 = smem_u32(bars), empty0 = full0 + 8u * SP_RING;
    const unsigned tfull0 = empty0 + 8u * SP_RING, tempty0 = tfull0 + 8u * SP_SLOTS, wfull = tempty0 + 8u * SP_SLOTS;
    unsigned* tmem_slot = (unsigned*)(bars + 2 * SP_RING + 2 * SP_SLOTS + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    pdl_launch_dependents();
    if (warp == 0) {
        for (int i = lane; i < 2 * SP_RING + 2 * SP_SLOTS + 1; i += 32)
            mbar_init(full0 + 8u * i, i >= SP_RING && i < 2 * SP_RING ? SP_ISSUERS
                                                                      : (i >= 2 * SP_RING + SP_SLOTS && i < 2 * SP_RING + 2 * SP_SLOTS ? SP_EPI_WARPS : 1));
        if (lane == 0) {
            *abort_flag = 0;
            prefetch_tensor_map(&tmX);
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
    const unsigned tmem_base = *tmem_slot;
    const int ahead = a.KH / 2;   // row pair q reads ring chunks q .. q + ahead
    auto band_rows = [&](int band) { return min(a.P, a.poH - band * a.P); };
    const int step_n = (int)gridDim.x / a.bands, step_b = (int)gridDim.x - step_n * a.bands;
    const int n_first = (int)blockIdx.x / a.bands, band_first = (int)blockIdx.x - n_first * a.bands;

    constexpr int WRITER1 = SP_EPI_WARP0 + SP_EPI_WARPS + SP_ISSUERS - 1;   // the second of the RAW form's writers
    if (warp == 0 || (RAW && warp >= WRITER1)) {
        // ------------------------------------------------------------------ TMA producer, or writers: pairs of image rows
        if (warp == 0 && elect_one()) {
            mbar_expect_tx(wfull, (unsigned)a.w_bytes);
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(smem_u32(smem)), "l"(a.w), "r"((unsigned)a.w_bytes), "r"(wfull) : "memory");
        }
        __syncwarp();
        pdl_wait();   // weights are constants; the re-laid image is the previous kernel's output
        const unsigned bytes = (unsigned)(2 * a.Wp * 16), ring_s = smem_u32(ring);
        unsigned seq = 0;
        bool ok = true;
        int n = n_first, band = band_first;
        const unsigned me = warp == 0 ? 0u : (unsigned)(warp - WRITER1 + 1);
        constexpr int GROUPS = 5;   // per lane: two rows of at most 65 groups
        for (int item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
            const int chunks = band_rows(band) + 1 + ahead, row0 = 2 * band * a.P;
            for (int c = 0; c < chunks; ++c, ++seq) {
                if (RAW) {
                    if (seq % SP_WRITERS != me) continue;
                    // all loads of the chunk are on their way before the slot is waited for
                    unsigned w[GROUPS][2][3];
                    const unsigned row_words = (unsigned)a.W * 3u / 4u;
#pragma unroll
                    for (int k = 0; k < GROUPS; ++k) {
                        const int t = lane + 32 * k, r = t >= a.groups_per_row ? 1 : 0, x0 = 4 * (t - r * a.groups_per_row) - (a.shift + 3) / 4 * 4;
#pragma unroll
                        for (int dy = 0; dy < 2; ++dy) {
                            const int y = 2 * (row0 + 2 * c + r) + dy - a.shift;
                            const bool in = t < 2 * a.groups_per_row && (unsigned)y < (unsigned)a.H && (unsigned)x0 < (unsigned)a.W;
                            const unsigned* p = (const unsigned*)a.raw + (size_t)(unsigned)(n * a.H + y) * row_words + (unsigned)x0 * 3u / 4u;
#pragma unroll
                            for (int j = 0; j < 3; ++j) w[k][dy][j] = in ? __ldg(p + j) : 0u;
                        }
                    }
                    const unsigned slot = seq & (SP_RING - 1), ph = (seq / SP_RING) & 1u;
                    if (!mbar_wait_issuer(empty0 + 8u * slot, ph ^ 1u, abort_flag, a.status, 1)) { ok = false; break; }
#pragma unroll
                    for (int k = 0; k < GROUPS; ++k) {
                        const int t = lane + 32 * k, r = t >= a.groups_per_row ? 1 : 0, x0 = 4 * (t - r * a.groups_per_row) - (a.shift + 3) / 4 * 4;
                        const int X = (x0 + a.shift) / 2;   // first of the two pixels; -1 where the shift is no multiple of four
                        if (t >= 2 * a.groups_per_row) continue;
                        unsigned px[2][4];
#pragma unroll
                        for (int dy = 0; dy < 2; ++dy) {
                            const unsigned* v = w[k][dy];
                            px[dy][0] = v[0] & 0xffffffu;
                            px[dy][1] = __byte_perm(v[0], v[1], 0x0543) & 0xffffffu;
                            px[dy][2] = __byte_perm(v[1], v[2], 0x0432) & 0xffffffu;
                            px[dy][3] = v[2] >> 8;
                        }
                        uint4* o = (uint4*)(ring + (size_t)slot * a.chunk_alloc) + r * a.Wp + X;
                        if (X >= 0 && X < a.Wp) o[0] = make_uint4(px[0][0], px[0][1], px[1][0], px[1][1]);
                        if (X + 1 < a.Wp) o[1] = make_uint4(px[0][2], px[0][3], px[1][2], px[1][3]);
                    }
                    fence_async_smem();   // generic stores, read by the tensor core through the async proxy
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full0 + 8u * slot);
                    continue;
                }
                const unsigned slot = seq & (SP_RING - 1), ph = (seq / SP_RING) & 1u;
                if (!mbar_wait_issuer(empty0 + 8u * slot, ph ^ 1u, abort_flag, a.status, 1)) { ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(full0 + 8u * slot, bytes);
                    tma_load_3d(ring_s + slot * (unsigned)a.chunk_alloc, &tmX, full0 + 8u * slot, 0, row0 + 2 * c, a.n_base + n);   // rows below the image arrive as zeros
                }
                __syncwarp();
            }
            n += step_n;
            band += step_b;
            if (band >= a.bands) { band -= a.bands; ++n; }
        }
    } else if (warp == 1 || warp == SP_EPI_WARP0 + SP_EPI_WARPS) {
        // ------------------------------------------------------------------ MMA issuers
        // One alone took 1030 cycles per row pair, its waits and commits on top of the 620 the tensor pipe is busy
        const unsigned me = warp == 1 ? 0u : 1u;
        bool ok = (int)blockIdx.x >= a.items || mbar_wait_issuer(wfull, 0, abort_flag, a.status, 8);
        // weights per filter row: [m / 8][k / 16][m % 8][16 bytes]; positions: 16-byte rows, the next 16 bytes of K one pixel on
        const unsigned w_hi = sp_desc_hi((unsigned)(a.KWp * 128)), x_hi = sp_desc_hi(128u);
        const unsigned w_lo0 = sp_desc_lo(smem_u32(smem), 128u), x_lo0 = sp_desc_lo(smem_u32(ring), 16u);
        const unsigned w_row = (unsigned)((128 * a.KWp * 16) >> 4), chunk16 = (unsigned)(a.chunk_alloc >> 4);
        unsigned seq = 0, acc = 0, have = 0;   // first chunk of the row pair; accumulators used; chunks known to be there
        int band = band_first;
        for (int item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
            const int pairs = band_rows(band) + 1;
            for (int q = 0; q < pairs; ++q, ++seq, ++acc) {
                if ((acc & 1u) != me) continue;
                const unsigned slot = acc & (SP_SLOTS - 1), sph = (acc / SP_SLOTS) & 1u;
                if (!mbar_wait_issuer(tempty0 + 8u * slot, sph ^ 1u, abort_flag, a.status, 2)) { ok = false; break; }
                for (; ok && have <= seq + (unsigned)ahead; ++have)
                    ok = mbar_wait_issuer(full0 + 8u * (have & (SP_RING - 1)), (have / SP_RING) & 1u, abort_flag, a.status, 3);
                if (!ok) break;
                tc_fence_after();
                unsigned x[5];   // ring chunks of the pair
#pragma unroll
                for (int i = 0; i < (SHAPE == 1 ? 3 : (SHAPE == 2 ? 2 : 5)); ++i) x[i] = x_lo0 + ((seq + (unsigned)i) & (SP_RING - 1)) * chunk16;
                const unsigned d = tmem_base + slot * 128u;
                if (elect_one()) {
                    if (SHAPE == 1) sp_issue_pair<4, 2>(d, x, (unsigned)a.Wp, x_hi, w_lo0, w_hi, a.idesc);
                    else if (SHAPE == 2) sp_issue_pair<2, 1>(d, x, (unsigned)a.Wp, x_hi, w_lo0, w_hi, a.idesc);
                    else
                        for (int ky = 0; ky <= a.KH; ++ky) {
                            const unsigned xr = x_lo0 + ((seq + (unsigned)(ky >> 1)) & (SP_RING - 1)) * chunk16 + (unsigned)((ky & 1) * a.Wp);
                            for (int j = 0; 2 * j < a.KWp; ++j)
                                sp_mma(d, w_lo0 + (unsigned)ky * w_row + 16u * j, w_hi, xr + 2u * j, x_hi, a.idesc, (ky | j) ? 1u : 0u);
                        }
                    tc_commit(tfull0 + 8u * slot);
                    // This issuer is done with chunks q and q + 1 (its next pair is q + 2), after its last pair of the band with all of
                    // them.  A chunk is free when both issuers are; chunk 0 only has this one.
                    const int last = q >= pairs - 2 ? pairs - 1 + ahead : q + 1;
                    if (q == 0) tc_commit(empty0 + 8u * (seq & (SP_RING - 1)));
                    for (int i = q; i <= last; ++i) tc_commit(empty0 + 8u * ((seq + (unsigned)(i - q)) & (SP_RING - 1)));
                }
                __syncwarp();
            }
            seq += (unsigned)ahead;   // the next band starts behind this one's last rows
            band += step_b;
            if (band >= a.bands) band -= a.bands;
        }
    } else {
        // ------------------------------------------------------------------ epilogue warps
        const int quad = warp & 3, group = (warp - SP_EPI_WARP0) >> 2;
        const int ch = quad * 16 + (lane & 15);
        const bool second = lane >= 16;         // the pair's second convolution row; finishes the right half of the columns
        const int lo = __ldg(a.fq + 0 * a.cpad + ch), hi = __ldg(a.fq + 1 * a.cpad + ch), mu = __ldg(a.fq + 2 * a.cpad + ch);
        const int ad = __ldg(a.fq + 3 * a.cpad + ch), sh = __ldg(a.fq + 4 * a.cpad + ch);
        const int pos0 = group * 2 * HP + (second ? HP : 0);   // this lane's first pooled column
        const int valid = min(HP, a.poW - pos0);               // and how many of its columns exist
        const unsigned lane_base = tmem_base + ((unsigned)(quad * 32) << 16);
        const unsigned col0 = (unsigned)(group * 4 * HP);      // first convolution column of the warp, 4 HP + 1 in all
        const unsigned col_last = min(col0 + 32u, 127u);       // HP = 8: the 33rd (rows of 64 pooled columns do not occur)
        pdl_wait();   // the output buffer may still be read by the previous kernel
        unsigned acc = 0;
        bool ok = true;
        int n = n_first, band = band_first;
        for (int item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
            const int rows = band_rows(band);
            uint8_t* o = a.out + (((size_t)n * a.poH + band * a.P) * a.poW + pos0) * SP_CHANNELS + ch;
            int best[HP];
#pragma unroll
            for (int i = 0; i < HP; ++i) best[i] = 0;
            for (int q = 0; q <= rows; ++q, ++acc) {
                const unsigned slot = acc & (SP_SLOTS - 1), sph = (acc / SP_SLOTS) & 1u;
                if (!mbar_wait_warp(tfull0 + 8u * slot, sph, abort_flag, a.status, 4)) { ok = false; break; }
                tc_fence_after();
                unsigned v[33];
                const unsigned t = lane_base + slot * 128u;
                tc_ld32(t + col0, v);
                if (HP == 8) asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v[32]) : "r"(t + col_last) : "memory");
                tc_wait_ld_into(v);
                if (HP == 8) asm volatile("" : "+r"(v[32])::"memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty0 + 8u * slot);
                int y[HP + 1];
#pragma unroll
                for (int i = 0; i < HP; ++i) {
                    // maxima of three columns: pooled columns i (left half) and i + HP (right half) of this lane's row
                    const int l = max(max((int)v[2 * i], (int)v[2 * i + 1]), (int)v[2 * i + 2]);
                    const int r2 = i + 1 == HP ? (int)v[HP == 8 ? 32 : 4 * HP] : (int)v[2 * (i + HP) + 2];
                    const int r = max(max((int)v[2 * (i + HP)], (int)v[2 * (i + HP) + 1]), r2);
                    const int own = second ? r : l;
                    const int other = __shfl_xor_sync(0xffffffffu, second ? l : r, 16);
                    const int first_row = second ? other : own;
                    y[i] = rescale<CLAMP, FORM>(max(best[i], first_row), lo, hi, mu, ad, sh);
                    best[i] = max(own, other);
                }
                if (q > 0) {
                    y[HP] = 0;
#pragma unroll
                    for (int i = 0; i < HP; i += 2) {
                        const unsigned w = sp_pack2(y[i], y[i + 1], a.out_hi > 127);
                        if (i < valid) o[(size_t)i * SP_CHANNELS] = (uint8_t)w;
                        if (i + 1 < valid) o[(size_t)(i + 1) * SP_CHANNELS] = (uint8_t)(w >> 8);
                    }
                    o += (size_t)a.poW * SP_CHANNELS;
                }
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
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// The kernels of a form, by [the image as it is][filter shape][pooled columns per lane].  Each form of the rescale is an object of its own
// (stem_pool_int.cu, stem_pool_float.cu, stem_pool_wide.cu): loading one takes time by its size, and a process rarely uses two.
typedef void (*StemPoolKernel)(const CUtensorMap, const StemPoolArgs);
extern const StemPoolKernel stem_pool_int[2][3][4], stem_pool_int_clamped[2][3][4], stem_pool_float[2][3][4], stem_pool_float_clamped[2][3][4],
    stem_pool_wide[2][3][4], stem_pool_wide_clamped[2][3][4];
#define N2D2B_SP0(S, C, F, R) {stem_pool_tcgen05_kernel<4, S, C, F, R>, stem_pool_tcgen05_kernel<6, S, C, F, R>, \
                               stem_pool_tcgen05_kernel<7, S, C, F, R>, stem_pool_tcgen05_kernel<8, S, C, F, R>}
#define N2D2B_SP1(C, F, R) {N2D2B_SP0(0, C, F, R), N2D2B_SP0(1, C, F, R), N2D2B_SP0(2, C, F, R)}
#define N2D2B_STEM_POOL_KERNELS(C, F) {N2D2B_SP1(C, F, false), N2D2B_SP1(C, F, true)}

}  // namespace n2d2b
