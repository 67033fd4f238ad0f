// Depthwise 3x3 layer and the 1x1 layer behind it as one kernel: what the depthwise part computes goes through shared memory into the
// tensor cores and never to HBM.
//
//   A[P x C] (u8) = rescale(depthwise 3x3 of the input)     CUDA cores, byte dot products
//   D[P x N] (s32, TMEM) = A * B[N x C]^T (s8)              tcgen05.mma kind::i8
//   out = rescale(D)                                        epilogue warps, straight to NHWC
//
// A CTA takes a run of output row segments (a segment is a whole output row, or an equal part of one wider than 126 pixels) and
// works them off in tiles of up to 128 pixels; tiles of few channels go in blocks of several that share a patch and its barriers.  Per K block
// of BK = 128 (64, 32) channels a patch of input rows arrives by TMA (the unit zero-fills the border); a warp walks along a segment, a lane
// owns four channels.  Of every input column it reads three words and transposes them once to one word per channel of three rows, which
// serves three output pixels: three byte dot products, about 1.5 permutes and 0.75 loads per output.  The requantised word goes into the
// swizzled K-major operand tile.  One warp issues the MMAs over all column blocks of the CTA (the operand tile stays until the last of them),
// eight or twelve warps drain the accumulators beside the twelve or eight that fill the operand.  Rows of a tile beyond its pixels hold
// whatever is there: their sums are not stored.
//
// What bounds it: up to 256 channels instructions (63 to 73 % of the issue slots; per 32 depthwise outputs 18 with as many 1x1 outputs behind them, 31 with
// twice as many, their waits included); from 512 outputs on the waits for operand slots, which a tile of two passes hands back in the second (45 to 55 %).
// The same twenty warps doing both kinds of work in turn were slower (MobileNet at 256 images 814 us against 685): every wait then stalls both.
// As two kernels the depthwise output crosses L2 or HBM twice, and the pair costs two hand-overs between kernels of 1.3 to 2 us each:
// 14 x 14 x 512 at 256 images 46 us as two launches by themselves, 33 as one.
#pragma once
#include "kernels.h"
#include "tc_common.cuh"

namespace n2d2b {

static constexpr int DP_BOX_N = 64;           // weight rows per TMA box
static constexpr int DP_WARP0 = 4, DP_WARPS = 20;   // the warps of the epilogue, then those of the depthwise part
static constexpr int DP_THREADS = 32 * (DP_WARP0 + DP_WARPS);
static constexpr int DP_MAX_PATCH = 4, DP_MAX_A = 16, DP_MAX_B = 8, DP_MAX_ACC = 4;
// patch_full, a_full, a_empty, b_full, b_empty, tmem_full, tmem_empty, resident weights, constants, depthwise constants
static constexpr int DP_BARS = DP_MAX_PATCH + 2 * DP_MAX_A + 2 * DP_MAX_B + 2 * DP_MAX_ACC + 3;
static constexpr int DP_PARAM_BYTES = FAST_NP * 256 * 4;   // the 1x1 layer's constants of one column block

// How the constants of a cell are applied
// (DPF_UNIT: 32-bit without clamps, every multiplier 1 - a single shift: the addend then starts the dot product)
static constexpr int DPF_INT = 0, DPF_CLAMP = 1, DPF_WIDE = 2, DPF_UNIT = 3;
__host__ __device__ constexpr bool dpf_clamp(int f) { return f == DPF_CLAMP; }
// rows of the five of a FastQuant that the form reads
__host__ __device__ constexpr int dpf_rows(int f)
{
    return f == DPF_INT ? 0x1c : (f == DPF_CLAMP ? 0x1f : (f == DPF_WIDE ? 0x1d : 0x18));
}
__host__ __device__ constexpr int dpf_ef(int f) { return f == DPF_WIDE ? EF_WIDE : 0; }

struct DwPwArgs {
    int C, N, kchunks, oH, oW, pT, pL;
    int seg, segs_per_row;       // output pixels of a segment, segments per output row
    int rt;                      // segments of a full tile
    int subs;                    // tiles of a block: they share patches and barriers
    unsigned rcp_rt;             // (i * rcp_rt) >> 16 = i / rt
    int unit0, units;            // segments of this call
    int groups, nsplit;          // CTAs = groups of units x column ranges
    int bn, passes;              // columns per accumulator, accumulators per tile
    int acc_shift, epi_warps, epi_groups;
    int item, parts;             // output pixels of a work item, work items per segment
    unsigned rcp_parts;          // (i * rcp_parts) >> 16 = i / parts
    int pitch, patch_bytes, np;  // bytes of a patch row, of a slot; slots
    int a_sub, a_bytes, na;      // bytes of a tile's operand block (BK x pixels rounded up to 8 rows), of a slot (all tiles of a block); slots
    int b_bytes, nb;             // bytes of a weight slot (bn x BK); slots (0: resident)
    unsigned idesc, tmem_cols;
    const int4* dw_w;            // [3][C / 4]: per channel the bytes w(0, kx), w(1, kx), w(2, kx), 0
    const int* dw_fq;
    int dw_cpad;
    int dw_shared;               // the depthwise layer's weights and constants are copied to shared memory first (else read where they are)
    const int* fq;
    int cpad, out_unsigned;
    uint8_t* out;
    int* status;
};

// Three rows of four channels -> one word per channel (byte 3 is not used: its weight is zero)
__device__ __forceinline__ void dp_turn(const unsigned (&r)[3], unsigned (&x)[4])
{
    const unsigned a = __byte_perm(r[0], r[1], 0x5140), b = __byte_perm(r[0], r[1], 0x7362);
    x[0] = __byte_perm(a, r[2], 0x4410);
    x[1] = __byte_perm(a, r[2], 0x5532);
    x[2] = __byte_perm(b, r[2], 0x6610);
    x[3] = __byte_perm(b, r[2], 0x7732);
}

__device__ __forceinline__ int dp_dot(unsigned x, int w, int acc)
{
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(x), "r"(w), "r"(acc));
    return d;
}

// The constants of a lane's four channels
struct DpConsts {
    int w[3][4];
    int lo[4], hi[4], mu[4], ad[4], sh[4];
};

// One work item of a lane: `n` output pixels (all lanes of the warp alike), of which the first `keep` are stored.
// pa: byte offset in dynamic shared memory of the lane's word in the item's first input column; pb: shared-memory address of its byte column in
// the item's first row of the operand tile, before the swizzle (which goes by address bits)
template <int BK, int S, int F>
__device__ __forceinline__ void dp_item(unsigned pa, unsigned pitch, unsigned pb, int n, int keep, const DpConsts& k)
{
    unsigned char* const sm = dyn_smem();
    constexpr unsigned XM = (unsigned)(BK / 16 - 1) << 4;
    unsigned pr1 = pa + pitch, pr2 = pr1 + pitch;
    auto load = [&](unsigned (&r)[3], int col) {
        r[0] = *(const unsigned*)(sm + pa + col * BK);
        r[1] = *(const unsigned*)(sm + pr1 + col * BK);
        r[2] = *(const unsigned*)(sm + pr2 + col * BK);
    };
    auto step = [&](int cols) { pa += cols * BK; pr1 += cols * BK; pr2 += cols * BK; };
    auto emit = [&](const unsigned (&x0)[4], const unsigned (&x1)[4], const unsigned (&x2)[4]) {
        int y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int d = dp_dot(x2[j], k.w[2][j], dp_dot(x1[j], k.w[1][j], dp_dot(x0[j], k.w[0][j], F == DPF_UNIT ? k.ad[j] : 0)));
            y[j] = F == DPF_UNIT ? d >> k.sh[j] : rescale<dpf_clamp(F), dpf_ef(F)>(d, k.lo[j], k.hi[j], k.mu[j], k.ad[j], k.sh[j]);
        }
        const unsigned v = pack4_sat(y[0], y[1], y[2], y[3], true);
        // (one lane group per warp: every pixel of the item is stored)
        if (BK == 128 || keep > 0) asm volatile("st.shared.b32 [%0], %1;" ::"r"(pb ^ ((pb >> 3) & XM)), "r"(v));
        if (BK != 128) --keep;
        pb += BK;
    };
    if (S == 1) {
        unsigned r[3], x0[4], x1[4], x2[4];
        load(r, 0);
        dp_turn(r, x0);
        load(r, 1);
        dp_turn(r, x1);
        load(r, 2);
        // (whole groups of three without a test between: the words change roles, not registers)
        for (; n >= 3; n -= 3) {
            dp_turn(r, x2);
            load(r, 3);
            emit(x0, x1, x2);
            dp_turn(r, x0);
            load(r, 4);
            emit(x1, x2, x0);
            dp_turn(r, x1);
            load(r, 5);
            emit(x2, x0, x1);
            step(3);
        }
        if (n > 0) {
            dp_turn(r, x2);
            load(r, 3);
            emit(x0, x1, x2);
            if (n > 1) {
                dp_turn(r, x0);
                emit(x1, x2, x0);
            }
        }
    } else {
        unsigned r0[3], r1[3], x0[4], x1[4], x2[4];
        load(r0, 0);
        dp_turn(r0, x0);
        load(r0, 1);
        load(r1, 2);
        for (; n >= 2; n -= 2) {
            dp_turn(r0, x1);
            dp_turn(r1, x2);
            load(r0, 3);
            load(r1, 4);
            emit(x0, x1, x2);
            dp_turn(r0, x1);
            dp_turn(r1, x0);
            load(r0, 5);
            load(r1, 6);
            emit(x2, x1, x0);
            step(4);
        }
        if (n > 0) {
            dp_turn(r0, x1);
            dp_turn(r1, x2);
            emit(x0, x1, x2);
        }
    }
}

// Bounded wait of a working warp: it sleeps between polls, which would take a tenth of the issue slots from the warps that work
__device__ __forceinline__ bool dp_wait(unsigned bar, unsigned parity, volatile int* abort_flag, int* status, int code)
{
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    const unsigned long long t0 = globaltimer_ns();
    while (true) {
#pragma unroll 1
        for (int i = 0; i < 16; ++i) {
            __nanosleep(100);
            if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
        }
        if (__any_sync(0xffffffffu, *abort_flag != 0)) return false;
        if (__any_sync(0xffffffffu, globaltimer_ns() - t0 > WAIT_LIMIT_NS)) {
            *abort_flag = 1;
            atomicCAS(status, 0, code);
            return false;
        }
    }
}

// The blocks of a CTA in turn: where the one at hand lies, walked without divisions
struct DpBlock {
    int u, end;            // first unit, end of the CTA's range
    int img, y, part;      // image, output row, segment of the row
    int nseg;
    __device__ __forceinline__ void start(const DwPwArgs& a, int u_begin, int u_end)
    {
        u = u_begin;
        end = u_end;
        const int row = u / a.segs_per_row;
        part = u - row * a.segs_per_row;
        img = row / a.oH;
        y = row - img * a.oH;
        nseg = min(a.rt * a.subs, end - u);
    }
    __device__ __forceinline__ bool valid() const { return nseg > 0; }
    __device__ __forceinline__ void next(const DwPwArgs& a)
    {
        u += nseg;
        if (a.segs_per_row == 1) y += nseg;
        else if (++part == a.segs_per_row) { part = 0; ++y; }   // (one segment a block)
        while (y >= a.oH) { y -= a.oH; ++img; }
        nseg = min(a.rt * a.subs, end - u);
    }
    __device__ __forceinline__ int cols(const DwPwArgs& a) const { return a.segs_per_row == 1 ? a.oW : min(a.seg, a.oW - part * a.seg); }   // of a segment
};

template <int S, int DWF, int PWF>
__global__ void __launch_bounds__(DP_THREADS, 1)
dwpw_i8_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const DwPwArgs a, int bk)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    // weights, operand slots (an MMA reads 128 rows from the start of any of them: patches follow), patches, constants, barriers
    const int b_total = a.nb ? a.nb * a.b_bytes : a.passes * a.kchunks * a.b_bytes;
    unsigned char* const a_smem = smem + b_total;
    unsigned char* const p_smem = a_smem + a.na * a.a_bytes;
    int* const par = (int*)(p_smem + max(a.np * a.patch_bytes, 128 * bk));
    // weights and constants of the depthwise layer: rows of C words
    int* const dwc = par + a.passes * (DP_PARAM_BYTES / 4);
    constexpr int DW_ROWS = 3 + __builtin_popcount(dpf_rows(DWF));
    unsigned long long* const bars = (unsigned long long*)(dwc + (a.dw_shared ? DW_ROWS * a.C : 0));
    const unsigned pfull0 = smem_u32(bars), afull0 = pfull0 + 8u * DP_MAX_PATCH, aempty0 = afull0 + 8u * DP_MAX_A;
    const unsigned bfull0 = aempty0 + 8u * DP_MAX_A, bempty0 = bfull0 + 8u * DP_MAX_B;
    const unsigned tfull0 = bempty0 + 8u * DP_MAX_B, tempty0 = tfull0 + 8u * DP_MAX_ACC;
    const unsigned bres = tempty0 + 8u * DP_MAX_ACC, cready = bres + 8u, dready = cready + 8u;
    unsigned* const tmem_slot = (unsigned*)(bars + DP_BARS);
    volatile int* const abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    pdl_launch_dependents();

    if (warp == 0) {
        for (int i = lane; i < DP_BARS; i += 32) {
            unsigned n = 1;
            if (i >= DP_MAX_PATCH && i < DP_MAX_PATCH + DP_MAX_A) n = (unsigned)(DP_WARPS - a.epi_warps);                     // a_full
            else if (i >= DP_BARS - 3 - DP_MAX_ACC && i < DP_BARS - 3) n = (unsigned)(a.epi_warps / a.epi_groups);   // tmem_empty
            mbar_init(pfull0 + 8u * i, n);
        }
        if (lane == 0) {
            *abort_flag = 0;
            prefetch_tensor_map(&tmA);
            prefetch_tensor_map(&tmB);
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

    const int group = (int)blockIdx.x / a.nsplit, split = (int)blockIdx.x - group * a.nsplit;
    const int u_begin = a.unit0 + (int)((long long)a.units * group / a.groups);
    const int u_end = a.unit0 + (int)((long long)a.units * (group + 1) / a.groups);
    const int n_begin = split * a.passes * a.bn;
    bool ok = true;

    if (warp == 0) {
        // ------------------------------------------------------------------ input patches
        // The patch of a block goes out when its slot and its operand slot are both free, so the depthwise warps wait for one barrier only: the
        // slot was left when the operand block np patches back was complete (np <= na: that barrier is at most one phase further)
        pdl_wait();
        int slot = 0, aslot = 0, done_slot = 0, ahead = 0;
        unsigned aph = 1u, done_ph = 0;
        DpBlock t;
        t.start(a, u_begin, u_end);
        for (; t.valid() && ok; t.next(a)) {
            int rows = 0;
            for (int left = t.nseg, y = t.y; left > 0; y = 0) {
                const int cnt = min(left, a.oH - y);
                rows += (cnt - 1) * S + 3;
                left -= cnt;
            }
            for (int kc = 0; kc < a.kchunks; ++kc) {
                const unsigned bar = pfull0 + 8u * slot;
                if (ahead == a.np) {
                    if (!mbar_wait_issuer(afull0 + 8u * done_slot, done_ph, abort_flag, a.status, 21)) { ok = false; break; }
                    if (++done_slot == a.na) { done_slot = 0; done_ph ^= 1u; }
                } else {
                    ++ahead;
                }
                if (!mbar_wait_issuer(aempty0 + 8u * aslot, aph, abort_flag, a.status, 32)) { ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(bar, (unsigned)(rows * a.pitch));
                    unsigned dst = smem_u32(p_smem) + (unsigned)(slot * a.patch_bytes);
                    int img = t.img, y = t.y;
                    for (int left = t.nseg; left > 0; y = 0, ++img) {
                        const int cnt = min(left, a.oH - y), n = (cnt - 1) * S + 3;
                        for (int i = 0; i < n; ++i, dst += (unsigned)a.pitch)
                            tma_load_4d(dst, &tmA, bar, kc * bk, t.part * a.seg * S - a.pL, y * S - a.pT + i, img);
                        left -= cnt;
                    }
                }
                __syncwarp();
                if (++slot == a.np) slot = 0;
                if (++aslot == a.na) { aslot = 0; aph ^= 1u; }
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------------ weights: constants, so not after the previous kernel
        const int boxes = a.bn / DP_BOX_N, box_bytes = DP_BOX_N * bk;
        if (!a.nb) {
            if (u_begin < u_end && elect_one()) {
                mbar_expect_tx(bres, (unsigned)(a.passes * a.kchunks * a.b_bytes));
                unsigned dst = smem_u32(smem);
                for (int p = 0; p < a.passes; ++p)
                    for (int kc = 0; kc < a.kchunks; ++kc)
                        for (int b = 0; b < boxes; ++b, dst += (unsigned)box_bytes)
                            tma_load_2d(dst, &tmB, bres, kc * bk, n_begin + p * a.bn + b * DP_BOX_N);
            }
            __syncwarp();
        } else {
            int slot = 0;
            unsigned ph = 1u;
            for (int u = u_begin; u < u_end && ok; u += a.rt)   // (one tile a block)
                for (int p = 0; p < a.passes && ok; ++p)
                    for (int kc = 0; kc < a.kchunks; ++kc) {
                        const unsigned bar = bfull0 + 8u * slot;
                        if (!mbar_wait_issuer(bempty0 + 8u * slot, ph, abort_flag, a.status, 22)) { ok = false; break; }
                        if (elect_one()) {
                            mbar_expect_tx(bar, (unsigned)a.b_bytes);
                            unsigned dst = smem_u32(smem) + (unsigned)(slot * a.b_bytes);
                            for (int b = 0; b < boxes; ++b, dst += (unsigned)box_bytes)
                                tma_load_2d(dst, &tmB, bar, kc * bk, n_begin + p * a.bn + b * DP_BOX_N);
                        }
                        __syncwarp();
                        if (++slot == a.nb) { slot = 0; ph ^= 1u; }
                    }
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------------ constants, by the copy engine: threads that stored what they loaded
        // took 2 us of every CTA's start
        if (elect_one()) {
            if (a.dw_shared) {
                const unsigned row_bytes = 4u * (unsigned)a.C;
                mbar_expect_tx(dready, DW_ROWS * row_bytes);
                unsigned dst = smem_u32(dwc);
                bulk_load(dst, a.dw_w, 3 * row_bytes, dready);
                dst += 3 * row_bytes;
#pragma unroll
                for (int f = 0; f < FAST_NP; ++f)
                    if (dpf_rows(DWF) & (1 << f)) {
                        bulk_load(dst, a.dw_fq + f * a.dw_cpad, row_bytes, dready);
                        dst += row_bytes;
                    }
            }
            // (columns from cpad on belong to no output)
            int bytes = 0;
            for (int p = 0; p < a.passes; ++p) bytes += 4 * max(0, min(a.bn, a.cpad - (n_begin + p * a.bn)));
            mbar_expect_tx(cready, (unsigned)(__builtin_popcount(dpf_rows(PWF)) * bytes));
            for (int p = 0; p < a.passes; ++p) {
                const int n0 = n_begin + p * a.bn, cols = min(a.bn, a.cpad - n0);
                if (cols <= 0) break;
#pragma unroll
                for (int f = 0; f < FAST_NP; ++f)
                    if (dpf_rows(PWF) & (1 << f)) bulk_load(smem_u32(par) + (unsigned)(p * DP_PARAM_BYTES + f * 1024), a.fq + f * a.cpad + n0, 4u * (unsigned)cols, cready);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const unsigned desc_hi = (unsigned)(make_smem_desc(0u, bk) >> 32);
        const unsigned a_lo0 = (smem_u32(a_smem) & 0x3ffffu) >> 4, b_lo0 = (smem_u32(smem) & 0x3ffffu) >> 4;
        const unsigned a16 = (unsigned)(a.a_bytes >> 4), b16 = (unsigned)(a.b_bytes >> 4);
        int aslot0 = 0, bslot = 0;
        unsigned aph0 = 0, bph = 0, acc_it = 0;
        if (!a.nb && u_begin < u_end) ok = mbar_wait_issuer(bres, 0, abort_flag, a.status, 23);
        const int block = a.rt * a.subs;
        for (int u = u_begin; u < u_end && ok; u += block) {
            const int left = min(block, u_end - u);
            int aslot = aslot0;
            unsigned aph = aph0;
            for (int done = 0, sub = 0; done < left && ok; done += a.rt, ++sub) {
                const unsigned sub16 = (unsigned)(sub * a.a_sub) >> 4;
                const bool last_sub = done + a.rt >= left;
                for (int p = 0; p < a.passes && ok; ++p, ++acc_it) {
                    const unsigned as = acc_it & ((1u << a.acc_shift) - 1u);
                    if (!mbar_wait_issuer(tempty0 + 8u * as, ((acc_it >> a.acc_shift) & 1u) ^ 1u, abort_flag, a.status, 24)) { ok = false; break; }
                    const unsigned d_tmem = tmem_base + as * (unsigned)a.bn;
                    aslot = aslot0;
                    aph = aph0;
                    for (int kc = 0; kc < a.kchunks; ++kc) {
                        if (p == 0 && sub == 0 && !mbar_wait_issuer(afull0 + 8u * aslot, aph, abort_flag, a.status, 25)) { ok = false; break; }
                        if (a.nb && !mbar_wait_issuer(bfull0 + 8u * bslot, bph, abort_flag, a.status, 26)) { ok = false; break; }
                        tc_fence_after();
                        const unsigned al = a_lo0 + (unsigned)aslot * a16 + sub16;
                        const unsigned bl = b_lo0 + (a.nb ? (unsigned)bslot : (unsigned)(p * a.kchunks + kc)) * b16;
                        if (elect_one()) {
                            tc_mma_i8_lohi(d_tmem, al, bl, desc_hi, a.idesc, kc > 0 ? 1u : 0u);
                            if (bk >= 64) tc_mma_i8_lohi(d_tmem, al + 2u, bl + 2u, desc_hi, a.idesc, 1u);
                            if (bk == 128) {
                                tc_mma_i8_lohi(d_tmem, al + 4u, bl + 4u, desc_hi, a.idesc, 1u);
                                tc_mma_i8_lohi(d_tmem, al + 6u, bl + 6u, desc_hi, a.idesc, 1u);
                            }
                            if (a.nb) tc_commit(bempty0 + 8u * bslot);
                            if (last_sub && p + 1 == a.passes) tc_commit(aempty0 + 8u * aslot);   // no accumulator needs it any more
                            if (kc + 1 == a.kchunks) tc_commit(tfull0 + 8u * as);
                        }
                        __syncwarp();
                        if (++aslot == a.na) { aslot = 0; aph ^= 1u; }
                        if (a.nb && ++bslot == a.nb) { bslot = 0; bph ^= 1u; }
                    }
                }
            }
            aslot0 = aslot;
            aph0 = aph;
        }
    } else if (warp >= DP_WARP0 + a.epi_warps) {
        // ------------------------------------------------------------------ depthwise warps
        const int q_shift = bk == 128 ? 5 : (bk == 64 ? 4 : 3);       // lanes per pixel: four channels each
        const int q = lane & ((1 << q_shift) - 1), sub = lane >> q_shift, sub_shift = 5 - q_shift;
        const unsigned chan = 4u * (unsigned)q;
        const unsigned a_s = smem_u32(a_smem), p_off = (unsigned)(p_smem - smem_raw);
        if (a.dw_shared)
            ok = mbar_wait_warp(dready, 0, abort_flag, a.status, 31);
        DpConsts k;
        int held = -1;      // the channel block whose constants the registers hold
        int pslot = 0, aslot = 0;
        unsigned pph = 0;
        const int dw_warps = DP_WARPS - a.epi_warps;
        int mine = warp - DP_WARP0 - a.epi_warps;       // this warp's first item of the block at hand: items are dealt out across blocks
        DpBlock t;
        t.start(a, u_begin, u_end);
        for (; t.valid() && ok; t.next(a)) {
            const int items = t.nseg * a.parts, warp_items = (items + (1 << sub_shift) - 1) >> sub_shift, cols = t.cols(a);
            const int run1 = min(t.nseg, a.oH - t.y), rows1 = (run1 - 1) * S + 3, rows_image = (a.oH - 1) * S + 3;
            for (int kc = 0; kc < a.kchunks; ++kc) {
                if (mine < warp_items && held != kc) {
                    held = kc;
                    const int c0 = 4 * ((kc << q_shift) + q);
                    auto get = [&](int (&v)[4], const int* global, int row) {
                        const int4 w = a.dw_shared ? *(const int4*)(dwc + row * a.C + c0) : __ldg((const int4*)(global + c0));
                        v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w;
                    };
#pragma unroll
                    for (int kx = 0; kx < 3; ++kx) get(k.w[kx], (const int*)a.dw_w + (size_t)kx * a.C, kx);
                    int row = 3;
                    if (dpf_rows(DWF) & 1) get(k.lo, a.dw_fq, row++);
                    if (dpf_rows(DWF) & 2) get(k.hi, a.dw_fq + a.dw_cpad, row++);
                    if (dpf_rows(DWF) & 4) get(k.mu, a.dw_fq + 2 * a.dw_cpad, row++);
                    if (dpf_rows(DWF) & 8) get(k.ad, a.dw_fq + 3 * a.dw_cpad, row++);
                    if (dpf_rows(DWF) & 16) get(k.sh, a.dw_fq + 4 * a.dw_cpad, row++);
                }
                if (!dp_wait(pfull0 + 8u * pslot, pph, abort_flag, a.status, 28)) { ok = false; break; }
                for (; mine < warp_items; mine += dw_warps) {
                    const int idx = (mine << sub_shift) + sub;
                    int r = (int)(((unsigned)idx * a.rcp_parts) >> 16), x = (idx - r * a.parts) * a.item;
                    int keep = min(a.item, cols - x);
                    int row = r * S;
                    if (r >= run1) {
                        int rr = r - run1;
                        row = rows1;
                        while (rr >= a.oH) { rr -= a.oH; row += rows_image; }
                        row += rr * S;
                    }
                    if (idx >= items) { keep = 0; r = 0; x = 0; row = 0; }
                    const unsigned pa = p_off + (unsigned)(pslot * a.patch_bytes + row * a.pitch + x * S * bk) + chan;
                    const int sub_tile = (int)(((unsigned)r * a.rcp_rt) >> 16);
                    const unsigned pb = a_s + (unsigned)(aslot * a.a_bytes + sub_tile * a.a_sub + ((r - sub_tile * a.rt) * a.seg + x) * bk) + chan;
                    const int n = sub_shift ? (int)__reduce_max_sync(0xffffffffu, (unsigned)max(keep, 0)) : keep;
                    if (bk == 128) dp_item<128, S, DWF>(pa, (unsigned)a.pitch, pb, n, keep, k);
                    else if (bk == 64) dp_item<64, S, DWF>(pa, (unsigned)a.pitch, pb, n, keep, k);
                    else dp_item<32, S, DWF>(pa, (unsigned)a.pitch, pb, n, keep, k);
                }
                mine -= warp_items;
                fence_async_smem();   // generic-proxy stores, read by the tensor core through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(afull0 + 8u * aslot);
                if (++pslot == a.np) { pslot = 0; pph ^= 1u; }
                if (++aslot == a.na) aslot = 0;
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue of the 1x1 layer
        // Narrow accumulators go to groups of four warps in turn (a warp's fixed work per accumulator is that of 32 columns), wide ones to two warps
        // a quadrant
        const int quad = warp & 3, fours = (warp - DP_WARP0) >> 2;
        const int part = a.epi_groups == 1 ? fours : 0;
        int turn = a.epi_groups == 1 ? 0 : fours;      // accumulators until this warp's next one
        EpiTile e;
        e.N = a.N;
        e.wp = a.epi_groups == 1 ? a.bn / 2 : a.bn;
        const int cbase = part * e.wp;
        unsigned acc_it = 0;
        ok = mbar_wait_warp(cready, 0, abort_flag, a.status, 30);
        pdl_wait();   // the constants are nobody's output; the tensors are
        unsigned rowoff[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) rowoff[k] = (unsigned)((lane >> 2) + 8 * k) * (unsigned)a.N;
        DpBlock t;
        t.start(a, u_begin, u_end);
        for (; t.valid() && ok; t.next(a))
        for (int done = 0; done < t.nseg && ok; done += a.rt) {
            const int pixels = min(a.rt, t.nseg - done) * t.cols(a);
            // (rows of a block follow one another across images; a block of several tiles has whole rows)
            const long long pixel0 = ((long long)t.img * a.oH + t.y + done) * a.oW + t.part * a.seg;
            for (int p = 0; p < a.passes; ++p, ++acc_it) {
                if (turn-- > 0) continue;
                turn = a.epi_groups - 1;
                const int n0 = n_begin + p * a.bn;
                const unsigned as = acc_it & ((1u << a.acc_shift) - 1u);
                if (!dp_wait(tfull0 + 8u * as, (acc_it >> a.acc_shift) & 1u, abort_flag, a.status, 29)) { ok = false; break; }
                tc_fence_after();
                e.n0 = n0;
                e.par_off = (unsigned)((unsigned char*)(par + p * FAST_NP * 256) - smem_raw);
                if (quad * 32 < pixels) {
                    unsigned rowok = 0;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (quad * 32 + (lane >> 2) + 8 * k < pixels) rowok |= 1u << k;
                    uint8_t* const out = a.out + (size_t)(pixel0 + quad * 32) * a.N + n0 + cbase;
                    const unsigned tbase = tmem_base + ((unsigned)(quad * 32) << 16) + as * (unsigned)a.bn + (unsigned)cbase;
                    if (a.out_unsigned) epi_drain_direct<dpf_clamp(PWF), dpf_ef(PWF) | EF_OUT_UNSIGNED>(e, tbase, cbase, out, rowoff, rowok, lane);
                    else epi_drain_direct<dpf_clamp(PWF), dpf_ef(PWF)>(e, tbase, cbase, out, rowoff, rowok, lane);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty0 + 8u * as);
            }
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

typedef void (*DwPwKernel)(const CUtensorMap, const CUtensorMap, const DwPwArgs, int);
// [stride - 1]; the forms beside the 32-bit ones are an object of their own
extern const DwPwKernel dwpw_wide[2], dwpw_wide_1x1[2], dwpw_wide_depthwise[2];

}  // namespace n2d2b
