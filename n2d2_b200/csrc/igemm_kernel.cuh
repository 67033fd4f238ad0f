// Implicit-GEMM convolution / fully-connected kernel on the Blackwell tensor cores.
//
//   D[M x N] (int32, in TMEM) = A[M x K] (u8 or s8 activations, NHWC) * B[N x K]^T (s8 weights, OHWI)
//   M = output pixels (batch * oH * oW), N = output channels, K = taps * Cin walked tap by tap.
//
// One persistent CTA per SM loops over 128 x BN output tiles.  Three warps issue TMA loads into a
// multi-stage shared-memory ring (A tile through a 2-D tiled map for a plain GEMM, or through an
// im2col map that applies stride / padding / dilation and zero-fills the halo; B tile through a 2-D
// map, or once into a resident block when the layer's weights are small), warp 1 issues
// tcgen05.mma kind::i8 into a ring of TMEM accumulators, warps 2-17 drain the finished ones with
// tcgen05.ld and run the fused epilogue (bias, per-channel rescale, rounding, saturation, ReLU,
// optional residual add + second rescale) straight to int8 NHWC: a warp takes the 32 rows of its
// TMEM lane quadrant and 64 of the tile's columns, so narrow tiles go to the warps in groups of one tile each.  Cells on the 32-bit epilogue store their weight
// rows permuted inside blocks of 32 (16) output channels, so that the column pairs a TMEM load hands a
// thread are 8 (4) consecutive channels: constants, residual and output move as 128- and 64-bit accesses.  This replaces the reference's
// cudnnConvolutionForward + cudnnAddTensor + Scaling kernel + cudnnActivationForward sequence
// (src/Cell/ConvCell_Frame_CUDA.cpp:1169-1270) and its cublasGemm FC
// (src/Cell/FcCell_Frame_CUDA.cpp:308-427).
//
// The kernel is launched with programmatic stream serialization: barriers, TMEM, constants, tensor maps,
// resident weights and the first ring fill of streamed ones are set up while the previous kernel drains;
// activations are touched only after griddepcontrol.wait.
//
// Every wait on an mbarrier is bounded: a wait that does not complete within about a second sets
// *status_word and makes the whole CTA drain and exit, so a wrong descriptor cannot hang the GPU.
#pragma once
#include "kernels.h"
#include "tc_common.cuh"

namespace n2d2b {

static constexpr int BM = 128;
static constexpr int EPI_WARP0 = 2;
static constexpr int NUM_EPI_WARPS = 16;      // four per TMEM lane quadrant
static constexpr int MAX_ACC = 8;             // TMEM accumulators: 512 columns of 64
static constexpr int REGION_BYTES = 2048;     // staging per epilogue warp: 32 rows x up to 64 bytes
static constexpr int NUM_PRODUCERS = 3;       // warps that issue TMA loads: warp 0 and the last two of the CTA
static constexpr int NUM_THREADS = 32 * (EPI_WARP0 + NUM_EPI_WARPS + NUM_PRODUCERS - 1);
static constexpr int W4_UNPACK_WARPS = 4;     // extra warps of the packed-int4 variant

// A number of output pixels as (columns, rows, images)
struct PixelStep { int x, y, n; };

struct IgemmArgs {
    int M, N, Cin, taps, BK, BN, stages, a_im2col;
    int grouped;        // block-diagonal layer (depthwise as groups of BN channels): a column block reads its own input channels
    int res_slots;          // staging regions per epilogue warp of a residual cell (2 or 4)
    int m_base;         // first output row of this call within the tensors (a batch slice starts at image img0)
    int takers;         // producers that work (at most as many as ring slots)
    int late_weights;   // weights only after the dependency wait
    int parts, groups;  // warps per quadrant that share a tile, and tiles in the hands of the epilogue at once (parts * groups = 4)
    int acc_shift;      // log2 of the number of TMEM accumulators
    int b_resident;     // the CTA's whole weight block stays in shared memory (its column block never changes)
    int oW, oH, kW, sX, sY, pL, pT, dX, dY;
    int num_m_tiles, num_n_tiles;
    PixelStep adv_tiles, adv_one;   // the step in m (step_m tiles or tile pairs) and one 128-row tile, in pixel coordinates
    int step_m, step_n;   // gridDim.x / num_n_tiles and gridDim.x % num_n_tiles: one persistent-loop step in tile coordinates
    int ef;               // EF_* switches of the 32-bit epilogue
    unsigned idesc;
    unsigned tmem_cols;
    int out_dtype;
    void* out;
    int ldo;             // stores from the registers: bytes of an output row (N of them wanted)
    int* status;
    QuantDev q;
    Residual r;
    // fast 32-bit epilogue: y = (clamp(acc, lo, hi) * mult + add) >> shift, rows of cpad entries
    const int* fq;      // [FAST_NP][cpad] of the cell
    const int* fq2;     // [FAST_NP][cpad] of the fused residual sum (nullptr without one)
    int cpad;
    int t_lo, t_hi;     // saturation range of the cell's own output (before the residual add)
    int out_unsigned;   // final 8-bit range: 1 = [0,255], 0 = [-128,127]
    int dp_a_signed;    // dot-product form of the residual stage: operand signedness
};

// Position of an output pixel in its image batch, walked without divisions
struct PixelPos {
    int ox, oy, n;
    __device__ __forceinline__ void start(const IgemmArgs& a, int m)
    {
        const int t = m / a.oW;
        ox = m - t * a.oW;
        n = t / a.oH;
        oy = t - n * a.oH;
    }
    __device__ __forceinline__ void advance(const IgemmArgs& a, const PixelStep& d)
    {
        ox += d.x;
        oy += d.y;
        n += d.n;
        if (ox >= a.oW) { ox -= a.oW; ++oy; }
        if (oy >= a.oH) { oy -= a.oH; ++n; }
    }
};

// ----------------------------------------------------------------------------- the kernel
// Eight packed 4-bit weights (one 32-bit word: byte i = elements 2i in the high and 2i + 1 in the low nibble) as
// eight signed bytes holding 16 x the weight: the nibble moves to the top of its byte, which is the value times 16
// with the right sign and needs no sign extension.  The accumulator then holds 16 x the sum, a multiple of 16: the
// epilogue shifts it right by four first, which is exact.
__device__ __forceinline__ void expand_int4_x16(unsigned x, unsigned& w0, unsigned& w1)
{
    const unsigned hi = x & 0xF0F0F0F0u, lo = (x << 4) & 0xF0F0F0F0u;
    w0 = __byte_perm(hi, lo, 0x5140);   // hi.b0, lo.b0, hi.b1, lo.b1
    w1 = __byte_perm(hi, lo, 0x7362);   // hi.b2, lo.b2, hi.b3, lo.b3
}

// W4: the weights sit in HBM as packed 4-bit values.  The producer's TMA load brings a BN x BK/2-byte packed block
// into the stage beside the operand tiles; four extra warps expand it into the swizzled int8 B tile the MMA reads
// (as 16 x the weight, see expand_int4_x16) and signal the issuing thread through one more barrier per stage.
// DRY: a short launch (up to two tiles per CTA) spends a microsecond per role on instruction-cache misses once its data is
// there, so its issuer and epilogue warps run through their loop bodies once, without effect, while the previous kernel
// still works.  A variant of its own: the flag tests cost the epilogue of long launches 2-3 % (conv2.x of ResNet-50 at 1024 images
// with the residual sum 418 us against 403).
template <int MODE, bool W4, bool DRY>
__global__ void __launch_bounds__(W4 ? NUM_THREADS + 32 * W4_UNPACK_WARPS : NUM_THREADS, 1)
igemm_i8_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                        const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmR,
                        const IgemmArgs a)
{
    constexpr bool FAST = MODE != 0;
    constexpr bool RES = (MODE == 2 || MODE == 4 || MODE == 5);
    constexpr bool CLAMP = (MODE == 1 || MODE == 2);
    constexpr bool DP = (MODE == 5);
    extern __shared__ unsigned char smem_raw[];
    // 1024-byte alignment of the tile ring (required by the 128-byte swizzle)
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int a_stage_bytes = BM * a.BK;
    const int b_stage_bytes = a.BN * a.BK;
    const int p_stage_bytes = W4 ? b_stage_bytes / 2 : 0;                       // packed weights of the stage
    const int stage_bytes = a_stage_bytes + (a.b_resident ? 0 : b_stage_bytes) + p_stage_bytes;
    const int tx_bytes = a_stage_bytes + (W4 ? p_stage_bytes : (a.b_resident ? 0 : b_stage_bytes));   // what TMA delivers per stage
    const int kchunks = (a.Cin + a.BK - 1) / a.BK;
    const int num_kb = a.taps * kchunks;
    // resident weights first (one BN x BK block per K block), then the ring of activation (and weight) stages
    unsigned char* res_b = smem;
    unsigned char* tiles = smem + (a.b_resident ? (size_t)num_kb * b_stage_bytes : 0);
    unsigned char* stage_out = tiles + (size_t)a.stages * stage_bytes;
    // output staging: one region per epilogue warp (32 rows x up to 64 bytes, swizzled for TMA)
    // cells with a fused residual keep two or four regions per warp so that the residual of the next tiles arrives early
    const int regions_per_warp = RES ? a.res_slots : 1;
    unsigned long long* bars = (unsigned long long*)(stage_out + NUM_EPI_WARPS * REGION_BYTES * regions_per_warp);
    // bars: full[stages], empty[stages], tmem_full[8], tmem_empty[8], params_ready[2], residual[4 * NUM_EPI_WARPS],
    //       resident weights, dry run
    const unsigned full0 = smem_u32(bars);
    const unsigned empty0 = full0 + 8u * a.stages;
    const unsigned tfull0 = empty0 + 8u * a.stages;
    const unsigned tempty0 = tfull0 + 8u * MAX_ACC;
    const unsigned pready0 = tempty0 + 8u * MAX_ACC;
    const unsigned rbar0 = pready0 + 16u;
    const unsigned bfull = rbar0 + 8u * (4 * NUM_EPI_WARPS);
    const unsigned bready0 = bfull + 16u;                                       // W4: expanded weights of a stage are in place
    unsigned* tmem_slot = (unsigned*)(bars + 2 * a.stages + 2 * MAX_ACC + 2 + 4 * NUM_EPI_WARPS + 2 + (W4 ? a.stages : 0));
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    // [2 buffers][2 quant sets][FAST_NP][256], 16-byte aligned for vector loads
    int* epi_params = (int*)(((uintptr_t)(tmem_slot + 4) + 15) & ~(uintptr_t)15);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    // the producer this warp is, or -1
    constexpr int LAST_PRODUCERS = EPI_WARP0 + NUM_EPI_WARPS + (W4 ? W4_UNPACK_WARPS : 0);
    const int producer = warp == 0 ? 0 : (warp >= LAST_PRODUCERS ? warp - LAST_PRODUCERS + 1 : -1);
    pdl_launch_dependents();

    if (warp == 0) {
        // one barrier per lane and pass: 80 of them in turn on one thread delayed the whole CTA
        const int nb = 2 * a.stages + 2 * MAX_ACC + 2 + 4 * NUM_EPI_WARPS + 2;
        for (int i = lane; i < nb; i += 32) {
            const int j = i - (2 * a.stages + MAX_ACC);   // tmem_empty collects the warps of a tile, params_ready[2] all epilogue warps
            unsigned n = 1;
            if (j >= 0 && j < MAX_ACC) n = FAST ? 4u * a.parts : NUM_EPI_WARPS;
            else if (j >= MAX_ACC && j < MAX_ACC + 2) n = NUM_EPI_WARPS;
            else if (i == nb - 2) n = NUM_PRODUCERS;      // resident weights
            mbar_init(full0 + 8u * i, n);
        }
        if (W4 && lane < a.stages) mbar_init(bready0 + 8u * lane, W4_UNPACK_WARPS);
        if (lane == 0) {
            *abort_flag = 0;
            prefetch_tensor_map(&tmA);
            prefetch_tensor_map(&tmB);
            if (FAST) prefetch_tensor_map(&tmO);
            if (RES) prefetch_tensor_map(&tmR);
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
    const unsigned tiles_s = smem_u32(tiles), res_b_s = smem_u32(res_b);

    const int num_tiles = a.num_m_tiles * a.num_n_tiles;

    if (producer >= 0) {
        // ------------------------------------------------------------------ TMA producers
        // A ring slot costs its producer 300-500 cycles (a wait, an expect_tx, one or two loads and the counters around
        // them, in one warp's instruction latencies), a K block of the tensor pipe 200 (64 columns) to 512 (256): with
        // one producer the loads, not the bandwidth behind them, bounded every streamed layer.  Three take every third
        // ring fill each - never more producers than slots: a producer may be one phase of a slot's barrier ahead, which
        // its own previous fill guarantees as long as that lies at most a whole ring back, and two phases ahead look like
        // none to a parity wait.  Whatever does not depend on the previous kernel's output - the coordinates of the first tile, the first fill
        // of streamed weights - comes before the wait: cold parameters and divisions cost 0.7 us there.
        bool ok = true;
        const int first = (int)blockIdx.x;
        int m_tile = first / a.num_n_tiles, n_tile = first - m_tile * a.num_n_tiles;
        int m0 = a.m_base + m_tile * BM, n0 = n_tile * a.BN;
        PixelPos px;
        px.start(a, m0);
        int iw0 = px.ox * a.sX - a.pL, ih0 = px.oy * a.sY - a.pT, in0 = px.n;
        const int takers = a.takers;
        const int my_turn = producer < takers ? producer : 0x40000000;   // ring fills until this producer's first one (never, if idle)
        unsigned pre = 0;   // ring fills whose weights are issued before the wait
        if (a.late_weights) pdl_wait();
        if (first < num_tiles) {
            if (!a.b_resident) pre = (unsigned)(num_kb < a.stages ? num_kb : a.stages);
            const int nload = a.b_resident ? num_kb : (int)pre;
            if (elect_one()) {
                // resident: the launch keeps every CTA on one column block, its weights are fetched once.  Streamed: the
                // first fill of the ring needs nothing of the previous kernel either.
                int own = 0;
                if (a.b_resident) {
                    for (int i = my_turn; i < num_kb; i += takers) own += b_stage_bytes;
                    mbar_expect_tx(bfull, (unsigned)own);
                }
                int kc = 0, kcoord = 0, turn = my_turn;
                for (int i = 0; i < nload; ++i) {
                    if (turn == 0) {
                        turn = takers;
                        if (a.b_resident) {
                            tma_load_2d(res_b_s + (unsigned)(i * b_stage_bytes), &tmB, bfull, kcoord, n0);
                        } else {
                            const unsigned bar = full0 + 8u * i, dst = tiles_s + (unsigned)(i * stage_bytes + a_stage_bytes);
                            mbar_expect_tx(bar, (unsigned)tx_bytes);
                            if (W4) tma_load_2d(dst + b_stage_bytes, &tmB, bar, kcoord >> 1, n0);   // packed: two per byte
                            else tma_load_2d(dst, &tmB, bar, kcoord, n0);
                        }
                    }
                    --turn;
                    if (++kc == kchunks) {
                        kc = 0;
                        kcoord += a.Cin - (kchunks - 1) * a.BK;
                    } else {
                        kcoord += a.BK;
                    }
                }
            }
            __syncwarp();
        }
        bool waited = false;
        const bool im2col = a.a_im2col != 0, load_b = !a.b_resident;
        const unsigned ring_end = full0 + 8u * a.stages, to_empty = 8u * a.stages;
        unsigned bar = full0, dst = tiles_s, ph = 1u, it = 0;
        int turn = my_turn;    // ring fills until this producer's next one
        for (int tile = first; tile < num_tiles && ok; tile += gridDim.x) {
            int kx = 0, ky = 0, kc = 0, kcoord = 0;   // kcoord = tap * Cin + kc * BK
            const int c0 = a.grouped ? n0 : 0;
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                if (turn == 0) {
                    turn = takers;
                    if (!mbar_wait_issuer(bar + to_empty, ph, abort_flag, a.status, 1)) { ok = false; break; }
                    if (!waited) {   // weights are constants; the activations are the previous kernel's output
                        pdl_wait();
                        waited = true;
                    }
                    if (elect_one()) {
                        const bool weights = it >= pre;   // else they are on their way
                        if (weights) mbar_expect_tx(bar, (unsigned)tx_bytes);
                        if (im2col) tma_load_im2col_4d(dst, &tmA, bar, kc * a.BK + c0, iw0, ih0, in0, (unsigned short)(kx * a.dX), (unsigned short)(ky * a.dY));
                        else tma_load_2d(dst, &tmA, bar, kcoord, m0);
                        if (weights && load_b) {
                            if (W4) tma_load_2d(dst + (unsigned)(a_stage_bytes + b_stage_bytes), &tmB, bar, kcoord >> 1, n0);
                            else tma_load_2d(dst + (unsigned)a_stage_bytes, &tmB, bar, kcoord, n0);
                        }
                    }
                    __syncwarp();
                }
                --turn;
                bar += 8u;
                dst += (unsigned)stage_bytes;
                if (bar == ring_end) { bar = full0; dst = tiles_s; ph ^= 1u; }
                if (++kc == kchunks) {
                    kc = 0;
                    kcoord += a.Cin - (kchunks - 1) * a.BK;
                    if (++kx == a.kW) { kx = 0; ++ky; }
                } else {
                    kcoord += a.BK;
                }
            }
            m_tile += a.step_m;
            n_tile += a.step_n;
            px.advance(a, a.adv_tiles);
            if (n_tile >= a.num_n_tiles) { n_tile -= a.num_n_tiles; ++m_tile; px.advance(a, a.adv_one); }
            m0 = a.m_base + m_tile * BM;
            n0 = n_tile * a.BN;
            iw0 = px.ox * a.sX - a.pL;
            ih0 = px.oy * a.sY - a.pT;
            in0 = px.n;
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        unsigned acc_it = 0;
        bool ok = true;
        if (a.b_resident && (int)blockIdx.x < num_tiles) ok = mbar_wait_issuer(bfull, 0, abort_flag, a.status, 8);
        int s = 0;
        unsigned ph = 0;
        // upper descriptor word: stride between 8-row groups, version, swizzle; lower word: address / 16
        const unsigned desc_hi = (unsigned)(make_smem_desc(0u, a.BK) >> 32);
        const unsigned a_lo0 = (tiles_s & 0x3ffffu) >> 4, b_res0 = (res_b_s & 0x3ffffu) >> 4;
        const unsigned stage16 = (unsigned)(stage_bytes >> 4), a16 = (unsigned)(a_stage_bytes >> 4);
        const unsigned b16 = (unsigned)(b_stage_bytes >> 4);
        unsigned a_lo = a_lo0;
        MBAR_PEEK_DECLARE();
        bool dry = DRY;
        for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++acc_it) {
            const unsigned as = acc_it & ((1u << a.acc_shift) - 1u);
            const unsigned aph = (acc_it >> a.acc_shift) & 1u;
            if (!mbar_wait_issuer(tempty0 + 8u * as, aph ^ 1u, abort_flag, a.status, 2)) { ok = false; break; }
            const unsigned d_tmem = tmem_base + as * (unsigned)a.BN;
            unsigned b_res = b_res0;
            for (int kb = dry ? -1 : 0; kb < num_kb; ++kb) {   // -1: operands and accumulator of the first K block as they are
                if (!dry && !mbar_peeked() && !mbar_wait_issuer(full0 + 8u * s, ph, abort_flag, a.status, 3)) { ok = false; break; }
                if (W4 && !dry && !mbar_wait_issuer(bready0 + 8u * s, ph, abort_flag, a.status, 11)) { ok = false; break; }
                tc_fence_after();
                const unsigned al = a_lo, b_lo = a.b_resident ? b_res : a_lo + a16;
                const unsigned acc = kb > 0 ? 1u : 0u, ebar = dry ? bfull + 8u : empty0 + 8u * s;
                if (!dry) {
                    a_lo += stage16;
                    b_res += b16;
                    if (++s == a.stages) { s = 0; ph ^= 1u; a_lo = a_lo0; }
                }
                dry = false;
                mbar_peek(full0 + 8u * s, ph);
                if (elect_one()) {
                    // advancing K by 32 bytes inside the swizzle span = +2 in the 16-byte address field
                    tc_mma_i8_lohi(d_tmem, al, b_lo, desc_hi, a.idesc, acc);
                    if (a.BK >= 64) tc_mma_i8_lohi(d_tmem, al + 2u, b_lo + 2u, desc_hi, a.idesc, 1u);
                    if (a.BK == 128) {
                        tc_mma_i8_lohi(d_tmem, al + 4u, b_lo + 4u, desc_hi, a.idesc, 1u);
                        tc_mma_i8_lohi(d_tmem, al + 6u, b_lo + 6u, desc_hi, a.idesc, 1u);
                    }
                    tc_commit(ebar);  // frees the stage once these MMAs have read it
                    if (kb + 1 == num_kb) tc_commit(tfull0 + 8u * as);
                }
                __syncwarp();
            }
        }
    } else if (W4 && warp >= EPI_WARP0 + NUM_EPI_WARPS) {
        // ------------------------------------------------------------------ int4 expansion warps
        // Stage s may be rewritten once full[s] has completed for the new fill: the producer only refills a stage
        // after the MMAs that read its previous contents have committed (empty[s]).
        const int ut = (warp - (EPI_WARP0 + NUM_EPI_WARPS)) * 32 + lane;
        const int cpr_shift = a.BK == 128 ? 3 : (a.BK == 64 ? 2 : 1);   // 16-byte chunks per B row: BK / 16
        const int total_chunks = a.BN << cpr_shift;
        const int half_bk = a.BK >> 1;
        int s = 0;
        unsigned ph = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
            for (int kb = 0; kb < num_kb; ++kb) {
                if (!mbar_wait_warp(full0 + 8u * s, ph, abort_flag, a.status, 12)) { ok = false; break; }
                unsigned char* bt = tiles + (size_t)s * stage_bytes + a_stage_bytes;
                const unsigned char* pk = bt + b_stage_bytes;
#pragma unroll 2
                for (int id = ut; id < total_chunks; id += 32 * W4_UNPACK_WARPS) {
                    const int row = id >> cpr_shift, ch = id & ((1 << cpr_shift) - 1);
                    const uint2 p = *(const uint2*)(pk + row * half_bk + ch * 8);
                    uint4 o;
                    expand_int4_x16(p.x, o.x, o.y);
                    expand_int4_x16(p.y, o.z, o.w);
                    *(uint4*)(bt + swz_off(row, ch * 16, a.BK)) = o;
                }
                fence_async_smem();   // generic-proxy stores, read by the tensor core through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(bready0 + 8u * s);
                if (++s == a.stages) { s = 0; ph ^= 1u; }
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue warps
        const int quad = warp & 3;                       // TMEM lane quadrant this warp may read
        // Warps w, w + 4, w + 8, w + 12 share a quadrant.  A tile of 256 columns goes to all four, 64 columns each; of narrower
        // tiles every warp still takes 64 columns and 128 / 64-column tiles are dealt out to two / four groups: the fixed
        // work of a warp per tile (waits, fences, the store) equals that of 16 to 32 columns of arithmetic.
        const int part4 = (warp - EPI_WARP0) >> 2;       // 0..3 within the quadrant
        const int part = FAST ? part4 & (a.parts - 1) : part4, group = FAST ? part4 / a.parts : 0;
        const int wp = a.BN / a.parts;
        const int row = quad * 32 + lane;
        const int epi_tid = (warp - EPI_WARP0) * 32 + lane;
        // the exact 64-bit epilogue works in 32-column chunks on the first two warps of each quadrant
        const int cols_per_warp = a.BN / 2;
        unsigned acc_it = (unsigned)group, mine = 0;   // the CTA's tiles so far, and this group's
        unsigned stage_it = 0;
        EpiState est;
        perm_rowbase(est.rb, wp, lane, wp >= 32 ? 4 : 2);
        int staged_n_tile = -1;
        int* par = epi_params;
        bool ok = true;
        const int bn_shift = 31 - __clz(a.BN);
        // Stages a column block's per-channel constants (once per CTA when the grid is a multiple of the number of column
        // blocks).  Two buffers: the other one may still be read by slower warps, this one is free once everybody
        // passed the previous barrier.
        auto stage_constants = [&](int n_tile) -> bool {
            par = epi_params + (size_t)(stage_it & 1u) * (2 * FAST_NP * 256);
            const int per_set = FAST_NP << bn_shift, all = a.fq2 ? 2 * per_set : per_set;
            for (int i = epi_tid; i < all; i += 32 * NUM_EPI_WARPS) {
                const int set = i >= per_set ? 1 : 0;
                const int prm = (i - set * per_set) >> bn_shift, c = i & (a.BN - 1);
                par[(set * FAST_NP + prm) * 256 + c] = __ldg((set ? a.fq2 : a.fq) + (size_t)prm * a.cpad + n_tile * a.BN + c);
            }
            const unsigned pb = pready0 + 8u * (stage_it & 1u);
            __syncwarp();
            if (lane == 0) mbar_arrive(pb);
            if (!mbar_wait_warp(pb, (stage_it >> 1) & 1u, abort_flag, a.status, 5)) return false;
            staged_n_tile = n_tile;
            ++stage_it;
            return true;
        };
        if (FAST && (int)blockIdx.x < num_tiles) ok = stage_constants((int)blockIdx.x % a.num_n_tiles);   // constants: before the wait
        bool dry = DRY;
        if (!dry) pdl_wait();   // residual loads and output stores touch tensors the previous kernel reads or writes
        // several groups only where the CTA's column block never changes (step_n is 0 or the CTA has one tile)
        const int groups = FAST ? a.groups : 1;
        const int tile_step = groups * (int)gridDim.x, step_m = groups * a.step_m, step_n = groups > 1 ? 0 : a.step_n;
        const int m_first = (int)blockIdx.x / a.num_n_tiles;
        int m_next = m_first + group * a.step_m, n_next = (int)blockIdx.x - m_first * a.num_n_tiles;
        const int first_tile = (int)blockIdx.x + group * (int)gridDim.x;
        // residual loads run ahead of the tiles: pf_* walk the same tile sequence, res_slots - 1 tiles in front
        int pf_tile = first_tile, pf_m = m_next, pf_n = n_next;
        unsigned pf_it = 0;
        const unsigned slot_shift = a.res_slots == 4 ? 2u : 1u;
        const unsigned lookahead = a.res_slots == 4 ? 3u : 2u;
        const unsigned my_regions = (unsigned)(stage_out - smem_raw) + (unsigned)((warp - EPI_WARP0) * REGION_BYTES * regions_per_warp);
        const unsigned my_rbar = rbar0 + 32u * (unsigned)(warp - EPI_WARP0);
        for (int tile = first_tile; tile < num_tiles && ok;) {
            const int n_tile = n_next, m_tile = m_next;
            if (!dry) {
                m_next += step_m;
                n_next += step_n;
                if (n_next >= a.num_n_tiles) { n_next -= a.num_n_tiles; ++m_next; }
            }
            const int m0 = a.m_base + m_tile * BM, n0 = n_tile * a.BN;
            const unsigned as = acc_it & ((1u << a.acc_shift) - 1u);
            const unsigned aph = (acc_it >> a.acc_shift) & 1u;
            if (FAST && n_tile != staged_n_tile)
                if (!stage_constants(n_tile)) { ok = false; break; }
            const int m = m0 + row;
            const bool m_ok = m < a.m_base + a.M;
            const int cbase = part * cols_per_warp;
            if (FAST) {
                // fragment-layout epilogue with swizzled staging, TMA store and TMA residual load
                EpiTile e;
                e.tmem_acc = tmem_base + as * (unsigned)a.BN;
                e.BN = a.BN; e.N = a.N; e.M = a.m_base + a.M; e.m0 = m0; e.n0 = n0; e.out = (uint8_t*)a.out; e.ldo = a.ldo;
                e.wp = wp;
                e.par_off = (unsigned)((unsigned char*)par - smem_raw);
                e.region_off = my_regions;
                e.region_stride = RES ? REGION_BYTES : 0;
                e.slot_shift = slot_shift;
                e.rbar = my_rbar;
                if (RES && !dry) {
                    if (lane == 0) {
                        // two regions: the previous tile's store has finished reading, its region takes the next
                        // tile.  Four regions: the store before that one has, its region takes the tile two ahead,
                        // and nobody waits on a store that has only just been issued.
                        if (a.res_slots == 4) bulk_wait_read_1(); else bulk_wait_read_all();
                        while (pf_it < mine + lookahead && pf_tile < num_tiles) {
                            epi_issue_residual(&tmR, my_regions, REGION_BYTES, my_rbar, pf_it & ((1u << slot_shift) - 1u),
                                               pf_n * a.BN + part * e.wp, a.m_base + pf_m * BM + quad * 32, a.N, e.M, e.wp);
                            ++pf_it;
                            pf_tile += tile_step;
                            pf_m += step_m;
                            pf_n += step_n;
                            if (pf_n >= a.num_n_tiles) { pf_n -= a.num_n_tiles; ++pf_m; }
                        }
                    }
                    __syncwarp();
                }
                e.tfull = tfull0 + 8u * as; e.tfull_parity = aph; e.tempty = tempty0 + 8u * as;
                e.abort_flag = abort_flag; e.status = a.status; e.dry = dry;
                e.ef = a.ef;
                e.t_lo = a.t_lo; e.t_hi = a.t_hi;
                if (!fast_epilogue_tile<RES, CLAMP, DP, true, W4, DRY>(&tmO, &tmR, e, quad, part, lane, est)) { ok = false; break; }
                if (dry) {
                    dry = false;
                    pdl_wait();
                    continue;
                }
                tile += tile_step;
                acc_it += (unsigned)groups;
                ++mine;
                continue;
            } else {
                if (!mbar_wait_warp(tfull0 + 8u * as, aph, abort_flag, a.status, 4)) { ok = false; break; }
                tc_fence_after();
                for (int cc = 0; cc < cols_per_warp && part < 2; cc += 32) {
                    const int c0 = cbase + cc;
                    unsigned v[32];
                    const unsigned taddr = tmem_base + ((unsigned)(quad * 32) << 16) + as * (unsigned)a.BN + (unsigned)c0;
                    const int nbase = n0 + c0;
                    tc_ld32(taddr, v);
                    tc_wait_ld_into(v);
                    if (!m_ok || nbase >= a.N) continue;
                    int y[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const int n = nbase + j;
                        if (n < a.N) {
                            // W4: the accumulator holds 16 x the sum (a multiple of 16: the shift is exact)
                            const long long x = (long long)(W4 ? ((int)v[j] >> 4) : (int)v[j]) + (a.q.bias ? (long long)a.q.bias[n] : 0ll);
                            int t = requant64(x, n, a.q);
                            if (a.r.ptr) {
                                const long long u = (long long)t
                                    + (long long)load_i8(a.r.ptr, (size_t)m * a.N + n, a.r.is_unsigned != 0);
                                t = requant64(u, n, a.r.q2);
                            }
                            y[j] = t;
                        } else {
                            y[j] = 0;
                        }
                    }
                    if (a.out_dtype == DT_I8) {
                        uint8_t* op = (uint8_t*)a.out + (size_t)m * a.N + nbase;
                        if ((a.N % 16 == 0) && nbase + 32 <= a.N) {
                            unsigned wds[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                wds[i] = ((unsigned)y[4 * i] & 0xffu) | (((unsigned)y[4 * i + 1] & 0xffu) << 8)
                                       | (((unsigned)y[4 * i + 2] & 0xffu) << 16) | (((unsigned)y[4 * i + 3] & 0xffu) << 24);
                            ((uint4*)op)[0] = make_uint4(wds[0], wds[1], wds[2], wds[3]);
                            ((uint4*)op)[1] = make_uint4(wds[4], wds[5], wds[6], wds[7]);
                        } else {
                            for (int j = 0; j < 32 && nbase + j < a.N; ++j) op[j] = (uint8_t)y[j];
                        }
                    } else {
                        int32_t* op = (int32_t*)a.out + (size_t)m * a.N + nbase;
                        for (int j = 0; j < 32 && nbase + j < a.N; ++j) op[j] = y[j];
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty0 + 8u * as);
            tile += (int)gridDim.x;
            ++acc_it;
        }
        // no bulk store may still be reading this CTA's shared memory when it exits (its writes complete with the grid)
        if (FAST && lane == 0) bulk_wait_read_all();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(a.tmem_cols) : "memory");
    }
}

typedef void (*IgemmKernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const IgemmArgs);
extern const IgemmKernel igemm_w4_kernels[6];   // by MODE, of packed 4-bit weights: an object of its own, loaded by the networks that have some

}  // namespace n2d2b
