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
#include <cstdio>
#include <cstring>
#include <algorithm>
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
    int* status;
    QuantDev q;
    Residual r;
    // fast 32-bit epilogue: y = (clamp(acc, lo, hi) * mult + add) >> shift, rows of cpad entries
    const int* fq;      // [FAST_NP][cpad] of the cell
    const int* fq2;     // [FAST_NP][cpad] of the fused residual sum (nullptr without one)
    int cpad;
    int t_lo, t_hi;     // saturation range of the cell's own output (before the residual add)
    int out_unsigned;   // final 8-bit range: 1 = [0,255], 0 = [-128,127]
    unsigned dp_xor;    // dot-product form of the residual stage: byte flips and operand signedness
    int dp_a_signed;
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
                e.BN = a.BN; e.N = a.N; e.M = a.m_base + a.M; e.m0 = m0; e.n0 = n0; e.out = (uint8_t*)a.out;
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
                e.t_lo = a.t_lo; e.t_hi = a.t_hi; e.dp_xor = a.dp_xor;
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
                        case 0: perm_block<4, false, CLAMP, false, EF_PERM>(va, vb, par_off, pc, region_off, rb, 0, lane, 0, 0, 0u); break;
                        case EF_OUT_UNSIGNED:
                            perm_block<4, false, CLAMP, false, EF_OUT_UNSIGNED | EF_PERM>(va, vb, par_off, pc, region_off, rb, 0, lane, 0, 0, 0u);
                            break;
                        case EF_WIDE: perm_block<4, false, false, false, EF_WIDE | EF_PERM>(va, vb, par_off, pc, region_off, rb, 0, lane, 0, 0, 0u); break;
                        case EF_WIDE | EF_OUT_UNSIGNED:
                            perm_block<4, false, false, false, EF_WIDE | EF_OUT_UNSIGNED | EF_PERM>(va, vb, par_off, pc, region_off, rb, 0, lane, 0, 0, 0u);
                            break;
                        case EF_FLOAT: perm_block<4, false, CLAMP, false, EF_FLOAT | EF_PERM>(va, vb, par_off, pc, region_off, rb, 0, lane, 0, 0, 0u); break;
                        default:
                            perm_block<4, false, CLAMP, false, EF_FLOAT | EF_OUT_UNSIGNED | EF_PERM>(va, vb, par_off, pc, region_off, rb, 0, lane, 0, 0, 0u);
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
    if (!plan->a_im2col) {
        const cuuint64_t dims[2] = {(cuuint64_t)g.C, (cuuint64_t)plan->M};
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
        if (res) {
            rc = g_encode_tiled(&plan->tmR, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)res, dims, strides, box, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(wb), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (rc != CUDA_SUCCESS) { *why = "cuTensorMapEncodeTiled failed for the residual matrix"; return -1; }
        }
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
    if (form == EF_WIDE) return rescale<false, EF_WIDE>(x, c[0], 0, c[2 * stride], c[3 * stride], c[4 * stride]);
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
                    a4 ^= a.dp_xor;
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

// Eight weights per thread; at most a few megabytes that stay in L2
__global__ void __launch_bounds__(256) widen_int4_kernel(const uint8_t* __restrict__ packed, int rows_src, int ng_src, int8_t* __restrict__ dst, int rows,
                                                         int ng_dst, unsigned words)
{
    pdl_launch_dependents();
    pdl_wait();   // the destination may still be read by the previous kernel
    const unsigned total = (unsigned)rows * words;   // 8-byte words of the destination
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const unsigned n = i / words, w = i - n * words;
        const int real = perm_real_channel((int)n, ng_dst);
        uint2 o = make_uint2(0u, 0u);
        if (real < rows_src) {
            int src = real;
            if (ng_src) {   // where the packed rows hold this channel (the inverse of perm_real_channel)
                const int j = real % (8 * ng_src), q = j / (2 * ng_src), r = j - q * 2 * ng_src;
                src = real - j + 8 * (r >> 1) + 2 * q + (r & 1);
            }
            unsigned lo, hi;
            expand_int4_x16(__ldg((const unsigned*)packed + (size_t)src * words + w), lo, hi);
            auto down = [](unsigned x) {   // 16 x the value in every byte -> the value
                const unsigned t = (x >> 4) & 0x0f0f0f0fu;
                return t | ((t & 0x08080808u) * 0x1eu);
            };
            o = make_uint2(down(lo), down(hi));
        }
        ((uint2*)dst)[i] = o;
    }
}

cudaError_t launch_widen_int4(const uint8_t* packed, int rows_src, int ng_src, int8_t* dst, int rows, int ng_dst, size_t row_bytes, cudaStream_t s)
{
    const unsigned words = (unsigned)(row_bytes / 8);
    const unsigned long long total = (unsigned long long)rows * words;
    if (total == 0) return cudaSuccess;
    if (total >= (1ull << 31)) return cudaErrorInvalidValue;
    const unsigned long long blocks = (total + 255) / 256;
    return launch_pdl(widen_int4_kernel, (int)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, s, packed, rows_src, ng_src, dst, rows, ng_dst, words);
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

cudaError_t launch_igemm(const IgemmPlan& plan, const QuantDev& q, const Residual& r, const FastQuant& fast, void* out,
                         int out_dtype, int m_base, int* status_word, cudaStream_t s)
{
    if (plan.M == 0 || plan.N == 0) return cudaSuccess;
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
    a.status = status_word;
    a.q = q;
    a.r = r;
    a.fq = fast.fq; a.fq2 = fast.fq2; a.cpad = fast.cpad; a.t_lo = fast.t_lo; a.t_hi = fast.t_hi;
    a.out_unsigned = fast.out_unsigned;
    a.dp_xor = fast.dp_xor;
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
    typedef void (*Kernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const IgemmArgs);
    static const Kernel kernels[3][6] = {
        {igemm_i8_tcgen05_kernel<0, false, false>, igemm_i8_tcgen05_kernel<1, false, false>, igemm_i8_tcgen05_kernel<2, false, false>,
         igemm_i8_tcgen05_kernel<3, false, false>, igemm_i8_tcgen05_kernel<4, false, false>, igemm_i8_tcgen05_kernel<5, false, false>},
        {igemm_i8_tcgen05_kernel<0, false, false>, igemm_i8_tcgen05_kernel<1, false, true>, igemm_i8_tcgen05_kernel<2, false, true>,
         igemm_i8_tcgen05_kernel<3, false, true>, igemm_i8_tcgen05_kernel<4, false, true>, igemm_i8_tcgen05_kernel<5, false, true>},
        {igemm_i8_tcgen05_kernel<0, true, false>, igemm_i8_tcgen05_kernel<1, true, false>, igemm_i8_tcgen05_kernel<2, true, false>,
         igemm_i8_tcgen05_kernel<3, true, false>, igemm_i8_tcgen05_kernel<4, true, false>, igemm_i8_tcgen05_kernel<5, true, false>}};
    static SmemLimitSet limits[3][6];
    int tiles = a.num_m_tiles * a.num_n_tiles;
    // Few tiles, long K: a cluster of CTAs per tile
    const int num_kb = plan.taps * ((plan.Cin + plan.BK - 1) / plan.BK);
    if (use_fast && !plan.w4 && !plan.grouped && plan.BN == SPLIT_BN && igemm_split(tiles, num_kb, plan.num_sms)) {
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
    int grid = plan.grid < tiles ? plan.grid : tiles;
    // a grid that is a multiple of the number of column blocks keeps every CTA on one column block,
    // so its per-channel constants are staged once
    if (tiles > grid && a.num_n_tiles > 1 && grid > a.num_n_tiles) grid -= grid % a.num_n_tiles;
    // resident weights rely on exactly that (or on one tile per CTA)
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
    const int table = plan.w4 ? 2 : (tiles <= 2 * grid ? 1 : 0);
    if (cudaError_t e = raise_smem_limit(kernels[table][mode], limits[table][mode])) return e;
    return launch_pdl(kernels[table][mode], grid, NUM_THREADS + (plan.w4 ? 32 * W4_UNPACK_WARPS : 0), plan.smem_bytes, s,
                      plan.tmA, plan.tmB, plan.tmO, plan.tmR, a);
}

}  // namespace n2d2b
