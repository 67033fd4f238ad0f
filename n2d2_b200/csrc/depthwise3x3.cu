#include <algorithm>
#include "kernels.h"
#include "tc_common.cuh"

namespace n2d2b {

// Depthwise 3x3 convolution, stride 1 or 2, no dilation.  What bounds it is instruction issue on small maps and memory on large
// ones, so both are kept low: a thread owns four channels (one 32-bit word per pixel) of two horizontally adjacent
// output pixels and walks down a strip of output rows.  Of every input row it reads four (stride 2: five) words and
// transposes them once to one word per channel of four adjacent columns, which serves both pixels (the second one with its weights a
// byte higher) and up to three output rows: three byte dot products and about one byte permute per output, where the same on
// the tensor cores multiplies 64 x 64 blocks that are zero off the diagonal and moves nine shifted copies of the input
// through shared memory.  Three (two) rows are on their way while one is worked on.  Measured: 112 instructions per eight outputs,
// 64 % of the issue slots, two blocks per SM by registers (three, with spills, are slower); 14 x 14 x 512 at 256 images 24 us,
// 31 as block-diagonal groups (see use_dw3x3 for where each is taken).
struct DwSplit {
    int cwb;               // channel words per block
    int slots;             // positions a block works on at once (blockDim.x >= cwb * slots)
    int xunits, strips, rows;   // pairs of output columns, strips per image, output rows per strip
    unsigned jobs;         // images * strips * xunits
};

// Four pixels of four channels -> one word per channel
__device__ __forceinline__ void dw_transpose4(unsigned p0, unsigned p1, unsigned p2, unsigned p3, unsigned (&t)[4])
{
    const unsigned a = __byte_perm(p0, p1, 0x5140), b = __byte_perm(p0, p1, 0x7362);
    const unsigned c = __byte_perm(p2, p3, 0x5140), d = __byte_perm(p2, p3, 0x7362);
    t[0] = __byte_perm(a, c, 0x5410);
    t[1] = __byte_perm(a, c, 0x7632);
    t[2] = __byte_perm(b, d, 0x5410);
    t[3] = __byte_perm(b, d, 0x7632);
}

template <bool IN_UNSIGNED>
__device__ __forceinline__ int dw_dot(unsigned x, unsigned w, int acc)
{
    if (IN_UNSIGNED) asm("dp4a.u32.s32 %0, %1, %2, %0;" : "+r"(acc) : "r"(x), "r"(w));
    else asm("dp4a.s32.s32 %0, %1, %2, %0;" : "+r"(acc) : "r"(x), "r"(w));
    return acc;
}

template <bool IN_UNSIGNED, bool OUT_UNSIGNED, int S, bool CLAMP, int EF>
__global__ void __launch_bounds__(256, 2)
conv_depthwise3x3_kernel(const uint8_t* __restrict__ in, const int8_t* __restrict__ w_hwc, ConvGeom g, const int* __restrict__ fq,
                         int cpad, uint8_t* __restrict__ out, DwSplit d)
{
    constexpr int NQ = S == 1 ? 4 : 5;     // input columns of two output columns
    constexpr int NT = S == 1 ? 4 : 8;     // transposed words: per channel, at stride 2 once per output column
    pdl_launch_dependents();
    const int cw = g.C / 4;
    const int slot = (int)threadIdx.x / d.cwb;
    const int c4 = (int)blockIdx.y * d.cwb + ((int)threadIdx.x - slot * d.cwb);
    if (slot >= d.slots || c4 >= cw) return;
    // weights of filter row ky, channel j: bytes [w0 w1 w2 0]; constants: before the wait
    unsigned wt[3][4];
    int lo[4], hi[4], mu[4], ad[4], sh[4];
#pragma unroll
    for (int ky = 0; ky < 3; ++ky) {
        const unsigned* wp = (const unsigned*)(w_hwc + (size_t)(3 * ky) * g.C) + c4;
        dw_transpose4(__ldg(wp), __ldg(wp + cw), __ldg(wp + 2 * cw), 0u, wt[ky]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int ch = c4 * 4 + j;
        lo[j] = (CLAMP || (EF & EF_WIDE)) ? __ldg(fq + 0 * cpad + ch) : 0;
        hi[j] = CLAMP ? __ldg(fq + 1 * cpad + ch) : 0;
        mu[j] = __ldg(fq + 2 * cpad + ch);
        ad[j] = __ldg(fq + 3 * cpad + ch);
        sh[j] = __ldg(fq + 4 * cpad + ch);
    }
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    const size_t pitch = (size_t)g.W * cw, opitch = (size_t)g.oW * cw;
    for (unsigned job = blockIdx.x * d.slots + slot; job < d.jobs; job += gridDim.x * d.slots) {
        const unsigned t = job / d.xunits, b = t / d.strips;
        const int ox = 2 * (int)(job - t * d.xunits), oy0 = (int)(t - b * d.strips) * d.rows;
        const int n = min(d.rows, g.oH - oy0);
        const int ix = ox * S - g.pL;
        int iy = oy0 * S - g.pT;
        bool col[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) col[q] = (unsigned)(ix + q) < (unsigned)g.W;
        const bool two = ox + 1 < g.oW;
        const unsigned* p = (const unsigned*)in + ((long long)b * g.H + iy) * (long long)pitch + (long long)ix * cw + c4;
        unsigned* o = (unsigned*)out + ((size_t)b * g.oH + oy0) * opitch + (size_t)ox * cw + c4;
        const int iy_end = min(g.H, iy + S * (n - 1) + 3);   // rows past the strip's last one are not read
        auto load = [&](unsigned (&r)[NQ]) {
            const bool row = iy >= 0 && iy < iy_end;
#pragma unroll
            for (int q = 0; q < NQ; ++q) r[q] = row && col[q] ? __ldg(p + q * cw) : 0u;
            ++iy;
            p += pitch;
        };
        auto turn = [&](const unsigned (&r)[NQ], unsigned (&x)[NT]) {
            unsigned y[4];
            dw_transpose4(r[0], r[1], r[2], r[3], y);
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = y[j];
            if (S == 2) {
                // columns 1 .. 4: the word of columns 0 .. 3 moved down a byte, column 4 on top
#pragma unroll
                for (int j = 0; j < 4; ++j) x[4 + j] = __byte_perm(y[j], r[NQ - 1], 0x4321 + 0x1000 * j);
            }
        };
        auto emit = [&](const unsigned (&x0)[NT], const unsigned (&x1)[NT], const unsigned (&x2)[NT]) {
            int y0[4], y1[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                int a = 0, c = 0;
                a = dw_dot<IN_UNSIGNED>(x0[j], wt[0][j], a);
                c = dw_dot<IN_UNSIGNED>(x0[NT - 4 + j], wt[0][j] << 8, c);
                a = dw_dot<IN_UNSIGNED>(x1[j], wt[1][j], a);
                c = dw_dot<IN_UNSIGNED>(x1[NT - 4 + j], wt[1][j] << 8, c);
                a = dw_dot<IN_UNSIGNED>(x2[j], wt[2][j], a);
                c = dw_dot<IN_UNSIGNED>(x2[NT - 4 + j], wt[2][j] << 8, c);
                y0[j] = rescale<CLAMP, EF>(a, lo[j], hi[j], mu[j], ad[j], sh[j]);
                y1[j] = rescale<CLAMP, EF>(c, lo[j], hi[j], mu[j], ad[j], sh[j]);
            }
            o[0] = pack4_sat(y0[0], y0[1], y0[2], y0[3], OUT_UNSIGNED);
            if (two) o[cw] = pack4_sat(y1[0], y1[1], y1[2], y1[3], OUT_UNSIGNED);
            o += opitch;
        };
        if (S == 1) {
            unsigned r0[NQ], r1[NQ], r2[NQ], x0[NT], x1[NT], x2[NT];
            load(r0);
            load(r1);
            load(r2);
            turn(r0, x0);
            load(r0);
            turn(r1, x1);
            load(r1);
            for (int y = 0; y < n; y += 3) {
                turn(r2, x2);
                load(r2);
                emit(x0, x1, x2);
                if (y + 1 >= n) break;
                turn(r0, x0);
                load(r0);
                emit(x1, x2, x0);
                if (y + 2 >= n) break;
                turn(r1, x1);
                load(r1);
                emit(x2, x0, x1);
            }
        } else {
            unsigned r0[NQ], r1[NQ], x0[NT], x1[NT], x2[NT];
            load(r0);
            load(r1);
            turn(r0, x0);
            load(r0);
            for (int y = 0; y < n; y += 2) {
                turn(r1, x1);
                load(r1);
                turn(r0, x2);
                load(r0);
                emit(x0, x1, x2);
                if (y + 1 >= n) break;
                turn(r1, x1);
                load(r1);
                turn(r0, x0);
                load(r0);
                emit(x2, x1, x0);
            }
        }
    }
}

bool depthwise3x3_eligible(const ConvGeom& g)
{
    return g.kH == 3 && g.kW == 3 && g.dX == 1 && g.dY == 1 && g.sX == g.sY && (g.sX == 1 || g.sX == 2) && g.C % 4 == 0
        && g.groups == g.C && g.O == g.C;
}

template <bool IN_UNSIGNED, bool OUT_UNSIGNED, int S>
static cudaError_t launch_depthwise3x3(dim3 grid, int threads, cudaStream_t s, const uint8_t* in, const int8_t* w, const ConvGeom& g,
                                       const FastQuant& f, uint8_t* out, const DwSplit& d)
{
    if (f.form == EF_WIDE) return launch_pdl(f.need_clamp ? conv_depthwise3x3_kernel<IN_UNSIGNED, OUT_UNSIGNED, S, true, EF_WIDE>
                                                          : conv_depthwise3x3_kernel<IN_UNSIGNED, OUT_UNSIGNED, S, false, EF_WIDE>, grid, threads, 0, s, in, w, g, f.fq, f.cpad, out, d);
    if (f.form == EF_FLOAT) return launch_pdl(f.need_clamp ? conv_depthwise3x3_kernel<IN_UNSIGNED, OUT_UNSIGNED, S, true, EF_FLOAT>
                                                           : conv_depthwise3x3_kernel<IN_UNSIGNED, OUT_UNSIGNED, S, false, EF_FLOAT>,
                                              grid, threads, 0, s, in, w, g, f.fq, f.cpad, out, d);
    return launch_pdl(f.need_clamp ? conv_depthwise3x3_kernel<IN_UNSIGNED, OUT_UNSIGNED, S, true, 0>
                                   : conv_depthwise3x3_kernel<IN_UNSIGNED, OUT_UNSIGNED, S, false, 0>,
                      grid, threads, 0, s, in, w, g, f.fq, f.cpad, out, d);
}

cudaError_t launch_depthwise3x3(const void* in, int in_unsigned, const int8_t* w_hwc, const ConvGeom& g, const FastQuant& fast, void* out,
                                int num_sms, cudaStream_t s)
{
    if (!fast.enabled || !depthwise3x3_eligible(g)) return cudaErrorInvalidValue;
    if (g.B <= 0 || g.oW <= 0 || g.oH <= 0) return cudaSuccess;
    const int cw = g.C / 4;
    DwSplit d;
    const int blocks_y = (cw + 127) / 128;
    d.cwb = (cw + blocks_y - 1) / blocks_y;
    d.slots = 256 / d.cwb;
    d.xunits = (g.oW + 1) / 2;
    // Long strips read the fewest rows twice (two per strip), short ones fill the chip: halve them while there are not six jobs per
    // slot for an even finish, or, below eight rows, not even one
    const long long resident = std::max(1ll, (long long)num_sms * 2 / blocks_y) * d.slots;
    const long long columns = (long long)g.B * d.xunits;
    d.rows = g.oH;
    while (d.rows > 1 && columns * ((g.oH + d.rows - 1) / d.rows) < resident * (d.rows > 8 ? 6 : 1)) d.rows = (d.rows + 1) / 2;
    d.strips = (g.oH + d.rows - 1) / d.rows;
    const long long jobs = columns * d.strips;
    if (jobs >= (1ll << 31)) return cudaErrorInvalidValue;
    d.jobs = (unsigned)jobs;
    const long long blocks = (jobs + d.slots - 1) / d.slots, most = std::max(1ll, (long long)num_sms * 2 / blocks_y);
    const dim3 grid((unsigned)std::min(blocks, most), (unsigned)blocks_y);
    const int threads = (d.cwb * d.slots + 31) / 32 * 32;
    const uint8_t* ip = (const uint8_t*)in;
    uint8_t* op = (uint8_t*)out;
    switch ((in_unsigned ? 4 : 0) | (fast.out_unsigned ? 2 : 0) | (g.sX == 2 ? 1 : 0)) {
    case 0: return launch_depthwise3x3<false, false, 1>(grid, threads, s, ip, w_hwc, g, fast, op, d);
    case 1: return launch_depthwise3x3<false, false, 2>(grid, threads, s, ip, w_hwc, g, fast, op, d);
    case 2: return launch_depthwise3x3<false, true, 1>(grid, threads, s, ip, w_hwc, g, fast, op, d);
    case 3: return launch_depthwise3x3<false, true, 2>(grid, threads, s, ip, w_hwc, g, fast, op, d);
    case 4: return launch_depthwise3x3<true, false, 1>(grid, threads, s, ip, w_hwc, g, fast, op, d);
    case 5: return launch_depthwise3x3<true, false, 2>(grid, threads, s, ip, w_hwc, g, fast, op, d);
    case 6: return launch_depthwise3x3<true, true, 1>(grid, threads, s, ip, w_hwc, g, fast, op, d);
    default: return launch_depthwise3x3<true, true, 2>(grid, threads, s, ip, w_hwc, g, fast, op, d);
    }
}

}  // namespace n2d2b
