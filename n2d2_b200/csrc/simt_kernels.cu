// CUDA-core kernels of the quantized integer path: the layers that are not dense contractions
// (depthwise convolution, pooling, element-wise sum, stand-alone rescale) plus a direct convolution
// and a direct fully-connected kernel that accept any geometry.  Every kernel ends in the same
// requantisation epilogue (common.cuh), so no float tensor or separate Scaling pass exists between
// layers.  Activations are NHWC int8 (signed or unsigned per tensor) or int32.
#include <algorithm>
#include "kernels.h"
#include "tc_common.cuh"

namespace n2d2b {

static inline unsigned grid_for(size_t n, int block)
{
    size_t g = (n + block - 1) / block;
    const size_t cap = 303104;   // loops beyond: more blocks than any device holds at once
    return (unsigned)(g < cap ? (g ? g : 1) : cap);
}

template <typename T>
__device__ __forceinline__ void store_out(void* out, size_t i, int v);
template <>
__device__ __forceinline__ void store_out<int8_t>(void* out, size_t i, int v)
{
    ((int8_t*)out)[i] = (int8_t)v;  // the low byte is the value for both u8 and s8 tensors
}
template <>
__device__ __forceinline__ void store_out<int32_t>(void* out, size_t i, int v)
{
    ((int32_t*)out)[i] = v;
}

// ---------------------------------------------------------------------------------------------
// Direct convolution: one thread per output value, output channel fastest (NHWC).  Replaces the
// reference's ConvCell_Frame_Kernels::forward + forwardBias + Scaling + activation for geometries
// the tensor-core kernel does not take (few input channels, groups, dilation).
// ---------------------------------------------------------------------------------------------
template <typename OutT>
__global__ void conv_direct_kernel(const uint8_t* __restrict__ in, int in_unsigned,
                                   const int8_t* __restrict__ w, ConvGeom g, QuantDev q,
                                   Residual r, void* __restrict__ out, size_t total)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    const bool vec4 = (g.Cg % 4 == 0);
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int o = (int)(idx % g.O);
        size_t p = idx / g.O;
        const int ox = (int)(p % g.oW); p /= g.oW;
        const int oy = (int)(p % g.oH);
        const int b = (int)(p / g.oH);
        const int grp = o / g.Og;
        const int iy0 = oy * g.sY - g.pT, ix0 = ox * g.sX - g.pL;
        const int8_t* wo = w + (size_t)o * g.kH * g.kW * g.Cg;
        int acc = 0;
        for (int ky = 0; ky < g.kH; ++ky) {
            const int iy = iy0 + ky * g.dY;
            if (iy < 0 || iy >= g.H) continue;
            for (int kx = 0; kx < g.kW; ++kx) {
                const int ix = ix0 + kx * g.dX;
                if (ix < 0 || ix >= g.W) continue;
                const uint8_t* ip = in + (((size_t)b * g.H + iy) * g.W + ix) * g.C + (size_t)grp * g.Cg;
                const int8_t* wp = wo + (size_t)(ky * g.kW + kx) * g.Cg;
                if (vec4 && ((((uintptr_t)ip) | ((uintptr_t)wp)) & 3) == 0) {
                    const unsigned* ip4 = (const unsigned*)ip;
                    const int* wp4 = (const int*)wp;
                    if (in_unsigned)
                        for (int c = 0; c < g.Cg / 4; ++c) acc = dp4a_us(ip4[c], wp4[c], acc);
                    else
                        for (int c = 0; c < g.Cg / 4; ++c) acc = dp4a_ss((int)ip4[c], wp4[c], acc);
                } else {
                    for (int c = 0; c < g.Cg; ++c)
                        acc += load_i8(ip, c, in_unsigned) * (int)wp[c];
                }
            }
        }
        long long x = (long long)acc + (q.bias ? (long long)q.bias[o] : 0ll);
        int y = requant64(x, o, q);
        if (r.ptr) {
            const long long u = (long long)y + (long long)load_i8(r.ptr, idx, r.is_unsigned);
            y = requant64(u, o, r.q2);
        }
        store_out<OutT>(out, idx, y);
    }
}

cudaError_t launch_conv_direct(const void* in, int in_unsigned, const int8_t* w, const ConvGeom& g,
                               const QuantDev& q, const Residual& r, void* out, int out_dtype,
                               cudaStream_t s)
{
    const size_t total = (size_t)g.B * g.oH * g.oW * g.O;
    if (total == 0) return cudaSuccess;
    const int block = 256;
    const unsigned grid = grid_for(total, block);
    if (out_dtype == DT_I8)
        launch_pdl(conv_direct_kernel<int8_t>, grid, block, 0, s, (const uint8_t*)in, in_unsigned, w, g, q, r, out, total);
    else
        launch_pdl(conv_direct_kernel<int32_t>, grid, block, 0, s, (const uint8_t*)in, in_unsigned, w, g, q, r, out, total);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Depthwise convolution: HBM-bound (one multiply-add per loaded byte and tap), so it stays on the
// CUDA cores.  One thread owns 16 consecutive channels of one output pixel: every tap is one
// 128-bit load of the input and one of the weights, the result one 128-bit store.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void unpack16(const uint4& v, bool is_unsigned, int* x)
{
    const unsigned wds[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const unsigned byte = (wds[i] >> (8 * j)) & 0xffu;
            x[i * 4 + j] = is_unsigned ? (int)byte : (int)(int8_t)byte;
        }
}

__device__ __forceinline__ uint4 pack16(const int* y)
{
    unsigned wds[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        wds[i] = ((unsigned)y[i * 4] & 0xffu) | (((unsigned)y[i * 4 + 1] & 0xffu) << 8)
               | (((unsigned)y[i * 4 + 2] & 0xffu) << 16) | (((unsigned)y[i * 4 + 3] & 0xffu) << 24);
    return make_uint4(wds[0], wds[1], wds[2], wds[3]);
}

__global__ void conv_depthwise_kernel(const uint8_t* __restrict__ in, int in_unsigned,
                                      const int8_t* __restrict__ w_hwc, ConvGeom g, QuantDev q,
                                      uint8_t* __restrict__ out, size_t total_vec)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    const int cv = g.C / 16;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total_vec;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int c16 = (int)(idx % cv);
        size_t p = idx / cv;
        const int ox = (int)(p % g.oW); p /= g.oW;
        const int oy = (int)(p % g.oH);
        const int b = (int)(p / g.oH);
        const int c0 = c16 * 16;
        int acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0;
        const int iy0 = oy * g.sY - g.pT, ix0 = ox * g.sX - g.pL;
        for (int ky = 0; ky < g.kH; ++ky) {
            const int iy = iy0 + ky * g.dY;
            if (iy < 0 || iy >= g.H) continue;
            for (int kx = 0; kx < g.kW; ++kx) {
                const int ix = ix0 + kx * g.dX;
                if (ix < 0 || ix >= g.W) continue;
                const uint4 xv = *(const uint4*)(in + (((size_t)b * g.H + iy) * g.W + ix) * g.C + c0);
                const uint4 wv = __ldg((const uint4*)(w_hwc + (size_t)(ky * g.kW + kx) * g.C + c0));
                int xs[16], ws[16];
                unpack16(xv, in_unsigned != 0, xs);
                unpack16(wv, false, ws);
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[i] += xs[i] * ws[i];
            }
        }
        int y[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const long long x = (long long)acc[i] + (q.bias ? (long long)q.bias[c0 + i] : 0ll);
            y[i] = requant64(x, c0 + i, q);
        }
        *(uint4*)(out + idx * 16) = pack16(y);
    }
}

// Other depthwise 3x3 convolutions (dilated, unequal or larger strides) with the 32-bit epilogue.  A thread owns four channels (one 32-bit word per pixel) of
// four horizontally adjacent output pixels.  Its weights are kept as one word per (tap, channel) with the other three
// bytes cleared, so a channel's product is a single four-way byte dot product on the packed input word, without
// unpacking anything: 144 dp4a for 16 outputs.  One block per output row, no 64-bit index arithmetic.
// fq = [5][cpad] constants of the 32-bit rescale (lo, hi, mult, add, shift), proved exact on the host.
template <bool IN_UNSIGNED>
__device__ __forceinline__ void dw_mac4(int (&acc)[4], unsigned xv, const unsigned (&w)[4])
{
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (IN_UNSIGNED) asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(acc[j]) : "r"(xv), "r"(w[j]), "r"(acc[j]));
        else asm("dp4a.s32.s32 %0, %1, %2, %3;" : "=r"(acc[j]) : "r"(xv), "r"(w[j]), "r"(acc[j]));
    }
}

template <bool IN_UNSIGNED, bool CLAMP, bool OUT_UNSIGNED>
__global__ void __launch_bounds__(256)
conv_depthwise3x3_dp4a_kernel(const uint8_t* __restrict__ in, const int8_t* __restrict__ w_hwc, ConvGeom g,
                              const int* __restrict__ fq, int cpad, uint8_t* __restrict__ out)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    const int cw = g.C / 4;                        // channel words per pixel
    // blockDim.x is a multiple of cw: a thread keeps its channel word over the whole launch.  All offsets are 32-bit word indices (checked by the host).
    const int c4 = threadIdx.x % cw;
    const int xi = threadIdx.x / cw;
    const int xthreads = blockDim.x / cw;
    unsigned wm[9][4];
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        const unsigned wv = __ldg((const unsigned*)(w_hwc + (size_t)t * g.C) + c4);
#pragma unroll
        for (int j = 0; j < 4; ++j) wm[t][j] = wv & (0xffu << (8 * j));
    }
    int lo[4], hi[4], mu[4], ad[4], sh[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int ch = c4 * 4 + j;
        lo[j] = __ldg(fq + 0 * cpad + ch); hi[j] = __ldg(fq + 1 * cpad + ch);
        mu[j] = __ldg(fq + 2 * cpad + ch); ad[j] = __ldg(fq + 3 * cpad + ch); sh[j] = __ldg(fq + 4 * cpad + ch);
    }
    const unsigned* in_w = (const unsigned*)in + c4;
    unsigned* out_w = (unsigned*)out + c4;
    for (int row = blockIdx.x; row < g.B * g.oH; row += gridDim.x) {
        const int b = row / g.oH, oy = row - b * g.oH;
        const int iy0 = oy * g.sY - g.pT;
        unsigned rbase[3];
        bool rok[3];
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
            const int iy = iy0 + ky * g.dY;
            rok[ky] = iy >= 0 && iy < g.H;
            rbase[ky] = (unsigned)((b * g.H + (rok[ky] ? iy : 0)) * g.W * cw);
        }
        const unsigned obase = (unsigned)(row * g.oW * cw);
        for (int chunk0 = 0; chunk0 < g.oW; chunk0 += 4 * xthreads) {
            const int ox0 = chunk0 + 4 * xi;       // pixels ox0 .. ox0 + 3
            int acc[4][4];
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[p][j] = 0;
            {
                unsigned coff[4][3];
                bool cok[4][3];
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int kx = 0; kx < 3; ++kx) {
                        const int ix = (ox0 + p) * g.sX - g.pL + kx * g.dX;
                        cok[p][kx] = ix >= 0 && ix < g.W;
                        coff[p][kx] = (unsigned)((cok[p][kx] ? ix : 0) * cw);
                    }
#pragma unroll
                for (int ky = 0; ky < 3; ++ky)
#pragma unroll
                    for (int p = 0; p < 4; ++p)
#pragma unroll
                        for (int kx = 0; kx < 3; ++kx) {
                            const unsigned xv = (rok[ky] && cok[p][kx]) ? __ldg(in_w + rbase[ky] + coff[p][kx]) : 0u;
                            dw_mac4<IN_UNSIGNED>(acc[p], xv, wm[ky * 3 + kx]);
                        }
            }
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                if (ox0 + p >= g.oW) break;
                int y[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    int x = acc[p][j];
                    if (CLAMP) x = min(max(x, lo[j]), hi[j]);
                    y[j] = (x * mu[j] + ad[j]) >> sh[j];
                }
                unsigned tmp, d;
                if (OUT_UNSIGNED) {
                    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(tmp) : "r"(y[3]), "r"(y[2]), "r"(y[2]));   // upper half shifted out below
                    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(y[1]), "r"(y[0]), "r"(tmp));
                } else {
                    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(tmp) : "r"(y[3]), "r"(y[2]), "r"(y[2]));   // upper half shifted out below
                    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(y[1]), "r"(y[0]), "r"(tmp));
                }
                out_w[obase + (unsigned)((ox0 + p) * cw)] = d;
            }
        }
    }
}

// Dilated filters and larger strides whose rescale has the proved 32-bit form: the masked dot-product kernel
static bool depthwise3x3_masked(const ConvGeom& g, const FastQuant& fast)
{
    const int cw = g.C / 4;
    const bool idx32 = (long long)g.B * g.H * g.W * cw < (1ll << 31) && (long long)g.B * g.oH * g.oW * cw < (1ll << 31);
    return fast.enabled && fast.form == 0 && g.kH == 3 && g.kW == 3 && 256 % cw == 0 && idx32;
}

int depthwise_alignment(const ConvGeom& g, const FastQuant& fast)
{
    return (fast.enabled && depthwise3x3_eligible(g)) || depthwise3x3_masked(g, fast) ? 4 : 16;
}

cudaError_t launch_conv_depthwise(const void* in, int in_unsigned, const int8_t* w_hwc,
                                  const ConvGeom& g, const QuantDev& q, const FastQuant& fast, void* out, cudaStream_t s)
{
    if (fast.enabled && depthwise3x3_eligible(g)) return launch_depthwise3x3(in, in_unsigned, w_hwc, g, fast, out, current_sms(), s);
    if (depthwise3x3_masked(g, fast)) {
        const int cw = g.C / 4;
        const long long rows = (long long)g.B * g.oH;
        if (rows == 0 || g.oW == 0) return cudaSuccess;
        // few, long-lived blocks: a thread's weights and constants (29 loads) are fetched once and serve many rows
        const long long max_blocks = 6ll * current_sms();
        const unsigned grid = (unsigned)(rows < max_blocks ? rows : max_blocks);
        // a block's threads cover 4 * (threads / cw) pixels of a row per pass
        int threads = 256;
        while (threads > 32 && (threads / 2) % cw == 0 && 4 * (threads / 2 / cw) >= g.oW) threads /= 2;
        const uint8_t* ip = (const uint8_t*)in;
        uint8_t* op = (uint8_t*)out;
#define N2D2B_DW(U, C, O) launch_pdl(conv_depthwise3x3_dp4a_kernel<U, C, O>, grid, threads, 0, s, ip, w_hwc, g, fast.fq, fast.cpad, op)
        const int v = (in_unsigned ? 4 : 0) | (fast.need_clamp ? 2 : 0) | (fast.out_unsigned ? 1 : 0);
        switch (v) {
        case 0: N2D2B_DW(false, false, false); break;
        case 1: N2D2B_DW(false, false, true); break;
        case 2: N2D2B_DW(false, true, false); break;
        case 3: N2D2B_DW(false, true, true); break;
        case 4: N2D2B_DW(true, false, false); break;
        case 5: N2D2B_DW(true, false, true); break;
        case 6: N2D2B_DW(true, true, false); break;
        default: N2D2B_DW(true, true, true); break;
        }
#undef N2D2B_DW
        return cudaGetLastError();
    }

    const size_t total = (size_t)g.B * g.oH * g.oW * (g.C / 16);
    if (total == 0) return cudaSuccess;
    const int block = 256;
    launch_pdl(conv_depthwise_kernel, grid_for(total, block), block, 0, s, (const uint8_t*)in, in_unsigned, w_hwc, g, q,
                                                                   (uint8_t*)out, total);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Pooling (PoolCell): max over the in-image taps (0 for an all-padding window); average with the
// full window as divisor and truncation toward zero, as the reference's quantized PoolCell does.
// Vector path: 16 channels per thread when C % 16 == 0 and the tensor is int8.
// ---------------------------------------------------------------------------------------------
__global__ void pool_vec_kernel(const uint8_t* __restrict__ in, int in_unsigned, PoolGeom g,
                                uint8_t* __restrict__ out, size_t total_vec)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    const int cv = g.C / 16;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total_vec;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int c16 = (int)(idx % cv);
        size_t p = idx / cv;
        const int ox = (int)(p % g.oW); p /= g.oW;
        const int oy = (int)(p % g.oH);
        const int b = (int)(p / g.oH);
        const int iy0 = oy * g.sY - g.padY, ix0 = ox * g.sX - g.padX;
        int v[16];
        bool valid = false;
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0;
        for (int ky = 0; ky < g.pH; ++ky) {
            const int iy = iy0 + ky;
            if (iy < 0 || iy >= g.H) continue;
            for (int kx = 0; kx < g.pW; ++kx) {
                const int ix = ix0 + kx;
                if (ix < 0 || ix >= g.W) continue;
                const uint4 xv = *(const uint4*)(in + (((size_t)b * g.H + iy) * g.W + ix) * g.C + c16 * 16);
                int xs[16];
                unpack16(xv, in_unsigned != 0, xs);
                if (g.is_max) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = (!valid || xs[i] > v[i]) ? xs[i] : v[i];
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] += xs[i];
                }
                valid = true;
            }
        }
        if (!g.is_max) {
            const int count = g.pH * g.pW;
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = v[i] / count;  // C division truncates toward zero
        }
        *(uint4*)(out + idx * 16) = pack16(v);
    }
}

// Max pooling, 16 channels per thread, one block per output row: the window bounds of the row are
// computed once, the maximum runs on four bytes at a time, and no thread divides 64-bit indices.
template <bool UNSIGNED>
__global__ void pool_max_row_kernel(const uint8_t* __restrict__ in, PoolGeom g, uint8_t* __restrict__ out)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    const int cv = g.C / 16;
    for (int row = blockIdx.x; row < g.B * g.oH; row += gridDim.x) {
        const int b = row / g.oH, oy = row - b * g.oH;
        const int iy0 = oy * g.sY - g.padY;
        const int ky_lo = iy0 < 0 ? -iy0 : 0;
        const int ky_hi = (g.H - iy0) < g.pH ? (g.H - iy0) : g.pH;
        const uint8_t* img = in + (size_t)b * g.H * g.W * g.C;
        uint8_t* orow = out + (size_t)row * g.oW * g.C;
        for (int t = threadIdx.x; t < g.oW * cv; t += blockDim.x) {
            const int ox = t / cv, c16 = t - ox * cv;
            const int ix0 = ox * g.sX - g.padX;
            const int kx_lo = ix0 < 0 ? -ix0 : 0;
            const int kx_hi = (g.W - ix0) < g.pW ? (g.W - ix0) : g.pW;
            uint4 m = make_uint4(0u, 0u, 0u, 0u);
            if (g.pH == 3 && g.pW == 3 && ky_lo == 0 && ky_hi == 3 && kx_lo == 0 && kx_hi == 3) {
                // a whole 3x3 window: nine independent loads in flight, then the maxima (the general loop below
                // would wait for each load in turn)
                const uint8_t* p = img + ((size_t)iy0 * g.W + ix0) * g.C + c16 * 16;
                const size_t rs = (size_t)g.W * g.C;
                uint4 x[9];
#pragma unroll
                for (int ky = 0; ky < 3; ++ky)
#pragma unroll
                    for (int kx = 0; kx < 3; ++kx) x[ky * 3 + kx] = __ldg((const uint4*)(p + ky * rs + (size_t)kx * g.C));
                m = x[0];
#pragma unroll
                for (int i = 1; i < 9; ++i) {
                    if (UNSIGNED) {
                        m.x = __vmaxu4(m.x, x[i].x); m.y = __vmaxu4(m.y, x[i].y);
                        m.z = __vmaxu4(m.z, x[i].z); m.w = __vmaxu4(m.w, x[i].w);
                    } else {
                        m.x = __vmaxs4(m.x, x[i].x); m.y = __vmaxs4(m.y, x[i].y);
                        m.z = __vmaxs4(m.z, x[i].z); m.w = __vmaxs4(m.w, x[i].w);
                    }
                }
                *(uint4*)(orow + (size_t)t * 16) = m;
                continue;
            }
            bool first = true;
            for (int ky = ky_lo; ky < ky_hi; ++ky) {
                const uint8_t* p = img + ((size_t)(iy0 + ky) * g.W + ix0) * g.C + c16 * 16;
                for (int kx = kx_lo; kx < kx_hi; ++kx) {
                    const uint4 xv = __ldg((const uint4*)(p + (size_t)kx * g.C));
                    if (first) {
                        m = xv;
                        first = false;
                    } else if (UNSIGNED) {
                        m.x = __vmaxu4(m.x, xv.x); m.y = __vmaxu4(m.y, xv.y);
                        m.z = __vmaxu4(m.z, xv.z); m.w = __vmaxu4(m.w, xv.w);
                    } else {
                        m.x = __vmaxs4(m.x, xv.x); m.y = __vmaxs4(m.y, xv.y);
                        m.z = __vmaxs4(m.z, xv.z); m.w = __vmaxs4(m.w, xv.w);
                    }
                }
            }
            *(uint4*)(orow + (size_t)t * 16) = m;   // an all-padding window stays 0
        }
    }
}

template <typename ElemT>
__global__ void pool_scalar_kernel(const void* __restrict__ in, int in_unsigned, PoolGeom g,
                                   void* __restrict__ out, size_t total)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(idx % g.C);
        size_t p = idx / g.C;
        const int ox = (int)(p % g.oW); p /= g.oW;
        const int oy = (int)(p % g.oH);
        const int b = (int)(p / g.oH);
        const int iy0 = oy * g.sY - g.padY, ix0 = ox * g.sX - g.padX;
        long long v = 0;
        bool valid = false;
        for (int ky = 0; ky < g.pH; ++ky) {
            const int iy = iy0 + ky;
            if (iy < 0 || iy >= g.H) continue;
            for (int kx = 0; kx < g.pW; ++kx) {
                const int ix = ix0 + kx;
                if (ix < 0 || ix >= g.W) continue;
                const size_t ii = (((size_t)b * g.H + iy) * g.W + ix) * g.C + c;
                long long x;
                if (sizeof(ElemT) == 4) x = ((const int32_t*)in)[ii];
                else x = load_i8(in, ii, in_unsigned != 0);
                if (g.is_max) v = (!valid || x > v) ? x : v;
                else v += x;
                valid = true;
            }
        }
        if (!g.is_max) v = v / (long long)(g.pH * g.pW);
        if (sizeof(ElemT) == 4) ((int32_t*)out)[idx] = (int32_t)v;
        else ((int8_t*)out)[idx] = (int8_t)v;
    }
}

// Average over the whole feature map (the pooling cell before the classifier): one thread per four channels of
// an image, so a warp reads 128 consecutive bytes per pixel and every load of the pixel loop is independent of
// the others.  Bytes are summed as two pairs of 16-bit lanes (signed inputs are biased to unsigned by flipping
// the top bit and un-biased at the end; up to 257 pixels fit a lane).  Divides by the window size and truncates
// toward zero like the reference's quantized cell.
template <bool UNSIGNED>
__global__ void pool_global_avg_kernel(const uint8_t* __restrict__ in, int pixels, int C, size_t total_words,
                                       uint8_t* __restrict__ out)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    const int cw = C / 4;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total_words; idx += (size_t)gridDim.x * blockDim.x) {
        const size_t b = idx / cw;
        const int w = (int)(idx - b * cw);
        const unsigned* p = (const unsigned*)(in + b * (size_t)pixels * C) + w;
        unsigned even = 0, odd = 0;   // bytes 0, 2 and bytes 1, 3 as 16-bit lanes
#pragma unroll 7
        for (int i = 0; i < pixels; ++i) {
            unsigned x = __ldg(p + (size_t)i * cw);
            if (!UNSIGNED) x ^= 0x80808080u;
            even += x & 0x00ff00ffu;
            odd += (x >> 8) & 0x00ff00ffu;
        }
        int v[4] = {(int)(even & 0xffffu), (int)(odd & 0xffffu), (int)(even >> 16), (int)(odd >> 16)};
        unsigned o = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!UNSIGNED) v[j] -= 128 * pixels;
            o |= ((unsigned)(v[j] / pixels) & 0xffu) << (8 * j);   // C division truncates toward zero
        }
        ((unsigned*)out)[idx] = o;
    }
}

cudaError_t launch_pool(const void* in, int in_unsigned, const PoolGeom& g, void* out, cudaStream_t s)
{
    // int8 tensors; int32 tensors go through launch_pool_i32
    const int block = 256;
    const bool vec = g.C % 16 == 0 && (((uintptr_t)in | (uintptr_t)out) & 15) == 0;   // (the input may be the caller's buffer)
    if (vec && g.is_max) {
        const long long rows = (long long)g.B * g.oH;
        if (rows == 0 || g.oW == 0) return cudaSuccess;
        const int items = g.oW * (g.C / 16);
        const int threads = items >= 256 ? 256 : ((items + 31) / 32) * 32;
        const unsigned grid = (unsigned)(rows < (1ll << 20) ? rows : (1ll << 20));
        if (in_unsigned) launch_pdl(pool_max_row_kernel<true>, grid, threads, 0, s, (const uint8_t*)in, g, (uint8_t*)out);
        else launch_pdl(pool_max_row_kernel<false>, grid, threads, 0, s, (const uint8_t*)in, g, (uint8_t*)out);
    } else if (!g.is_max && g.C % 4 == 0 && g.pH == g.H && g.pW == g.W && g.padY == 0 && g.padX == 0 && g.oH == 1 && g.oW == 1
               && g.H * g.W <= 257 && ((uintptr_t)in & 3) == 0 && ((uintptr_t)out & 3) == 0) {
        const size_t total = (size_t)g.B * (g.C / 4);
        if (total == 0) return cudaSuccess;
        if (in_unsigned)
            launch_pdl(pool_global_avg_kernel<true>, grid_for(total, block), block, 0, s, (const uint8_t*)in, g.H * g.W, g.C, total, (uint8_t*)out);
        else
            launch_pdl(pool_global_avg_kernel<false>, grid_for(total, block), block, 0, s, (const uint8_t*)in, g.H * g.W, g.C, total, (uint8_t*)out);
    } else if (vec) {
        const size_t total = (size_t)g.B * g.oH * g.oW * (g.C / 16);
        if (total == 0) return cudaSuccess;
        launch_pdl(pool_vec_kernel, grid_for(total, block), block, 0, s, (const uint8_t*)in, in_unsigned, g, (uint8_t*)out, total);
    } else {
        const size_t total = (size_t)g.B * g.oH * g.oW * g.C;
        if (total == 0) return cudaSuccess;
        launch_pdl(pool_scalar_kernel<int8_t>, grid_for(total, block), block, 0, s, in, in_unsigned, g, out, total);
    }
    return cudaGetLastError();
}

cudaError_t launch_pool_i32(const void* in, const PoolGeom& g, void* out, cudaStream_t s)
{
    const size_t total = (size_t)g.B * g.oH * g.oW * g.C;
    if (total == 0) return cudaSuccess;
    launch_pdl(pool_scalar_kernel<int32_t>, grid_for(total, 256), 256, 0, s, in, 0, g, out, total);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Element-wise sum of up to four tensors (ElemWiseCell, Sum, unit weights) followed by the cell's
// own requantisation; with a single input it is the stand-alone ScalingCell.
// ---------------------------------------------------------------------------------------------
template <typename OutT>
__global__ void elemwise_sum_kernel(SumInputs ins, size_t total, int C, QuantDev q, void* __restrict__ out)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(idx % C);
        long long x = 0;
        for (int k = 0; k < ins.n; ++k) {
            if (ins.dtype[k] == DT_I32) x += ((const int32_t*)ins.ptr[k])[idx];
            else x += load_i8(ins.ptr[k], idx, ins.is_unsigned[k] != 0);
        }
        if (q.bias) x += q.bias[c];
        store_out<OutT>(out, idx, requant64(x, c, q));
    }
}

// Fast path: two int8 inputs, int8 output, 16 values per thread.
__global__ void elemwise_sum2_vec_kernel(const uint8_t* __restrict__ a, int a_unsigned,
                                         const uint8_t* __restrict__ b, int b_unsigned, size_t total_vec,
                                         int C, QuantDev q, uint8_t* __restrict__ out)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total_vec;
         idx += (size_t)gridDim.x * blockDim.x) {
        const uint4 av = *(const uint4*)(a + idx * 16);
        const uint4 bv = *(const uint4*)(b + idx * 16);
        int xa[16], xb[16], y[16];
        unpack16(av, a_unsigned != 0, xa);
        unpack16(bv, b_unsigned != 0, xb);
        const int c0 = (int)((idx * 16) % C);
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = requant64((long long)xa[i] + xb[i], c0 + i, q);
        *(uint4*)(out + idx * 16) = pack16(y);
    }
}

cudaError_t launch_elemwise_sum(const SumInputs& ins, size_t pixels, int C, const QuantDev& q,
                                void* out, int out_dtype, cudaStream_t s)
{
    const size_t total = pixels * (size_t)C;
    if (total == 0) return cudaSuccess;
    const int block = 256;
    if (ins.n == 2 && out_dtype == DT_I8 && ins.dtype[0] == DT_I8 && ins.dtype[1] == DT_I8 && C % 16 == 0
        && !q.bias && (((uintptr_t)ins.ptr[0] | (uintptr_t)ins.ptr[1] | (uintptr_t)out) & 15) == 0) {
        launch_pdl(elemwise_sum2_vec_kernel, grid_for(total / 16, block), block, 0, s, 
            (const uint8_t*)ins.ptr[0], ins.is_unsigned[0], (const uint8_t*)ins.ptr[1], ins.is_unsigned[1],
            total / 16, C, q, (uint8_t*)out);
    } else if (out_dtype == DT_I8) {
        launch_pdl(elemwise_sum_kernel<int8_t>, grid_for(total, block), block, 0, s, ins, total, C, q, out);
    } else {
        launch_pdl(elemwise_sum_kernel<int32_t>, grid_for(total, block), block, 0, s, ins, total, C, q, out);
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Stand-alone rescale (n2d2b_scaling_propagate): int32 [pixels][C] -> 8 bits.  HBM-bound: 5 bytes per value.  The
// per-channel constants travel in the kernel's own parameters (up to 28 KB), so the call needs no device memory and no
// copy; a thread keeps the constants of its four channels in registers and walks rows that lie a whole number of channel
// periods apart.  Channel counts that are no multiple of four repeat their constants over lcm(4, C) values, so the loads
// stay 128 bits wide.  128 x 28 x 28 x 128 values (64 MB in and out): 0.119 ms as one thread per value with the exact
// 64-bit form and its constants fetched per value; with two cudaMalloc / cudaFree around it the call took 0.858 ms.
// ---------------------------------------------------------------------------------------------
static constexpr int RESCALE_MAX_C = 1024;   // channels per launch: seven words of constants each stay below the 32 KB of parameters
static constexpr int RESCALE_FEW = 1024;     // words of the small parameter block (the host copies the whole block per launch)

template <int WORDS>
struct RescaleArgs {
    const int32_t* in;
    uint8_t* out;
    unsigned long long total;   // values of the tensors
    long long rows;             // rows of `width` values (width = C, or lcm(4, C) over the flattened tensor)
    int ld, c0, width, C;       // value v of row r: index r * ld + c0 + v, channel v mod C
    int per_block;              // rows a block takes at once
    int out_lo, out_hi;         // FORM 2: what QuantDev holds
    int mode, act, is_clipped, sat_thr;
    int words[WORDS];   // FORM 0 / 1: [5][C] of the 32-bit / floating-point form; FORM 2: [7][C] (bias, p0, p1, fscale, clips)
};

// FORM 0: 32-bit form (clamped), 1: floating-point form (clamped), 2: exact 64-bit form
template <int FORM, int VEC, int WORDS>
__global__ void __launch_bounds__(1024) rescale_i32_kernel(const __grid_constant__ RescaleArgs<WORDS> a)
{
    // parameters indexed by the thread: read through a generic pointer, as coalesced loads instead of serialised
    // constant-bank accesses
    const int* words = a.words;
    asm volatile("" : "+l"(words));
    const int vq = a.width / VEC;
    const int q = threadIdx.x % vq, r0 = threadIdx.x / vq;
    int k[5][VEC], ch[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
        ch[j] = (q * VEC + j) % a.C;
        if (FORM != 2)
#pragma unroll
            for (int p = 0; p < 5; ++p) k[p][j] = words[p * a.C + ch[j]];
    }
    QuantDev qd;
    if (FORM == 2) {
        qd.mode = a.mode; qd.act = a.act; qd.saturate = 1; qd.out_lo = a.out_lo; qd.out_hi = a.out_hi;
        qd.is_clipped = a.is_clipped; qd.sat_thr = a.sat_thr; qd.bias = nullptr;
        qd.p0 = words + a.C; qd.p1 = words + 2 * a.C; qd.fscale = (const float*)(words + 3 * a.C);
        qd.clip_thr = words + 4 * a.C; qd.clip_val = words + 5 * a.C; qd.clip_f = (const float*)(words + 6 * a.C);
    }
    const bool out_unsigned = a.out_lo >= 0;
    auto one = [&](int x, int j) -> int {
        if (FORM == 0) return (min(max(x, k[0][j]), k[1][j]) * k[2][j] + k[3][j]) >> k[4][j];
        if (FORM == 1) return float_round_scaled(fminf(fmaxf(__int2float_rn(x), __int_as_float(k[0][j])), __int_as_float(k[1][j])),
                                                 __int_as_float(k[2][j]));
        return requant64((long long)x, ch[j], qd);
    };
    constexpr int U = 4;   // rows in flight per thread
    const long long step = (long long)gridDim.x * a.per_block;
    for (long long r = (long long)blockIdx.x * a.per_block + r0; r < a.rows; r += U * step) {
        int x[U][VEC];
        bool full[U];
        unsigned long long at[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long ru = r + u * step;
            at[u] = (unsigned long long)ru * (unsigned)a.ld + (unsigned)(a.c0 + q * VEC);
            full[u] = ru < a.rows && at[u] + VEC <= a.total;
            if constexpr (VEC == 4) {
                const int4 v = full[u] ? __ldcs((const int4*)(a.in + at[u])) : make_int4(0, 0, 0, 0);
                x[u][0] = v.x; x[u][1] = v.y; x[u][2] = v.z; x[u][3] = v.w;
            } else {
                x[u][0] = full[u] ? a.in[at[u]] : 0;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (full[u]) {
                if constexpr (VEC == 4) {
                    int y[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) y[j] = one(x[u][j], j);
                    *(unsigned*)(a.out + at[u]) = pack4_sat(y[0], y[1], y[2], y[3], out_unsigned);
                } else {
                    a.out[at[u]] = (uint8_t)pack4_sat(one(x[u][0], 0), 0, 0, 0, out_unsigned);
                }
            } else if (VEC == 4 && r + u * step < a.rows) {
                // the last values of a tensor that is no multiple of four
                for (int j = 0; j < VEC && at[u] + j < a.total; ++j)
                    a.out[at[u] + j] = (uint8_t)pack4_sat(one(a.in[at[u] + j], j), 0, 0, 0, out_unsigned);
            }
        }
    }
}

template <int WORDS>
static cudaError_t launch_rescale(const int32_t* in, void* out, size_t pixels, int C, int form, const int32_t* words, const QuantDev& q,
                                  cudaStream_t s)
{
    typedef void (*Kernel)(const RescaleArgs<WORDS>);
    static const Kernel kernels[6] = {rescale_i32_kernel<0, 1, WORDS>, rescale_i32_kernel<1, 1, WORDS>, rescale_i32_kernel<2, 1, WORDS>,
                                      rescale_i32_kernel<0, 4, WORDS>, rescale_i32_kernel<1, 4, WORDS>, rescale_i32_kernel<2, 4, WORDS>};
    const int np = form == 2 ? 7 : 5;
    RescaleArgs<WORDS> a;
    a.in = in;
    a.out = (uint8_t*)out;
    a.total = (unsigned long long)pixels * (unsigned)C;
    a.out_lo = q.out_lo; a.out_hi = q.out_hi; a.mode = q.mode; a.act = q.act; a.is_clipped = q.is_clipped; a.sat_thr = q.sat_thr;
    const bool aligned = !((uintptr_t)in & 15) && !((uintptr_t)out & 3);
    for (int c0 = 0; c0 < C; c0 += RESCALE_MAX_C) {
        const int n = C - c0 < RESCALE_MAX_C ? C - c0 : RESCALE_MAX_C;
        int vec;
        if (n == C) {
            // one launch: the flattened tensor in rows of lcm(4, C) values
            vec = aligned ? 4 : 1;
            const int mult = vec == 1 || C % 4 == 0 ? 1 : (C % 2 == 0 ? 2 : 4);
            a.width = C * mult;
            a.ld = a.width;
        } else {
            vec = aligned && C % 4 == 0 ? 4 : 1;
            a.width = n;
            a.ld = C;
        }
        a.rows = (long long)((n == C) ? (a.total + a.width - 1) / a.width : pixels);
        a.c0 = c0;
        a.C = n;
        for (int p = 0; p < np; ++p) std::copy(words + (size_t)p * C + c0, words + (size_t)p * C + c0 + n, a.words + (size_t)p * n);
        const int vq = a.width / vec;                    // at most 1024
        a.per_block = vq >= 256 ? 1 : 256 / vq;
        const long long blocks = (a.rows + a.per_block - 1) / a.per_block;
        const int threads = vq * a.per_block;
        const long long most = (long long)current_sms() * (2048 / threads > 16 ? 16 : 2048 / threads);   // resident blocks
        kernels[(vec == 4 ? 3 : 0) + form]<<<(unsigned)(blocks < most ? blocks : most), threads, 0, s>>>(a);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// words: [5][C] (form 0, 1) or [7][C] (form 2) constants on the host
cudaError_t launch_rescale_i32(const int32_t* in, void* out, size_t pixels, int C, int form, const int32_t* words, const QuantDev& q,
                               cudaStream_t s)
{
    if (pixels == 0 || C == 0) return cudaSuccess;
    if ((form == 2 ? 7 : 5) * C <= RESCALE_FEW) return launch_rescale<RESCALE_FEW>(in, out, pixels, C, form, words, q, s);
    return launch_rescale<7 * RESCALE_MAX_C>(in, out, pixels, C, form, words, q, s);
}

// ---------------------------------------------------------------------------------------------
// Fully connected on CUDA cores: one warp per (image, output), lanes stride over K, shuffle-reduce.
// ---------------------------------------------------------------------------------------------
template <typename OutT>
__global__ void fc_direct_kernel(const uint8_t* __restrict__ in, int in_unsigned,
                                 const int8_t* __restrict__ w, int B, int K, int O, QuantDev q,
                                 void* __restrict__ out)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    const int lane = threadIdx.x & 31;
    const size_t warp = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5;
    const size_t nwarps = ((size_t)gridDim.x * blockDim.x) >> 5;
    for (size_t idx = warp; idx < (size_t)B * O; idx += nwarps) {
        const int o = (int)(idx % O);
        const int b = (int)(idx / O);
        const uint8_t* ip = in + (size_t)b * K;
        const int8_t* wp = w + (size_t)o * K;
        int acc = 0;
        for (int k = lane; k < K; k += 32) acc += load_i8(ip, k, in_unsigned != 0) * (int)wp[k];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
        if (lane == 0) {
            const long long x = (long long)acc + (q.bias ? (long long)q.bias[o] : 0ll);
            store_out<OutT>(out, idx, requant64(x, o, q));
        }
    }
}

cudaError_t launch_fc_direct(const void* in, int in_unsigned, const int8_t* w, int B, int K, int O,
                             const QuantDev& q, void* out, int out_dtype, cudaStream_t s)
{
    const size_t total = (size_t)B * O;
    if (total == 0) return cudaSuccess;
    const int block = 256;
    const unsigned grid = grid_for(total * 32, block);
    if (out_dtype == DT_I8)
        launch_pdl(fc_direct_kernel<int8_t>, grid, block, 0, s, (const uint8_t*)in, in_unsigned, w, B, K, O, q, out);
    else
        launch_pdl(fc_direct_kernel<int32_t>, grid, block, 0, s, (const uint8_t*)in, in_unsigned, w, B, K, O, q, out);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Output edge: estimated label = the class with the highest score, the first one among equals
// (Target top-1, src/Target/Target_CUDA_kernels.cu:88-104 of the reference: `if (tmp > maxVal)`).
// One warp per (image, pixel); scores are [pixels][C] int8 or int32.
// ---------------------------------------------------------------------------------------------
// 8 bytes per thread when both row lengths allow it, bytes otherwise
template <typename V>
__global__ void drop_padded_columns_kernel(const V* __restrict__ src, int ld, V* __restrict__ dst, int C, size_t rows)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    const size_t total = rows * (size_t)C;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t r = i / (size_t)C;
        dst[i] = src[r * (size_t)ld + (i - r * (size_t)C)];
    }
}

cudaError_t launch_drop_padded_columns(const uint8_t* src, int ld, uint8_t* dst, int C, size_t rows, cudaStream_t s)
{
    if (rows == 0) return cudaSuccess;
    const bool vec = (C % 8 == 0) && (ld % 8 == 0) && !((uintptr_t)src & 7) && !((uintptr_t)dst & 7);
    const size_t total = vec ? rows * (size_t)(C / 8) : rows * (size_t)C;
    const int threads = 256;
    const int blocks = (int)std::min<size_t>((total + threads - 1) / threads, 8 * (size_t)current_sms());
    if (vec)
        launch_pdl(drop_padded_columns_kernel<uint2>, blocks, threads, 0, s, (const uint2*)src, ld / 8, (uint2*)dst, C / 8, rows);
    else
        launch_pdl(drop_padded_columns_kernel<uint8_t>, blocks, threads, 0, s, src, ld, dst, C, rows);
    return cudaGetLastError();
}

template <typename T>
__global__ void argmax_kernel(const T* __restrict__ scores, size_t pixels, int C, int32_t* __restrict__ labels,
                              int32_t* __restrict__ values)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    const int lane = threadIdx.x & 31;
    const size_t warps = (size_t)gridDim.x * (blockDim.x >> 5);
    for (size_t p = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); p < pixels; p += warps) {
        const T* row = scores + p * (size_t)C;
        int best = INT32_MIN, idx = 0x7fffffff;
        for (int c = lane; c < C; c += 32) {
            const int v = (int)row[c];
            if (v > best || idx == 0x7fffffff) { best = v; idx = c; }   // ascending c within a lane: the first of equals stays
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const int ob = __shfl_xor_sync(0xffffffffu, best, off), oi = __shfl_xor_sync(0xffffffffu, idx, off);
            if (oi != 0x7fffffff && (idx == 0x7fffffff || ob > best || (ob == best && oi < idx))) { best = ob; idx = oi; }
        }
        if (lane == 0) {
            labels[p] = idx;
            if (values) values[p] = best;
        }
    }
}

cudaError_t launch_argmax(const void* scores, int dtype, int is_unsigned, size_t pixels, int C, int32_t* labels, int32_t* values,
                          cudaStream_t s)
{
    if (pixels == 0 || C == 0) return cudaSuccess;
    const int block = 256;
    const unsigned grid = grid_for(pixels * 32, block);
    if (dtype == DT_I32) launch_pdl(argmax_kernel<int32_t>, grid, block, 0, s, (const int32_t*)scores, pixels, C, labels, values);
    else if (is_unsigned) launch_pdl(argmax_kernel<uint8_t>, grid, block, 0, s, (const uint8_t*)scores, pixels, C, labels, values);
    else launch_pdl(argmax_kernel<int8_t>, grid, block, 0, s, (const int8_t*)scores, pixels, C, labels, values);
    return cudaGetLastError();
}

// Target top-N (src/Target/Target_CUDA_kernels.cu:44-86).  The reference orders a pixel's scores with an exchange
// sort, "for x: for y: if (v[y] < v[x]) swap(x, y)", quadratic in the number of classes; among equal scores (int8
// logits tie all the time) the classes end in the order those exchanges leave.  That order has a closed form, which
// this kernel evaluates in O(topN x classes) per pixel:
//   * pass x = 0 leaves the minimum at position 0; every position where the running minimum dropped receives the
//     element the minimum displaced;
//   * every later pass x inserts element x into the descending prefix behind its equals, and each group of equal,
//     smaller scores gives its first element to the group below and takes the element coming from above, i.e. the
//     group is rotated by one.
// So a group of equal scores r, read in position order after pass 0, is a queue that appends on a score == r and
// moves its head to its tail on a score > r (when it holds more than one element).  The groups are emitted from the
// highest score down until topN entries are out.  One warp per pixel takes 32 classes at a time: pass 0 is a prefix
// minimum over (score, class), a block of classes without a score > r appends in parallel, and only the at most topN
// larger scores are walked one by one (33 images, 1000 classes, top 5: 94 us with both scans on one lane, 18 with a scan and two
// votes for every block, 13 since blocks that change nothing are passed over).
// Shared memory: three int arrays of C entries.  Output [image][k][pixel of the image], like the reference.
template <typename T>
__global__ void topn_kernel(const T* __restrict__ scores, size_t pixels, size_t hw, int C, int topN, int32_t* __restrict__ labels,
                            int32_t* __restrict__ values)
{
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    extern __shared__ int topn_smem[];
    int* val = topn_smem;
    int* ids = val + C;
    int* buf = ids + C;
    const int lane = threadIdx.x;
    const unsigned before = (1u << lane) - 1u;
    for (size_t p = blockIdx.x; p < pixels; p += gridDim.x) {
        const T* row = scores + p * (size_t)C;
        // pass 0: where the running minimum drops, the element it displaces moves in; the minimum ends at position 0.
        // key = score (biased to unsigned) and class: the smallest key is the first of the smallest scores
        const unsigned long long none = ~0ull;
        unsigned long long run = none;   // minimum of the blocks before this one
        // (eight blocks' loads at a time; a block whose smallest score is not below the running minimum drops nothing: most of them)
        int run_v = INT32_MAX;
        for (int s0 = 0; s0 < C; s0 += 256) {
            int ahead[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) ahead[j] = s0 + 32 * j + lane < C ? (int)row[s0 + 32 * j + lane] : INT32_MAX;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int c0 = s0 + 32 * j, c = c0 + lane, v = ahead[j];
                if (c0 >= C) break;
                if (c0 > 0 && __reduce_min_sync(0xffffffffu, v) >= run_v) {
                    if (c < C) {
                        val[c] = v;
                        ids[c] = c;
                    }
                    continue;
                }
                const unsigned long long own = c < C ? ((unsigned long long)((unsigned)v ^ 0x80000000u) << 32 | (unsigned)c) : none;
                unsigned long long inc = own;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const unsigned long long o = __shfl_up_sync(0xffffffffu, inc, off);
                    if (lane >= off && o < inc) inc = o;
                }
                unsigned long long prev = __shfl_up_sync(0xffffffffu, inc, 1);
                if (lane == 0 || run < prev) prev = run;
                if (c < C) {
                    const bool drop = c > 0 && own < prev;
                    val[c] = drop ? (int)((unsigned)(prev >> 32) ^ 0x80000000u) : v;
                    ids[c] = drop ? (int)(unsigned)prev : c;
                }
                const unsigned long long blk = __shfl_sync(0xffffffffu, inc, 31);
                if (blk < run) run = blk;
                run_v = (int)((unsigned)(run >> 32) ^ 0x80000000u);
            }
        }
        __syncwarp();
        if (lane == 0) {
            val[0] = (int)((unsigned)(run >> 32) ^ 0x80000000u);
            ids[0] = (int)(unsigned)run;
        }
        __syncwarp();
        const size_t img = p / hw, pix = p - img * hw;
        int32_t* lab = labels + img * (size_t)topN * hw + pix;
        int32_t* vout = values ? values + img * (size_t)topN * hw + pix : nullptr;
        int emitted = 0;
        long long prev = (long long)INT32_MAX + 1;
        while (emitted < topN) {
            // next group: the highest score below the previous group's, and its size
            int r = INT32_MIN, cnt = 0;
#pragma unroll 4
            for (int c = lane; c < C; c += 32) {
                const int v = val[c];
                if ((long long)v < prev) {
                    if (cnt == 0 || v > r) { r = v; cnt = 1; }
                    else if (v == r) ++cnt;
                }
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                const int orr = __shfl_xor_sync(0xffffffffu, r, off), oc = __shfl_xor_sync(0xffffffffu, cnt, off);
                if (oc) {
                    if (cnt == 0 || orr > r) { r = orr; cnt = oc; }
                    else if (orr == r) cnt += oc;
                }
            }
            if (cnt == 0) break;   // fewer than topN classes
            int h = 0, L = 0;      // head and length of the queue in buf[0, cnt)
            // blocks with a score of the group or above: their numbers first, without a vote per block
            for (int seg = 0; seg < C; seg += 1024) {
                unsigned mine = 0;
#pragma unroll 8
                for (int i = 0; i < 32; ++i) {
                    const int c = seg + 32 * i + lane;
                    if (c < C && val[c] >= r) mine |= 1u << i;
                }
                for (unsigned live = __reduce_or_sync(0xffffffffu, mine); live; live &= live - 1) {
                    const int c = seg + 32 * (__ffs(live) - 1) + lane;
                    const int v = c < C ? val[c] : INT32_MIN;
                    const unsigned in = __ballot_sync(0xffffffffu, c < C && v == r);
                    unsigned up = __ballot_sync(0xffffffffu, c < C && v > r);
                    if (up == 0) {
                        if (in & (1u << lane)) {
                            int t = h + L + __popc(in & before);
                            if (t >= cnt) t -= cnt;
                            buf[t] = ids[c];
                        }
                        L += __popc(in);
                    } else {
                        unsigned left = in | up;
                        while (left) {
                            // the elements up to the next larger score append, then that score turns the queue by one
                            const int u = up ? __ffs(up) - 1 : 32;
                            const unsigned run_in = in & left & (u < 32 ? (1u << u) - 1u : 0xffffffffu);
                            if (run_in & (1u << lane)) {
                                int t = h + L + __popc(run_in & before);
                                if (t >= cnt) t -= cnt;
                                buf[t] = ids[c];
                            }
                            L += __popc(run_in);
                            __syncwarp();
                            if (u < 32 && L > 1) {
                                if (L < cnt && lane == 0) {   // a full queue turns in place
                                    int t = h + L;
                                    if (t >= cnt) t -= cnt;
                                    buf[t] = buf[h];
                                }
                                if (++h == cnt) h = 0;
                            }
                            __syncwarp();
                            left = u < 31 ? left & ~((2u << u) - 1u) : 0u;
                            up = u < 31 ? up & ~((2u << u) - 1u) : 0u;
                        }
                    }
                }
            }
            __syncwarp();
            const int take = cnt < topN - emitted ? cnt : topN - emitted;
            for (int k = lane; k < take; k += 32) {
                int t = h + k;
                if (t >= cnt) t -= cnt;
                lab[(size_t)(emitted + k) * hw] = buf[t];
                if (vout) vout[(size_t)(emitted + k) * hw] = r;
            }
            emitted += cnt;
            prev = r;
            __syncwarp();
        }
        __syncwarp();
    }
}

// The same on 8-bit scores of up to 32 * NV classes, a lane's in its registers: key = (score + 1, from 1 to 256) << 10 | class, so that the smallest key is
// the first of the smallest scores and a group is found without a look at shared memory.  One warp's latencies bound it: 33 images, 1000 classes,
// top 5: 12.6 us a call with the scores in shared memory, 10.7 here.
template <typename T, int NV>
__global__ void __launch_bounds__(32) topn_bytes_kernel(const T* __restrict__ scores, size_t pixels, size_t hw, int C, int topN, int32_t* __restrict__ labels,
                                                        int32_t* __restrict__ values)
{
    constexpr int BIAS = sizeof(T) == 1 && T(-1) < T(0) ? 129 : 1;
    __shared__ unsigned short ids[32 * NV], buf[32 * NV];
    pdl_launch_dependents();
    pdl_wait();   // also before the stores: the previous kernel may still read the output buffer
    const int lane = threadIdx.x;
    const unsigned before = (1u << lane) - 1u;
    for (size_t p = blockIdx.x; p < pixels; p += gridDim.x) {
        const T* row = scores + p * (size_t)C;
        unsigned key[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) key[j] = 32 * j + lane < C ? (unsigned)((int)row[32 * j + lane] + BIAS) << 10 | (unsigned)(32 * j + lane) : 0xffffffffu;
        // pass 0 (see topn_kernel): where the running minimum drops, the element it displaces moves in
        unsigned run = 0xffffffffu;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            if (j > 0 && __reduce_min_sync(0xffffffffu, key[j]) >> 10 >= run >> 10) continue;   // drops nothing: most of them
            unsigned inc = key[j];
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const unsigned o = __shfl_up_sync(0xffffffffu, inc, off);
                if (lane >= off) inc = min(inc, o);
            }
            unsigned prev = __shfl_up_sync(0xffffffffu, inc, 1);
            prev = lane == 0 ? run : min(prev, run);
            if (32 * j + lane > 0 && key[j] < prev) key[j] = prev;
            run = min(run, __shfl_sync(0xffffffffu, inc, 31));
        }
        if (lane == 0) key[0] = run;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            if (32 * j + lane >= C) key[j] = 0u;   // below every score
            ids[32 * j + lane] = (unsigned short)(key[j] & 1023u);
        }
        __syncwarp();
        const size_t img = p / hw, pix = p - img * hw;
        int32_t* lab = labels + img * (size_t)topN * hw + pix;
        int32_t* vout = values ? values + img * (size_t)topN * hw + pix : nullptr;
        int emitted = 0;
        unsigned bound = 0xffffffffu;   // keys of the groups that are out start here
        while (emitted < topN) {
            unsigned top = 0;
#pragma unroll
            for (int j = 0; j < NV; ++j) top = max(top, key[j] < bound ? key[j] : 0u);
            const unsigned r = __reduce_max_sync(0xffffffffu, top) >> 10;
            if (r == 0) break;   // fewer than topN classes
            bound = r << 10;
            const unsigned above = (r + 1) << 10;
            unsigned ge = 0, gt = 0;   // bit j: this lane's score of block j is in the group or above, above
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                if (key[j] >= bound) ge |= 1u << j;
                if (key[j] >= above) gt |= 1u << j;
            }
            const int cnt = (int)__reduce_add_sync(0xffffffffu, (unsigned)__popc(ge & ~gt));
            int h = 0, L = 0;          // head and length of the queue in buf[0, cnt)
            for (unsigned live = __reduce_or_sync(0xffffffffu, ge); live; live &= live - 1) {
                const int j = __ffs(live) - 1, c = 32 * j + lane;
                const unsigned in = __ballot_sync(0xffffffffu, (ge & ~gt) >> j & 1u);
                unsigned up = __ballot_sync(0xffffffffu, gt >> j & 1u), left = in | up;
                while (left) {
                    // the elements up to the next larger score append, then that score turns the queue by one
                    const int u = up ? __ffs(up) - 1 : 32;
                    const unsigned run_in = in & left & (u < 32 ? (1u << u) - 1u : 0xffffffffu);
                    if (run_in & (1u << lane)) {
                        int t = h + L + __popc(run_in & before);
                        if (t >= cnt) t -= cnt;
                        buf[t] = ids[c];
                    }
                    L += __popc(run_in);
                    __syncwarp();
                    if (u < 32 && L > 1) {
                        if (L < cnt && lane == 0) {   // a full queue turns in place
                            int t = h + L;
                            if (t >= cnt) t -= cnt;
                            buf[t] = buf[h];
                        }
                        if (++h == cnt) h = 0;
                    }
                    __syncwarp();
                    left = u < 31 ? left & ~((2u << u) - 1u) : 0u;
                    up = u < 31 ? up & ~((2u << u) - 1u) : 0u;
                }
            }
            const int take = min(cnt, topN - emitted);
            for (int k = lane; k < take; k += 32) {
                int t = h + k;
                if (t >= cnt) t -= cnt;
                lab[(size_t)(emitted + k) * hw] = buf[t];
                if (vout) vout[(size_t)(emitted + k) * hw] = (int)r - BIAS;
            }
            emitted += cnt;
            __syncwarp();
        }
        __syncwarp();
    }
}

cudaError_t launch_topn(const void* scores, int dtype, int is_unsigned, size_t pixels, size_t hw, int C, int topN, int32_t* labels,
                        int32_t* values, cudaStream_t s)
{
    if (pixels == 0 || C == 0 || topN == 0) return cudaSuccess;
    const unsigned grid = (unsigned)std::min<size_t>(pixels, 16 * (size_t)current_sms());
    if (dtype != DT_I32 && C <= 1024) {
#define N2D2B_TOPN_BYTES(T)                                                                                                  \
    launch_pdl(C <= 128 ? topn_bytes_kernel<T, 4> : C <= 256 ? topn_bytes_kernel<T, 8> : C <= 512 ? topn_bytes_kernel<T, 16> \
                                                                                                  : topn_bytes_kernel<T, 32>, \
               grid, 32, 0, s, (const T*)scores, pixels, hw, C, topN, labels, values)
        return is_unsigned ? N2D2B_TOPN_BYTES(uint8_t) : N2D2B_TOPN_BYTES(int8_t);
#undef N2D2B_TOPN_BYTES
    }
    const size_t smem = (size_t)3 * C * sizeof(int);
#define N2D2B_TOPN(T)                                                                                                   \
    do {                                                                                                                \
        cudaError_t e = cudaFuncSetAttribute(topn_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);  \
        if (e != cudaSuccess) return e;                                                                                 \
        launch_pdl(topn_kernel<T>, grid, 32, smem, s, (const T*)scores, pixels, hw, C, topN, labels, values);                   \
    } while (0)
    if (dtype == DT_I32) N2D2B_TOPN(int32_t);
    else if (is_unsigned) N2D2B_TOPN(uint8_t);
    else N2D2B_TOPN(int8_t);
#undef N2D2B_TOPN
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Input edge: what the post-training quantization puts in front of the network
// (src/DeepNetQuantization.cpp:359-370: RangeAffineTransformation(Multiplies, 2^n - 1 or 2^(n-1) - 1) with
// Truncate): float stimuli [batch][channel][y][x] -> trunc(x * factor) as 8-bit [batch][y][x][channel].
// The product is a float32 multiply rounded to nearest, as on the reference's float tensors.
// ---------------------------------------------------------------------------------------------
// A block takes a run of pixels of the whole batch: it reads every channel plane along it (coalesced, all loads of a
// thread independent), collects the bytes in shared memory and writes them as words.  33 x 3 x 224 x 224: 28 us when
// every thread gathered one output byte through four 64-bit divisions.
static constexpr int STIM_THREADS = 256, STIM_BYTES = 3072;

__device__ __forceinline__ uint8_t quantize_stimulus(float x, float factor, int lo, int hi)
{
    const float v = truncf(__fmul_rn(x, factor));
    return (uint8_t)(int)fminf(fmaxf(v, (float)lo), (float)hi);
}

// CC: channels when known at compile time (0: any up to STIM_BYTES / STIM_THREADS).  `run` pixels per block, a multiple of 4
template <int CC>
__global__ void __launch_bounds__(STIM_THREADS)
quantize_stimuli_kernel(const float* __restrict__ in, int c_any, unsigned hw, unsigned pixels, int run, float factor, int lo, int hi,
                        uint8_t* __restrict__ out)
{
    __shared__ __align__(16) uint8_t bytes[STIM_BYTES];
    const int C = CC ? CC : c_any;
    for (unsigned p0 = blockIdx.x * (unsigned)run; p0 < pixels; p0 += gridDim.x * (unsigned)run) {
        const unsigned n = pixels - p0 < (unsigned)run ? pixels - p0 : (unsigned)run;
#pragma unroll 4
        for (unsigned i = threadIdx.x; i < n; i += STIM_THREADS) {
            const unsigned g = p0 + i, b = g / hw;
            const float* src = in + (size_t)b * C * hw + (g - b * hw);
#pragma unroll
            for (int c = 0; c < C; ++c) bytes[i * C + c] = quantize_stimulus(__ldcs(src + (size_t)c * hw), factor, lo, hi);
        }
        __syncthreads();
        uint8_t* dst = out + (size_t)p0 * C;   // a multiple of four bytes from the start
        const unsigned nb = n * C;
        if (((uintptr_t)out & 3) == 0) {
            for (unsigned i = threadIdx.x; i < nb / 4; i += STIM_THREADS) ((unsigned*)dst)[i] = ((const unsigned*)bytes)[i];
            for (unsigned i = (nb & ~3u) + threadIdx.x; i < nb; i += STIM_THREADS) dst[i] = bytes[i];
        } else {
            for (unsigned i = threadIdx.x; i < nb; i += STIM_THREADS) dst[i] = bytes[i];
        }
        __syncthreads();
    }
}

// many channels, or more pixels than 32 bits count: one thread per output byte
__global__ void quantize_stimuli_any_kernel(const float* __restrict__ in, int C, size_t hw, size_t total, float factor, int lo, int hi,
                                            uint8_t* __restrict__ out)
{
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        const size_t g = idx / C, b = g / hw;
        const int c = (int)(idx - g * C);
        out[idx] = quantize_stimulus(in[(b * C + c) * hw + (g - b * hw)], factor, lo, hi);
    }
}

cudaError_t launch_quantize_stimuli(const float* in, int B, int C, int H, int W, float factor, int lo, int hi, void* out, cudaStream_t s)
{
    const size_t hw = (size_t)H * W, pixels = (size_t)B * hw, total = pixels * C;
    if (total == 0) return cudaSuccess;
    if (C > STIM_BYTES / STIM_THREADS || pixels >= (1ull << 31)) {
        quantize_stimuli_any_kernel<<<grid_for(total, 256), 256, 0, s>>>(in, C, hw, total, factor, lo, hi, (uint8_t*)out);
        return cudaGetLastError();
    }
    // up to four pixels per thread; fewer when the blocks would not cover the GPU twice
    int run = STIM_BYTES / C & ~(STIM_THREADS - 1);
    if (run > 4 * STIM_THREADS) run = 4 * STIM_THREADS;
    const size_t twice = 8 * (size_t)current_sms();
    while (run > STIM_THREADS && (pixels + run - 1) / run < twice) run -= STIM_THREADS;
    const size_t blocks = (pixels + run - 1) / run;
    const unsigned grid = (unsigned)std::min<size_t>(blocks, 1u << 20);
    if (C == 3) quantize_stimuli_kernel<3><<<grid, STIM_THREADS, 0, s>>>(in, C, (unsigned)hw, (unsigned)pixels, run, factor, lo, hi, (uint8_t*)out);
    else if (C == 1) quantize_stimuli_kernel<1><<<grid, STIM_THREADS, 0, s>>>(in, C, (unsigned)hw, (unsigned)pixels, run, factor, lo, hi, (uint8_t*)out);
    else quantize_stimuli_kernel<0><<<grid, STIM_THREADS, 0, s>>>(in, C, (unsigned)hw, (unsigned)pixels, run, factor, lo, hi, (uint8_t*)out);
    return cudaGetLastError();
}

}  // namespace n2d2b
