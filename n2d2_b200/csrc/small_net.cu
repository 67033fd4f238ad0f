// A whole small network in one kernel.
//
// A network like the reference's MNIST models (a few hundred thousand multiply-accumulates and tens of kilobytes of weights per
// image) spends its time between the cells, not in them: six launches of 3 to 14 us for 0.2 us of arithmetic.  Here a
// CTA keeps the weights and rescale constants of every cell in shared memory, takes one image (or four) through all
// cells with a barrier between two, and writes only the final tensor; nothing else reaches HBM.
//
// Layout.  Every cell's input sits in shared memory as NHWC bytes with the cell's zero padding written out around it, so a
// filter row of a window is one run of kW * C bytes and no tap needs a bounds check.  Runs are cut into 32-bit words (the tail
// meets zero weights); the weights are stored as [kH * words][outputs], word k of output o holding four consecutive
// values, so that the lanes of a warp - consecutive outputs of one pixel - read consecutive words, and the activation
// word is a broadcast.  One thread computes one output, or two neighbouring ones when a cell has more outputs than the
// CTA has threads, with dp4a.  What bounds a pass is shared-memory bandwidth (two words per dp4a); four images per pass
// share every weight word.
#include <cstring>
#include <algorithm>
#include <vector>
#include <atomic>
#include "kernels.h"
#include "tc_common.cuh"

namespace n2d2b {

static constexpr int SN_THREADS = 512;
static constexpr int SN_SMEM_MAX = 220 * 1024;

// Quotient by a run-time constant: exact for n * d < 2^32 (rcp = ceil(2^32 / d))
__device__ __forceinline__ unsigned sn_div(unsigned n, unsigned d, unsigned rcp) { return d == 1 ? n : __umulhi(n, rcp); }

__device__ __forceinline__ int sn_requant(int acc, int o, const SmallCell& c, const int* cst)
{
    if (c.form < 0) return requant64((long long)acc + (c.q.bias ? (long long)__ldg(c.q.bias + o) : 0ll), o, c.q);
    const int lo = cst[o], hi = cst[c.Opad + o], mu = cst[2 * c.Opad + o], ad = cst[3 * c.Opad + o], sh = cst[4 * c.Opad + o];
    int y;
    if (c.form == EF_FLOAT) y = rescale<true, EF_FLOAT>(acc, lo, hi, mu, ad, sh);
    else if (c.form == EF_WIDE) y = rescale<false, EF_WIDE>(acc, lo, hi, mu, ad, sh);
    else y = rescale<true, 0>(acc, lo, hi, mu, ad, sh);
    return c.out_unsigned ? min(max(y, 0), 255) : min(max(y, -128), 127);
}

// Outputs o .. o + RO - 1 of one pixel of IPB images; p: first byte of the window in the first image
template <int IPB, int RO, bool UNSIGNED>
__device__ __forceinline__ void sn_conv_item(const SmallCell& c, const unsigned* wp, const uint8_t* p, int act_stride, int (&acc)[IPB][RO])
{
    auto mac = [&](int i, unsigned x, const unsigned (&wv)[RO]) {
#pragma unroll
        for (int r = 0; r < RO; ++r) acc[i][r] = UNSIGNED ? dp4a_us(x, (int)wv[r], acc[i][r]) : dp4a_ss((int)x, (int)wv[r], acc[i][r]);
    };
    auto weights = [&](unsigned (&wv)[RO]) {
        if constexpr (RO == 2) {
            const uint2 t = *(const uint2*)wp;
            wv[0] = t.x;
            wv[1] = t.y;
        } else {
            wv[0] = *wp;
        }
        wp += c.Opad;
    };
    for (int ky = 0; ky < c.kH; ++ky, p += c.step_ky) {
        if (c.aligned) {
#pragma unroll 4
            for (int j = 0; j < c.words; ++j) {
                unsigned wv[RO];
                weights(wv);
#pragma unroll
                for (int i = 0; i < IPB; ++i) mac(i, *(const unsigned*)(p + 4 * j + i * act_stride), wv);
            }
        } else {
            const unsigned off = (unsigned)((uintptr_t)p & 3u);
            unsigned cur[IPB];
#pragma unroll
            for (int i = 0; i < IPB; ++i) cur[i] = *(const unsigned*)(p - off + i * act_stride);
            for (int j = 0; j < c.words; ++j) {
                unsigned wv[RO];
                weights(wv);
#pragma unroll
                for (int i = 0; i < IPB; ++i) {
                    const unsigned nxt = *(const unsigned*)(p - off + 4 * (j + 1) + i * act_stride);
                    mac(i, __funnelshift_r(cur[i], nxt, 8u * off), wv);
                    cur[i] = nxt;
                }
            }
        }
    }
}

template <int IPB, int RO, bool UNSIGNED>
__device__ __forceinline__ void sn_conv(const SmallCell& c, const uint8_t* blob, uint8_t* acts, int act_stride, int nimg, uint8_t* const (&out)[2],
                                        size_t out_stride)
{
    const unsigned oq = (unsigned)c.Opad / RO;     // groups of RO outputs per pixel
    const unsigned items = oq * (unsigned)(c.oH * c.oW);
    const unsigned rcp_q = RO == 2 ? c.rcp_O2 : c.rcp_O;
    for (unsigned it = threadIdx.x; it < items; it += SN_THREADS) {
        const unsigned pix = sn_div(it, oq, rcp_q), o = (it - pix * oq) * RO;
        const unsigned oy = sn_div(pix, (unsigned)c.oW, c.rcp_oW), ox = pix - oy * (unsigned)c.oW;
        int acc[IPB][RO];
#pragma unroll
        for (int i = 0; i < IPB; ++i)
#pragma unroll
            for (int r = 0; r < RO; ++r) acc[i][r] = 0;
        sn_conv_item<IPB, RO, UNSIGNED>(c, (const unsigned*)(blob + c.w_off) + o, acts + c.in_off + oy * c.step_y + ox * c.step_x, act_stride, acc);
#pragma unroll
        for (int r = 0; r < RO; ++r) {
            if ((int)o + r >= c.O) break;
#pragma unroll
            for (int i = 0; i < IPB; ++i) {
                const int y = sn_requant(acc[i][r], (int)o + r, c, (const int*)(blob + c.cst_off));
                if (!c.last) {
                    acts[c.out_off + oy * c.out_row + ox * c.O + o + r + i * act_stride] = (uint8_t)y;
                } else if (i < nimg) {
                    const size_t at = (size_t)i * out_stride + pix * (size_t)c.O + o + r;
                    out[0][at] = (uint8_t)y;
                    if (out[1]) out[1][at] = (uint8_t)y;
                }
            }
        }
    }
}

template <int IPB>
__device__ __forceinline__ void sn_pool(const SmallCell& c, uint8_t* acts, int act_stride, int nimg, uint8_t* const (&out)[2], size_t out_stride)
{
    const unsigned items = (unsigned)(c.O * c.oH * c.oW);
    for (unsigned it = threadIdx.x; it < items; it += SN_THREADS) {
        const unsigned pix = sn_div(it, (unsigned)c.O, c.rcp_O), o = it - pix * (unsigned)c.O;
        const int oy = (int)sn_div(pix, (unsigned)c.oW, c.rcp_oW), ox = (int)pix - oy * c.oW;
        const int y0 = max(oy * c.sY - c.padY, 0), y1 = min(oy * c.sY - c.padY + c.kH, c.inH);
        const int x0 = max(ox * c.sX - c.padX, 0), x1 = min(ox * c.sX - c.padX + c.kW, c.inW);
#pragma unroll 1
        for (int i = 0; i < IPB; ++i) {
            const uint8_t* in = acts + c.in_off + i * act_stride + o;
            int v = 0;
            bool any = false;
            for (int y = y0; y < y1; ++y)
                for (int x = x0; x < x1; ++x) {
                    const int b = load_i8(in, (size_t)(y * c.inW + x) * c.O, c.in_unsigned != 0);
                    v = c.is_max ? ((!any || b > v) ? b : v) : v + b;
                    any = true;
                }
            if (!c.is_max) v /= c.kH * c.kW;   // truncates toward zero, the full window as divisor
            if (!c.last) {
                acts[c.out_off + oy * c.out_row + ox * c.O + o + i * act_stride] = (uint8_t)v;
            } else if (i < nimg) {
                const size_t at = (size_t)i * out_stride + it;
                out[0][at] = (uint8_t)v;
                if (out[1]) out[1][at] = (uint8_t)v;
            }
        }
    }
}

template <int IPB>
__global__ void __launch_bounds__(SN_THREADS) small_net_kernel(const __grid_constant__ SmallNetArgs a, const uint8_t* in, int batch, uint8_t* out,
                                                               uint8_t* out2)
{
    extern __shared__ __align__(16) uint8_t smem[];
    uint8_t* const acts = smem + a.blob_bytes;
    pdl_launch_dependents();
    // weights and constants, asynchronously: nothing of an earlier kernel is in them
    for (int i = threadIdx.x * 16; i < a.blob_bytes; i += SN_THREADS * 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem + i)), "l"(a.blob + i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int i = threadIdx.x * 4; i < IPB * a.act_stride; i += SN_THREADS * 4) *(unsigned*)(acts + i) = 0u;   // the padding borders stay zero
    pdl_wait();
    __syncthreads();
    for (int img = blockIdx.x * IPB; img < batch; img += gridDim.x * IPB) {
        const int nimg = batch - img < IPB ? batch - img : IPB;
        const uint8_t* src = in + (size_t)img * a.in_bytes;
        if (a.in_words && !((uintptr_t)in & 3)) {
            const unsigned n = (unsigned)a.in_bytes / 4u * (unsigned)nimg, per = (unsigned)a.in_bytes / 4u;
            for (unsigned i = threadIdx.x; i < n; i += SN_THREADS) {
                const unsigned k = IPB == 1 ? 0u : i / per;
                *(unsigned*)(acts + a.cell[0].in_off + k * a.act_stride + 4 * (i - k * per)) = __ldg((const unsigned*)src + i);
            }
        } else {
            const unsigned rb = (unsigned)a.in_row, n = (unsigned)a.in_bytes * (unsigned)nimg;
            for (unsigned i = threadIdx.x; i < n; i += SN_THREADS) {
                const unsigned k = i / (unsigned)a.in_bytes, j = i - k * (unsigned)a.in_bytes, r = j / rb;
                acts[a.in_place + k * a.act_stride + r * a.in_pitch + (j - r * rb)] = src[i];
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        uint8_t* const dst[2] = {out + (size_t)img * a.out_bytes, out2 ? out2 + (size_t)img * a.out_bytes : nullptr};
#pragma unroll 1
        for (int l = 0; l < a.nb_cells; ++l) {
            const SmallCell& c = a.cell[l];
            if (c.pool) sn_pool<IPB>(c, acts, a.act_stride, nimg, dst, (size_t)a.out_bytes);
            else if (c.two) {
                if (c.in_unsigned) sn_conv<IPB, 2, true>(c, smem, acts, a.act_stride, nimg, dst, (size_t)a.out_bytes);
                else sn_conv<IPB, 2, false>(c, smem, acts, a.act_stride, nimg, dst, (size_t)a.out_bytes);
            } else {
                if (c.in_unsigned) sn_conv<IPB, 1, true>(c, smem, acts, a.act_stride, nimg, dst, (size_t)a.out_bytes);
                else sn_conv<IPB, 1, false>(c, smem, acts, a.act_stride, nimg, dst, (size_t)a.out_bytes);
            }
            __syncthreads();
        }
    }
}

// ----------------------------------------------------------------------------- host side
static unsigned rcp32(unsigned d) { return d <= 1 ? 0u : (unsigned)(((1ull << 32) + d - 1) / d); }
static int round16(int n) { return (n + 15) & ~15; }

// A convolution (or fully-connected) cell: w is OHWI int8.  Appends its weights and constants to `blob` and its input to the activation area.
// in_pad: the cell's padding (top, left, bottom, right as far as any window reaches).
void small_net_add_conv(SmallNetPlan* p, const ConvGeom& g, int in_unsigned, int out_unsigned, const int8_t* w, int form, const int32_t* consts,
                        int cpad, const QuantDev& q)
{
    SmallCell c;
    memset(&c, 0, sizeof(c));
    const int run = g.kW * g.C;
    c.words = (run + 3) / 4;
    c.O = g.O;
    c.Opad = (g.O + 1) & ~1;
    c.kH = g.kH;
    c.kW = g.kW;
    c.oH = g.oH; c.oW = g.oW;
    // the padded input as far as any window reaches
    const int Wp = std::max(g.W + g.pL, (g.oW - 1) * g.sX + g.kW), Hp = std::max(g.H + g.pT, (g.oH - 1) * g.sY + (g.kH - 1) * g.dY + 1);
    const int pitch = Wp * g.C;
    c.step_x = g.sX * g.C;
    c.step_y = g.sY * pitch;
    c.step_ky = g.dY * pitch;
    c.aligned = (c.step_x % 4 == 0 && c.step_y % 4 == 0 && c.step_ky % 4 == 0) ? 1 : 0;
    c.rcp_O = rcp32((unsigned)c.Opad);
    c.rcp_O2 = rcp32((unsigned)c.Opad / 2);
    c.rcp_oW = rcp32((unsigned)g.oW);
    c.two = (long long)c.Opad * g.oH * g.oW > SN_THREADS ? 1 : 0;
    c.in_unsigned = in_unsigned;
    c.out_unsigned = out_unsigned;
    c.form = form;
    c.q = q;
    c.w_off = (int)p->blob.size();
    p->blob.resize(c.w_off + round16(g.kH * c.words * c.Opad * 4), 0);
    for (int o = 0; o < g.O; ++o)
        for (int ky = 0; ky < g.kH; ++ky)
            for (int i = 0; i < run; ++i)
                p->blob[c.w_off + ((size_t)(ky * c.words + i / 4) * c.Opad + o) * 4 + i % 4] = (uint8_t)w[((size_t)o * g.kH + ky) * run + i];
    c.cst_off = (int)p->blob.size();
    if (form >= 0) {
        p->blob.resize(c.cst_off + round16(5 * c.Opad * 4), 0);
        for (int r = 0; r < 5; ++r) memcpy(&p->blob[c.cst_off + (size_t)r * c.Opad * 4], consts + (size_t)r * cpad, (size_t)g.O * 4);
    }
    c.in_off = p->act_bytes;
    small_net_link(p, g.pT, g.pL, pitch, g.W * g.C, g.C, g.H, g.W, g.C);
    p->act_bytes += round16(Hp * pitch + 8);   // an unaligned run reads up to one word past its end
    p->cells.push_back(c);
}

void small_net_add_pool(SmallNetPlan* p, const PoolGeom& g, int in_unsigned)
{
    SmallCell c;
    memset(&c, 0, sizeof(c));
    c.pool = 1;
    c.is_max = g.is_max;
    c.O = g.C;
    c.kH = g.pH; c.kW = g.pW;
    c.oH = g.oH; c.oW = g.oW;
    c.inH = g.H; c.inW = g.W;
    c.sY = g.sY; c.sX = g.sX; c.padY = g.padY; c.padX = g.padX;
    c.rcp_O = rcp32((unsigned)g.C);
    c.rcp_oW = rcp32((unsigned)g.oW);
    c.in_unsigned = in_unsigned;
    c.in_off = p->act_bytes;
    small_net_link(p, 0, 0, g.W * g.C, g.W * g.C, g.C, g.H, g.W, g.C);
    p->act_bytes += round16(g.H * g.W * g.C + 8);
    p->cells.push_back(c);
}

// Points the previous cell's output (or the network input) at the input area the next cell is about to get
void small_net_link(SmallNetPlan* p, int pT, int pL, int pitch, int row_bytes, int pixel, int H, int W, int C)
{
    const int place = p->act_bytes + pT * pitch + pL * pixel;
    if (p->cells.empty()) {
        p->in_place = place;
        p->in_pitch = pitch;
        p->in_row = row_bytes;
        p->in_bytes = H * W * C;
        p->in_words = (pT == 0 && pL == 0 && pitch == row_bytes && p->in_bytes % 4 == 0) ? 1 : 0;
    } else {
        SmallCell& prev = p->cells.back();
        prev.out_off = place;
        // a fully-connected cell takes the map as one row: the rows then follow each other without padding
        prev.out_row = (H == 1 && W == 1) ? prev.oW * prev.O : pitch;
    }
}

bool small_net_finish(SmallNetPlan* p, int out_bytes)
{
    if (p->cells.size() < 2 || p->cells.size() > SMALL_NET_CELLS) return false;
    p->cells.back().last = 1;
    p->out_bytes = out_bytes;
    p->blob.resize(round16((int)p->blob.size()), 0);
    p->act_bytes = round16(p->act_bytes);
    if (p->blob.size() + p->act_bytes > (size_t)SN_SMEM_MAX) return false;
    p->group = p->blob.size() + 4 * (size_t)p->act_bytes <= (size_t)SN_SMEM_MAX ? 4 : 1;
    return true;
}

cudaError_t launch_small_net(const SmallNetPlan& p, const void* d_blob, const void* in, int batch, void* out, void* out2, int num_sms, cudaStream_t s)
{
    SmallNetArgs a;
    memset(&a, 0, sizeof(a));
    a.nb_cells = (int)p.cells.size();
    for (int i = 0; i < a.nb_cells; ++i) a.cell[i] = p.cells[i];
    a.blob = (const uint8_t*)d_blob;
    a.blob_bytes = (int)p.blob.size();
    a.act_stride = p.act_bytes;
    a.in_bytes = p.in_bytes; a.in_place = p.in_place; a.in_pitch = p.in_pitch; a.in_row = p.in_row; a.in_words = p.in_words;
    a.out_bytes = p.out_bytes;
    static std::atomic<bool> attr_set[64];   // set twice by racing first calls at worst: harmless
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(small_net_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, SN_SMEM_MAX);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(small_net_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, SN_SMEM_MAX);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    // one image per CTA while that gives every image a CTA at once, four per pass beyond
    const size_t smem1 = p.blob.size() + p.act_bytes, smem4 = p.blob.size() + 4 * (size_t)p.act_bytes;
    const int per_sm1 = smem1 <= 110 * 1024 ? 2 : 1, per_sm4 = smem4 <= 110 * 1024 ? 2 : 1;
    if (batch <= num_sms * per_sm1 || p.group == 1) {
        const int grid = std::min(batch, num_sms * per_sm1);
        return launch_pdl(small_net_kernel<1>, grid, SN_THREADS, smem1, s, a, (const uint8_t*)in, batch, (uint8_t*)out, (uint8_t*)out2);
    }
    const int grid = std::min((batch + 3) / 4, num_sms * per_sm4);
    return launch_pdl(small_net_kernel<4>, grid, SN_THREADS, smem4, s, a, (const uint8_t*)in, batch, (uint8_t*)out, (uint8_t*)out2);
}

}  // namespace n2d2b
