// A whole small network in one kernel.
//
// A network like the reference's MNIST models (a few hundred thousand multiply-accumulates and tens of kilobytes of weights per
// image) spends its time between the cells, not in them: six launches of 3 to 14 us for 0.2 us of arithmetic.  Here a
// CTA keeps the weights and rescale constants of every cell in shared memory, takes one image (or four) through all
// cells with a barrier between two, and writes only the final tensor; nothing else reaches HBM.
//
// Layout.  Every cell's input sits in shared memory as NHWC bytes with the cell's zero padding written out around it, so a
// filter row of a window is one run of kW * C bytes and no tap needs a bounds check.  Runs are cut into 32-bit words (the tail
// meets zero weights; cells whose windows start on any byte keep four copies of their input, see sn_put); the weights are stored as [kH * words][outputs], word k of output o holding four consecutive
// values, so that the lanes of a warp - consecutive outputs of one pixel - read consecutive words, and the activation
// word is a broadcast.  A thread computes two neighbouring outputs with dp4a; a cell with fewer outputs than threads deals the
// words of a window out to up to eight of them.  What bounds a pass is the latency of its cells in turn, then
// shared-memory bandwidth (three words per two dp4a); four images per pass share every weight word.
#include <cstring>
#include <algorithm>
#include <vector>
#include "kernels.h"
#include "tc_common.cuh"

namespace n2d2b {

static constexpr int SN_THREADS = 512;
static constexpr int SN_SMEM_MAX = 220 * 1024;

// Quotient by a run-time constant: exact for n * d < 2^32 (rcp = ceil(2^32 / d))
__device__ __forceinline__ unsigned sn_div(unsigned n, unsigned d, unsigned rcp) { return d == 1 ? n : __umulhi(n, rcp); }

__device__ __noinline__ int sn_requant_exact(int acc, int o, const QuantDev& q)
{
    return requant64((long long)acc + (q.bias ? (long long)__ldg(q.bias + o) : 0ll), o, q);
}

// Two neighbouring outputs of one pixel of IPB images.  p: first word of this thread's part of the window in the first image, wp:
// the outputs' weights there; n words of each filter row, `split` apart (the row is dealt out to that many threads).
template <int IPB, bool UNSIGNED>
__device__ __forceinline__ void sn_conv_item(int n, int kH, int step_ky, int wstep, const unsigned* wp, const uint8_t* p, int act_stride, int split,
                                             int (&acc)[IPB][2])
{
    auto mac = [&](int i, unsigned x, const uint2& w) {
        acc[i][0] = UNSIGNED ? dp4a_us(x, (int)w.x, acc[i][0]) : dp4a_ss((int)x, (int)w.x, acc[i][0]);
        acc[i][1] = UNSIGNED ? dp4a_us(x, (int)w.y, acc[i][1]) : dp4a_ss((int)x, (int)w.y, acc[i][1]);
    };
    for (int ky = 0; ky < kH; ++ky, p += step_ky) {
        const unsigned* x = (const unsigned*)p;
        int j = 0;
        for (; j + 4 <= n; j += 4, x += 4 * split, wp += 4 * wstep) {   // four words in flight
            uint2 w[4];
            unsigned v[4][IPB];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                w[k] = *(const uint2*)(wp + k * wstep);
#pragma unroll
                for (int i = 0; i < IPB; ++i) v[k][i] = *(const unsigned*)((const uint8_t*)(x + k * split) + i * act_stride);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int i = 0; i < IPB; ++i) mac(i, v[k][i], w[k]);
        }
        for (; j < n; ++j, x += split, wp += wstep) {
            const uint2 w = *(const uint2*)wp;
#pragma unroll
            for (int i = 0; i < IPB; ++i) mac(i, *(const unsigned*)((const uint8_t*)x + i * act_stride), w);
        }
    }
}

// One byte of the next cell's input.  A cell whose windows start on any byte keeps four copies of its input, copy k moved k
// bytes down: the word at byte b is then an aligned word of copy b mod 4.
__device__ __forceinline__ void sn_put(uint8_t* at, int copies, int copy_stride, int v)
{
    *at = (uint8_t)v;
    for (int k = 1; k < copies; ++k) at[k * copy_stride - k] = (uint8_t)v;
}

template <int IPB, bool UNSIGNED>
__device__ __forceinline__ void sn_conv(const SmallCell& cell, const uint8_t* blob, uint8_t* acts, int act_stride, int nimg, uint8_t* const (&out)[2],
                                        size_t out_stride)
{
    // The description's fields, all at once: they sit in the shared memory that the outputs are stored to, and read one by one
    // between those stores they cost a cell 1000 cycles
    const int opad = cell.Opad, O = cell.O, oW = cell.oW, kH = cell.kH, step_x = cell.step_x, step_y = cell.step_y, step_ky = cell.step_ky;
    const int log_split = cell.log_split, n = cell.words >> log_split, in_off = cell.in_off, copy_stride = cell.copy_stride, form = cell.form;
    const int last = cell.last, out_off = cell.out_off, out_row = cell.out_row, out_copies = cell.out_copies, out_copy_stride = cell.out_copy_stride;
    const unsigned rcp_O = cell.rcp_O, rcp_oW = cell.rcp_oW;
    const int sat_lo = cell.out_unsigned ? 0 : -128, sat_hi = cell.out_unsigned ? 255 : 127;
    const unsigned* const w0 = (const unsigned*)(blob + cell.w_off);
    const int* const cst = (const int*)(blob + cell.cst_off);
    const unsigned oq = (unsigned)opad / 2;     // pairs of outputs per pixel
    const unsigned items = oq * (unsigned)(cell.oH * oW), split = 1u << log_split;
    for (unsigned base = 0; base < (items << log_split); base += SN_THREADS) {
        const unsigned it = (base + threadIdx.x) >> log_split, part = threadIdx.x & (split - 1);
        const bool valid = it < items;
        const unsigned pix = sn_div(valid ? it : 0u, oq, rcp_O), o = ((valid ? it : 0u) - pix * oq) * 2;
        const unsigned oy = sn_div(pix, (unsigned)oW, rcp_oW), ox = pix - oy * (unsigned)oW;
        int2 k[5];   // this pair's constants, in flight during the products
        if (form >= 0)
#pragma unroll
            for (int r = 0; r < 5; ++r) k[r] = *(const int2*)(cst + r * opad + o);
        int acc[IPB][2];
#pragma unroll
        for (int i = 0; i < IPB; ++i) acc[i][0] = acc[i][1] = 0;
        if (valid) {
            const unsigned at = oy * step_y + ox * step_x, off = at & 3u;   // off: the copy in which this window is aligned (0 with one copy)
            sn_conv_item<IPB, UNSIGNED>(n, kH, step_ky, (int)split * opad, w0 + part * opad + o,
                                        acts + in_off + off * copy_stride + (at - off) + 4 * part, act_stride, (int)split, acc);
        }
        for (unsigned d = split >> 1; d; d >>= 1)
#pragma unroll
            for (int i = 0; i < IPB; ++i) {
                acc[i][0] += __shfl_xor_sync(0xffffffffu, acc[i][0], d);
                acc[i][1] += __shfl_xor_sync(0xffffffffu, acc[i][1], d);
            }
        if (!valid || part) continue;
        if (form < 0) {
#pragma unroll 1
            for (int i = 0; i < IPB; ++i) {
                acc[i][0] = sn_requant_exact(acc[i][0], (int)o, cell.q);
                if ((int)o + 1 < O) acc[i][1] = sn_requant_exact(acc[i][1], (int)o + 1, cell.q);
            }
        } else {
#pragma unroll
            for (int i = 0; i < IPB; ++i) {
                if (form == EF_FLOAT) {
                    acc[i][0] = rescale<true, EF_FLOAT>(acc[i][0], k[0].x, k[1].x, k[2].x, k[3].x, k[4].x);
                    acc[i][1] = rescale<true, EF_FLOAT>(acc[i][1], k[0].y, k[1].y, k[2].y, k[3].y, k[4].y);
                } else if (form == EF_WIDE) {
                    acc[i][0] = rescale<false, EF_WIDE>(acc[i][0], k[0].x, k[1].x, k[2].x, k[3].x, k[4].x);
                    acc[i][1] = rescale<false, EF_WIDE>(acc[i][1], k[0].y, k[1].y, k[2].y, k[3].y, k[4].y);
                } else {
                    acc[i][0] = rescale<true, 0>(acc[i][0], k[0].x, k[1].x, k[2].x, k[3].x, k[4].x);
                    acc[i][1] = rescale<true, 0>(acc[i][1], k[0].y, k[1].y, k[2].y, k[3].y, k[4].y);
                }
                acc[i][0] = min(max(acc[i][0], sat_lo), sat_hi);
                acc[i][1] = min(max(acc[i][1], sat_lo), sat_hi);
            }
        }
        const bool both = (int)o + 1 < O;
#pragma unroll
        for (int i = 0; i < IPB; ++i) {
            if (!last) {
                uint8_t* const at = acts + out_off + oy * out_row + ox * O + o + i * act_stride;
                sn_put(at, out_copies, out_copy_stride, acc[i][0]);
                if (both) sn_put(at + 1, out_copies, out_copy_stride, acc[i][1]);
            } else if (i < nimg) {
                const size_t at = (size_t)i * out_stride + pix * (size_t)O + o;
                out[0][at] = (uint8_t)acc[i][0];
                if (both) out[0][at + 1] = (uint8_t)acc[i][1];
                if (out[1]) {
                    out[1][at] = (uint8_t)acc[i][0];
                    if (both) out[1][at + 1] = (uint8_t)acc[i][1];
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
                sn_put(acts + c.out_off + oy * c.out_row + ox * c.O + o + i * act_stride, c.out_copies, c.out_copy_stride, v);
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
    __shared__ SmallCell cells[SMALL_NET_CELLS];
    uint8_t* const acts = smem + a.blob_bytes;
    // The cells' descriptions leave the parameter space before the wait: read there cell by cell, every first use was a constant-cache
    // miss and a cell of ten outputs took 2100 cycles.
    const unsigned* descr = (const unsigned*)a.cell;
    asm volatile("" : "+l"(descr));
    for (unsigned i = threadIdx.x; i < (unsigned)a.nb_cells * (unsigned)(sizeof(SmallCell) / 4); i += SN_THREADS) ((unsigned*)cells)[i] = descr[i];
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
            const unsigned per = (unsigned)a.in_bytes / 4u, n = per * (unsigned)nimg;
            for (unsigned i = threadIdx.x; i < n; i += SN_THREADS) {
                const unsigned k = IPB == 1 ? 0u : i / per, j = i - k * per;
                uint8_t* at = acts + a.in_place + k * a.act_stride + 4 * j;
                const unsigned w = __ldg((const unsigned*)src + i);
                *(unsigned*)at = w;
                if (a.in_copies > 1) {
                    const unsigned nxt = j + 1 < per ? __ldg((const unsigned*)src + i + 1) : 0u;
#pragma unroll
                    for (int q = 1; q < 4; ++q) *(unsigned*)(at + q * a.in_copy_stride) = __funnelshift_r(w, nxt, 8 * q);
                }
            }
        } else {
            const unsigned rb = (unsigned)a.in_row, n = (unsigned)a.in_bytes * (unsigned)nimg;
            for (unsigned i = threadIdx.x; i < n; i += SN_THREADS) {
                const unsigned k = i / (unsigned)a.in_bytes, j = i - k * (unsigned)a.in_bytes, r = j / rb;
                sn_put(acts + a.in_place + k * a.act_stride + r * a.in_pitch + (j - r * rb), a.in_copies, a.in_copy_stride, src[i]);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        uint8_t* const dst[2] = {out + (size_t)img * a.out_bytes, out2 ? out2 + (size_t)img * a.out_bytes : nullptr};
#pragma unroll 1
        for (int l = 0; l < a.nb_cells; ++l) {
            const SmallCell& c = cells[l];
            if (c.pool) sn_pool<IPB>(c, acts, a.act_stride, nimg, dst, (size_t)a.out_bytes);
            else if (c.in_unsigned) sn_conv<IPB, true>(c, smem, acts, a.act_stride, nimg, dst, (size_t)a.out_bytes);
            else sn_conv<IPB, false>(c, smem, acts, a.act_stride, nimg, dst, (size_t)a.out_bytes);
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
    int pitch = Wp * g.C;
    c.step_x = g.sX * g.C;
    // windows that start on any byte read from four copies of the input; their filter rows lie whole words apart in any case
    if (pitch % 4 != 0 && (g.oH > 1 || g.kH > 1)) pitch = (pitch + 3) & ~3;
    c.step_y = g.sY * pitch;
    c.step_ky = g.dY * pitch;
    const int copies = (c.step_x % 4 == 0 || g.oW == 1) ? 1 : 4;
    c.rcp_O = rcp32((unsigned)c.Opad / 2);
    c.rcp_oW = rcp32((unsigned)g.oW);
    while (c.log_split < 3 && ((long long)(c.Opad / 2) * g.oH * g.oW << (c.log_split + 1)) <= SN_THREADS && c.words % (2 << c.log_split) == 0) ++c.log_split;
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
    c.in_off = p->act_bytes + 4;               // the moved copies of the first bytes land in front
    c.in_off = (c.in_off + 3) & ~3;
    c.copy_stride = round16(Hp * pitch + 8);   // a run's last word may reach past its end
    small_net_link(p, c.in_off, copies, c.copy_stride, g.pT, g.pL, pitch, g.W * g.C, g.C, g.H, g.W, g.C);
    p->act_bytes = round16(c.in_off + copies * c.copy_stride);
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
    small_net_link(p, c.in_off, 1, 0, 0, 0, g.W * g.C, g.W * g.C, g.C, g.H, g.W, g.C);
    p->act_bytes += round16(g.H * g.W * g.C + 8);
    p->cells.push_back(c);
}

// Points the previous cell's output (or the network input) at the input area of the next cell
void small_net_link(SmallNetPlan* p, int in_off, int copies, int copy_stride, int pT, int pL, int pitch, int row_bytes, int pixel, int H, int W, int C)
{
    const int place = in_off + pT * pitch + pL * pixel;
    if (p->cells.empty()) {
        p->in_place = place;
        p->in_pitch = pitch;
        p->in_row = row_bytes;
        p->in_bytes = H * W * C;
        p->in_words = (pT == 0 && pL == 0 && pitch == row_bytes && p->in_bytes % 4 == 0) ? 1 : 0;
        p->in_copies = copies;
        p->in_copy_stride = copy_stride;
    } else {
        SmallCell& prev = p->cells.back();
        prev.out_off = place;
        // a fully-connected cell takes the map as one row: the rows then follow each other without padding
        prev.out_row = (H == 1 && W == 1) ? prev.oW * prev.O : pitch;
        prev.out_copies = copies;
        prev.out_copy_stride = copy_stride;
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
    a.in_copies = p.in_copies; a.in_copy_stride = p.in_copy_stride;
    a.in_bytes = p.in_bytes; a.in_place = p.in_place; a.in_pitch = p.in_pitch; a.in_row = p.in_row; a.in_words = p.in_words;
    a.out_bytes = p.out_bytes;
    static SmemLimitSet limits[2];
    // One image per CTA while that gives every image a CTA at once, four per pass beyond.  Up to one image per SM the CTA asks
    // for more than half of the shared memory: with room for two, the CTAs of a call pack onto the SMs that the call before
    // (64 images: 14.5 instead of 9.6 us) has left.
    size_t smem1 = p.blob.size() + p.act_bytes;
    const size_t smem4 = p.blob.size() + 4 * (size_t)p.act_bytes;
    const int per_sm1 = smem1 <= 110 * 1024 ? 2 : 1, per_sm4 = smem4 <= 110 * 1024 ? 2 : 1;
    if (batch <= num_sms * per_sm1 || p.group == 1) {
        const int grid = std::min(batch, num_sms * per_sm1);
        if (cudaError_t e = raise_smem_limit(small_net_kernel<1>, limits[0], SN_SMEM_MAX)) return e;
        if (batch <= num_sms) smem1 = std::max<size_t>(smem1, 120 * 1024);
        return launch_pdl(small_net_kernel<1>, grid, SN_THREADS, smem1, s, a, (const uint8_t*)in, batch, (uint8_t*)out, (uint8_t*)out2);
    }
    if (cudaError_t e = raise_smem_limit(small_net_kernel<4>, limits[1], SN_SMEM_MAX)) return e;
    const int grid = std::min((batch + 3) / 4, num_sms * per_sm4);
    return launch_pdl(small_net_kernel<4>, grid, SN_THREADS, smem4, s, a, (const uint8_t*)in, batch, (uint8_t*)out, (uint8_t*)out2);
}

}  // namespace n2d2b
