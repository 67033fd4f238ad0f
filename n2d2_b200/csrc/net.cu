// C ABI (include/n2d2b.h) and the static executor behind it: a quantized network is a list of cells
// in execution order, every tensor an NHWC buffer in HBM, every cell one kernel launch (a residual
// sum is folded into the producing convolution's epilogue when the graph allows it).
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "../../include/n2d2b.h"
#include "kernels.h"
#include "host_internal.h"
#include "tc_common.cuh"

using namespace n2d2b;

// ------------------------------------------------------------------------------------ errors
static thread_local char g_err[512] = "";

static int fail(int code, const char* fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

#define CUDA_TRY(expr)                                                                        \
    do {                                                                                      \
        cudaError_t e_ = (expr);                                                              \
        if (e_ != cudaSuccess)                                                                \
            return fail(N2D2B_ERR_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_), \
                        __FILE__, __LINE__);                                                  \
    } while (0)

// ------------------------------------------------------------------------------------ model
enum CellType { CELL_CONV, CELL_FC, CELL_POOL, CELL_SUM, CELL_SCALING };
enum Engine { ENG_TCGEN05, ENG_SIMT, ENG_DEPTHWISE, ENG_POOL, ENG_SUM, ENG_FUSED, ENG_STEM, ENG_PATCH, ENG_STEM_S2D, ENG_DWPW };

struct TensorRec {
    int C = 0, H = 0, W = 0;
    int dtype = DT_I8;
    int is_unsigned = 0;
    int producer = -1;
    int buffer = -1;      // index into Net::buffers, -1 for the network input
    bool readable = true;
    size_t elems() const { return (size_t)C * H * W; }
    size_t bytes_per_image() const { return elems() * (dtype == DT_I32 ? 4 : 1); }
};

struct QuantHost {
    int mode = SC_NONE, act = ACT_LINEAR, out_bits = 8, out_unsigned = 0, sat_thr = 0;
    int is_clipped = 0;
    int nb_channels = 0;
    std::vector<int32_t> bias, p0, p1, clip_thr, clip_val;
    std::vector<float> fscale, clip_f;
    bool has_bias = false;
    // device copy
    void* d_blob = nullptr;
    QuantDev dev{};
};

struct CellRec {
    CellType type;
    std::vector<int> inputs;
    int output = -1;
    n2d2b_conv_desc conv{};
    n2d2b_pool_desc pool{};
    ConvGeom geom{};
    PoolGeom pgeom{};
    QuantHost q;
    std::vector<int8_t> weights;  // host copy, OHWI int8 (int4 already widened)
    int wbits = 8;                // storage width the caller gave the weights in (8 or 4)
    int8_t* d_weights = nullptr;
    size_t d_weight_bytes = 0;    // bytes of weights this cell keeps in HBM
    Engine engine = ENG_SIMT;
    // fused residual sum
    int residual = -1;
    QuantHost q2;
    bool has_q2 = false;
    bool skipped = false;  // folded into another cell
    // 32-bit epilogue constants (tensor-core cells)
    FastQuant fast{};
    int* d_fast = nullptr;
    // a max pooling folded into the first-layer kernel (the cell's output then is the pooled tensor)
    bool pool_fused = false;
    PoolGeom fused_pool{};
    bool pool_first = false;  // by the kernel that pools the accumulators (stem_pool), else by the one that pools bytes
    StemPoolPlan stem_pool{};
    // first-layer tensor-core kernels
    StemPlan stem{};
    StemS2dPlan stem2{};
    void* d_pad4 = nullptr;   // input re-laid with 4 bytes per pixel and its zero padding written out
    // A cell whose output channels are not a multiple of 32 (a 1000-class classifier) cannot leave through the TMA
    // store of the 32-bit epilogue (rows of its output are not 16-byte multiples).  It runs with zero weight rows
    // appended up to pad_O channels into d_colpad ([pixels][pad_O]); a copy kernel then drops the padding.
    int pad_O = 0;
    void* d_colpad = nullptr;
    // stride-1 convolution from a shared-memory patch
    PatchPlan patch{};
    // a 1x1 cell that computes the depthwise cell in front of it too (its input then is that cell's input)
    int dw_cell = -1;
    DwPwPlan dwpw{};
    // packed 4-bit weights at large batches: widened to int8 by a small kernel into the network's scratch, then the int8
    // kernel of the layer (see plan_widened)
    enum { W8_NONE, W8_IGEMM, W8_PATCH } w8 = W8_NONE;
    IgemmPlan plan8{};
    PatchPlan patch8{};
    int w8_rows = 0, w8_ng_src = 0, w8_ng_dst = 0;
    size_t w8_offset = 0;         // in the network's scratch
    void* d_w8_out = nullptr;     // padded output matrix (see pad_O) of a widened cell
    // 3x3 depthwise cells on the tensor cores: weights as [kH][kW][C] for the calls that the dot-product kernel takes (see
    // dw3x3_faster), behind the block-diagonal ones in d_weights
    int8_t* d_dw3x3 = nullptr;
    // the two convolutions in front of a sum as one kernel (igemm_dual.cu): on the later one, which carries the sum, the index of the other and the
    // plan; on the other one the index of the later
    int dual_branch = -1, dual_sum = -1;
    bool dual_on = false, dual_always = false;   // always: in every call (packed weights: only where each call widens them)
    DualPlan dual{};
    PatchPlan dual_patch{};   // or by the patch kernel (proj_in set)
    // an expansion with its residual sum and the 1x1 cell behind it as one kernel (igemm_chain.cu): each other's index
    int chain_next = -1, chain_prev = -1;
    ChainPlan chain{};
    // tensor-core plan
    IgemmPlan plan{};
    bool probed = false;              // engine, plans and constants were found ahead of the buffers (probe_dense)
    const void* plan_input = nullptr;
    const void* plan_res = nullptr;   // a residual that is the network's input: the address the plan holds
    int plan_images = 0;              // images that the plan's maps over the network's input cover
};

struct n2d2b_net {
    int device = 0;
    int num_sms = 0;
    bool finalized = false;
    int max_batch = 0;
    unsigned flags = 0;
    std::vector<TensorRec> tensors;
    std::vector<CellRec> cells;
    std::vector<void*> buffers;
    std::vector<size_t> buffer_bytes;
    int* d_status = nullptr;
    void* d_w8 = nullptr;         // widened weights of the packed cells, of the call that is running
    long long w8_macs = 0;        // multiply-accumulates per image of the cells that have a widened form
    int call_batch = 0;           // images of the call that is running (its upload slices are smaller)
    bool call_widened = false;    // the call's weights are in d_w8
    int launches = 0;
    const void* last_input = nullptr;
    void* d_labels_scratch = nullptr;   // device labels / scores of the host-buffer top-N entry point
    size_t labels_scratch_bytes = 0;
    void* d_stage_in = nullptr;   // device staging of the host-buffer entry point
    void* d_stage_out = nullptr;
    // host-buffer entry point: the upload is cut into slices on its own stream so that the leading
    // cells (which need no tensor map and work slice by slice) run while later slices still arrive
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t slice_ready[8] = {nullptr};
    cudaEvent_t stage_free = nullptr;
    int head_cells = 0;
    int head_limit = 0;      // cells [0, head_limit) may run slice by slice: the buffer planner keeps their tensors apart
    int forced_slices = 0;   // n2d2b_net_set_slices: 0 = automatic
    // streaming host-buffer entry points (submit / wait): two staging sets, so that the upload of one batch runs
    // under the forward pass of the batch before it
    void* d_pipe_in[2] = {nullptr, nullptr};
    void* d_pipe_out[2] = {nullptr, nullptr};
    cudaEvent_t pipe_uploaded[2] = {nullptr, nullptr};
    cudaEvent_t pipe_computed[2] = {nullptr, nullptr};
    cudaEvent_t pipe_done[2] = {nullptr, nullptr};
    cudaStream_t download_stream = nullptr;
    bool pipe_busy[2] = {false, false};
    cudaStream_t pipe_stream[2] = {nullptr, nullptr};   // the stream each slot's work was queued on
    unsigned pipe_next = 0;
    // the whole network as one kernel (small chains of convolutions, poolings and fully-connected cells)
    SmallNetPlan small;
    void* d_small = nullptr;
};

static int validate_quant(const n2d2b_quant* qu, int channels, bool accumulators_have_bias, QuantHost& q,
                          const int32_t* bias)
{
    if (!qu) return fail(N2D2B_ERR_INVALID, "quant must not be NULL");
    const n2d2b_scaling& s = qu->scaling;
    q.mode = s.mode;
    q.act = qu->activation;
    q.out_bits = qu->out_bits;
    q.out_unsigned = qu->out_unsigned ? 1 : 0;
    q.sat_thr = qu->saturation_threshold;
    q.is_clipped = s.is_clipped ? 1 : 0;
    q.nb_channels = channels;
    if (q.mode < SC_NONE || q.mode > SC_DOUBLE_SHIFT) return fail(N2D2B_ERR_INVALID, "unknown scaling mode %d", q.mode);
    if (q.act < ACT_LINEAR || q.act > ACT_SATURATION) return fail(N2D2B_ERR_INVALID, "unknown activation %d", q.act);
    if (q.act == ACT_SATURATION && q.sat_thr < 0)
        return fail(N2D2B_ERR_INVALID, "saturation_threshold must not be negative (got %d)", q.sat_thr);
    if (q.mode != SC_NONE) {
        if (s.nb_channels != channels)
            return fail(N2D2B_ERR_INVALID, "scaling has %d channels, the cell has %d outputs", s.nb_channels, channels);
        // the integer modes throw on a non-quantized cell in the reference; a float-mode cell with
        // nbBits == 0 would produce fractional values, which this integer path cannot carry
        if (q.out_bits < 1 || q.out_bits > 8)
            return fail(N2D2B_ERR_INVALID, "out_bits must be in 1..8 (got %d)", q.out_bits);
    }
    q.p0.assign(channels, 0);
    q.p1.assign(channels, 0);
    q.fscale.assign(channels, 1.0f);
    q.clip_thr.assign(channels, 0);
    q.clip_val.assign(channels, 0);
    q.clip_f.assign(channels, 0.0f);
    switch (q.mode) {
    case SC_FLOAT_MULT:
        if (!s.fscale) return fail(N2D2B_ERR_INVALID, "FLOAT_MULT scaling needs fscale");
        for (int c = 0; c < channels; ++c) q.fscale[c] = s.fscale[c];
        break;
    case SC_FIXED_MULT16:
    case SC_FIXED_MULT32:
        if (!s.mult) return fail(N2D2B_ERR_INVALID, "FIXED_MULT scaling needs mult");
        for (int c = 0; c < channels; ++c) {
            const int f = s.frac_bits_per_channel ? s.frac_bits_per_channel[c] : s.frac_bits;
            if (f < 0 || f > 62) return fail(N2D2B_ERR_INVALID, "fractional bits %d out of range", f);
            q.p0[c] = s.mult[c];
            q.p1[c] = f;
        }
        break;
    case SC_SINGLE_SHIFT:
        if (!s.shift0) return fail(N2D2B_ERR_INVALID, "SINGLE_SHIFT scaling needs shift0");
        for (int c = 0; c < channels; ++c) {
            if (s.shift0[c] > 62) return fail(N2D2B_ERR_INVALID, "shift %d out of range", s.shift0[c]);
            q.p0[c] = s.shift0[c];
        }
        break;
    case SC_DOUBLE_SHIFT:
        if (!s.shift0 || !s.shift1) return fail(N2D2B_ERR_INVALID, "DOUBLE_SHIFT scaling needs shift0 and shift1");
        for (int c = 0; c < channels; ++c) {
            if (s.shift0[c] > 30 || s.shift1[c] > 62) return fail(N2D2B_ERR_INVALID, "shift pair out of range");
            q.p0[c] = s.shift0[c];
            q.p1[c] = s.shift1[c];
        }
        break;
    default:
        break;
    }
    // clipping only acts in the FLOAT and FIXED modes (CPU path of the reference)
    if (q.is_clipped && (q.mode == SC_FLOAT_MULT || q.mode == SC_FIXED_MULT16 || q.mode == SC_FIXED_MULT32)) {
        if (!s.clip) return fail(N2D2B_ERR_INVALID, "is_clipped needs clip values");
        for (int c = 0; c < channels; ++c) {
            const float cl = s.clip[c];
            if (!std::isfinite(cl)) return fail(N2D2B_ERR_INVALID, "clip[%d] is not finite", c);
            q.clip_f[c] = cl;
            q.clip_thr[c] = (int32_t)(cl > 0.0f ? std::floor(cl) : std::ceil(cl));
            q.clip_val[c] = (int32_t)std::round(cl);
        }
    } else {
        q.is_clipped = 0;
    }
    q.has_bias = accumulators_have_bias && bias != nullptr;
    q.bias.assign(channels, 0);
    if (q.has_bias)
        for (int c = 0; c < channels; ++c) q.bias[c] = bias[c];
    return 0;
}

static void quant_output_type(const QuantHost& q, int* dtype, int* is_unsigned)
{
    if (q.mode == SC_NONE) {
        *dtype = DT_I32;
        *is_unsigned = 0;
    } else {
        *dtype = DT_I8;
        *is_unsigned = q.out_unsigned;
    }
}

// The exact form's per-channel words [7][C]
static std::vector<int32_t> exact_words(const QuantHost& q)
{
    const int C = q.nb_channels;
    std::vector<int32_t> blob((size_t)C * 7);
    memcpy(&blob[0 * C], q.bias.data(), C * 4);
    memcpy(&blob[1 * C], q.p0.data(), C * 4);
    memcpy(&blob[2 * C], q.p1.data(), C * 4);
    memcpy(&blob[3 * C], q.fscale.data(), C * 4);
    memcpy(&blob[4 * C], q.clip_thr.data(), C * 4);
    memcpy(&blob[5 * C], q.clip_val.data(), C * 4);
    memcpy(&blob[6 * C], q.clip_f.data(), C * 4);
    return blob;
}

// The scalar fields of the device view
static void fill_quant_scalars(const QuantHost& q, QuantDev& v)
{
    v.mode = q.mode;
    v.act = q.act;
    v.saturate = (q.mode != SC_NONE) ? 1 : 0;
    if (q.out_unsigned) { v.out_lo = 0; v.out_hi = (1 << q.out_bits) - 1; }
    else { v.out_lo = -(1 << (q.out_bits - 1)); v.out_hi = (1 << (q.out_bits - 1)) - 1; }
    v.is_clipped = q.is_clipped;
    v.sat_thr = q.sat_thr;
}

static int upload_quant(QuantHost& q)
{
    const int C = q.nb_channels;
    const std::vector<int32_t> blob = exact_words(q);
    CUDA_TRY(cudaMalloc(&q.d_blob, blob.size() * 4 + 16));
    CUDA_TRY(cudaMemcpy(q.d_blob, blob.data(), blob.size() * 4, cudaMemcpyHostToDevice));
    int32_t* d = (int32_t*)q.d_blob;
    QuantDev& v = q.dev;
    fill_quant_scalars(q, v);
    v.bias = q.has_bias ? d + 0 * C : nullptr;
    v.p0 = d + 1 * C;
    v.p1 = d + 2 * C;
    v.fscale = (const float*)(d + 3 * C);
    v.clip_thr = d + 4 * C;
    v.clip_val = d + 5 * C;
    v.clip_f = (const float*)(d + 6 * C);
    return 0;
}

// ---- 32-bit epilogue constants ----------------------------------------------------------------
// For the shift and fixed-point modes the rescale of channel c is f(x) = (x * m + half) >> s with
// m >= 0, a non-decreasing function of x.  Saturating f(x) to [out_lo, out_hi] (and a ReLU) equals
// evaluating f on x clamped to [L, H], where H is the smallest x with f(x) >= out_hi and L the
// largest x with f(x) <= out_lo: the clamp bounds every product, so 32-bit arithmetic is exact.
// Clipping to [0, clip] before the rescale tightens the same clamp, and the bias is folded in:
//   y = (clamp(acc, L - b, H - b) * m + (b * m + half)) >> s.
// Returns false when some intermediate could leave 32 bits or the configuration is outside this
// form (float mode, negative multipliers, clip <= 0, out_bits != 8); the
// exact 64-bit epilogue is used then.
static long long ceil_div(long long a, long long b)  // b > 0
{
    return (a >= 0) ? (a + b - 1) / b : -((-a) / b);
}

// 64-bit form of the same rescale, for fixed-point scalings whose products leave 32 bits; the shifted result must fit 32 bits.  The final pack
// saturates.  A clipping to [0, clip] and the ReLU of a signed output become a clamp of the rescaled value to [0, row 1] (`need_clamp`; callers
// without one pass nullptr and are refused such cells): the rescale never decreases and gives 0 at 0.
static bool build_wide_quant(const QuantHost& q, int cpad, long long x_bound, std::vector<int32_t>& out, bool* need_clamp = nullptr)
{
    const bool floor0 = q.is_clipped || (q.act == ACT_RECTIFIER && !q.out_unsigned);
    if ((floor0 && !need_clamp) || q.act == ACT_SATURATION) return false;
    if (floor0) *need_clamp = true;
    const int C = q.nb_channels;
    out.assign((size_t)5 * cpad, 0);
    for (int c = 0; c < C; ++c) {
        long long m, s;
        if (q.mode == SC_SINGLE_SHIFT) { m = 1; s = q.p0[c]; }
        else if (q.mode == SC_DOUBLE_SHIFT) { m = 1 + (1ll << q.p0[c]); s = q.p1[c]; }
        else { m = q.p0[c]; s = q.p1[c]; }
        if (m < 0 || m > (1ll << 30) || s > 31) return false;
        const long long half = s > 0 ? (1ll << (s - 1)) : 0;
        const long long b = q.has_bias ? q.bias[c] : 0;
        if (std::llabs(b) > (1ll << 30)) return false;   // keeps every 64-bit intermediate below 2^61
        const long long add = b * m + half;                                   // < 2^62
        const long long worst = x_bound * m + std::llabs(add);               // < 2^62 for x_bound < 2^30
        if ((worst >> s) > (1ll << 31) - 2) return false;
        long long top = q.out_unsigned ? 255 : 127;
        if (q.is_clipped) {
            if (!(q.clip_f[c] > 0.0f)) return false;
            top = std::min(top, ((long long)q.clip_val[c] * m + half) >> s);
        }
        out[(size_t)1 * cpad + c] = (int32_t)top;
        out[(size_t)0 * cpad + c] = (int32_t)(add >> 32);
        out[(size_t)2 * cpad + c] = (int32_t)m;
        out[(size_t)3 * cpad + c] = (int32_t)(uint32_t)(add & 0xffffffffll);
        out[(size_t)4 * cpad + c] = (int32_t)s;
    }
    return true;
}

// Floating-point scaling: y = round(clamp(float(acc + bias), lo, hi) * factor), the final pack saturates.  Clipping to [0, clip]
// (to [clip, 0] for clip <= 0) before the rescale is the clamp: a sum inside the bound converts to a float that is not
// beyond it, one outside converts to the bound or further.  A ReLU in front of a signed output is the lower bound 0, which
// needs factors that are not negative; the sum has to stay inside 32 bits.  Rows: lo, hi, factor (floats), bias, unused.
static bool build_float_quant(const QuantHost& q, int cpad, long long x_bound, std::vector<int32_t>& out, bool* need_clamp)
{
    if (q.mode != SC_FLOAT_MULT || q.out_bits != 8 || q.act == ACT_SATURATION) return false;
    const bool relu_clamp = q.act == ACT_RECTIFIER && !q.out_unsigned;
    if (q.is_clipped || relu_clamp) *need_clamp = true;
    out.assign((size_t)5 * cpad, 0);
    for (int c = 0; c < q.nb_channels; ++c) {
        const float factor = q.fscale[c];
        if (!std::isfinite(factor) || !(factor >= 0.0f)) return false;
        const long long b = q.has_bias ? q.bias[c] : 0;
        if (std::llabs(b) + x_bound > (1ll << 31) - 1) return false;
        float lo = -INFINITY, hi = INFINITY;
        if (q.is_clipped) {
            lo = std::min(q.clip_f[c], 0.0f);
            hi = std::max(q.clip_f[c], 0.0f);
        }
        if (relu_clamp) {
            lo = std::max(lo, 0.0f);
            hi = std::max(hi, 0.0f);
        }
        memcpy(&out[(size_t)0 * cpad + c], &lo, 4);
        memcpy(&out[(size_t)1 * cpad + c], &hi, 4);
        memcpy(&out[(size_t)2 * cpad + c], &factor, 4);
        out[(size_t)3 * cpad + c] = (int32_t)b;
    }
    return true;
}

static bool build_fast_quant(const QuantHost& q, int cpad, long long x_bound, std::vector<int32_t>& out, int* eff_lo,
                             int* eff_hi, bool* need_clamp)
{
    if (q.mode != SC_SINGLE_SHIFT && q.mode != SC_DOUBLE_SHIFT && q.mode != SC_FIXED_MULT16 && q.mode != SC_FIXED_MULT32)
        return false;
    if (q.out_bits != 8) return false;
    const int C = q.nb_channels;
    long long out_hi = q.out_unsigned ? 255 : 127;
    long long out_lo = q.out_unsigned ? 0 : -128;
    if (q.act == ACT_RECTIFIER && out_lo < 0) out_lo = 0;
    if (q.act == ACT_SATURATION) {
        // saturate to the output range, then clamp to +-threshold: one clamp to the intersection
        out_hi = std::min(out_hi, (long long)q.sat_thr);
        out_lo = std::max(out_lo, -(long long)q.sat_thr);
        *need_clamp = true;
    }
    *eff_lo = (int)out_lo;
    *eff_hi = (int)out_hi;
    out.assign((size_t)5 * cpad, 0);
    const long long LIM = (1ll << 31) - 1;
    // without the clamps the final 8-bit pack does the saturation (and, for unsigned outputs, the ReLU)
    if (q.is_clipped || (q.act == ACT_RECTIFIER && !q.out_unsigned)) *need_clamp = true;
    for (int c = 0; c < C; ++c) {
        long long m, s;
        if (q.mode == SC_SINGLE_SHIFT) { m = 1; s = q.p0[c]; }
        else if (q.mode == SC_DOUBLE_SHIFT) { m = 1 + (1ll << q.p0[c]); s = q.p1[c]; }
        else { m = q.p0[c]; s = q.p1[c]; }
        if (m < 0 || s > 30) return false;
        const long long half = s > 0 ? (1ll << (s - 1)) : 0;
        long long L = 0, H = 0;
        if (m > 0) {
            H = ceil_div((out_hi << s) - half, m);
            L = ceil_div(((out_lo + 1) << s) - half, m) - 1;
        }
        // a threshold is met exactly only if the rescale of the bound gives it (a scale above 1 can step over it; the
        // native 8-bit bounds are the final pack's)
        if (q.act == ACT_SATURATION && m > 0 && (((H * m + half) >> s) > out_hi || ((L * m + half) >> s) < out_lo)) return false;
        if (q.is_clipped) {
            if (!(q.clip_f[c] > 0.0f)) return false;
            L = std::max(L, 0ll);
            H = std::min(H, (long long)q.clip_val[c]);
        }
        if (H < L) L = H;   // everything saturates to the same value
        const long long b = q.has_bias ? q.bias[c] : 0;
        long long lo = L - b, hi = H - b;
        const long long add = b * m + half;
        // |x| never exceeds x_bound, so clamp bounds beyond it are equivalent to it (min(max(x, lo), hi)
        // with lo > hi yields hi, which is then on the saturating side as well)
        lo = std::max(lo, -x_bound);
        hi = std::min(hi, x_bound);
        const long long p0 = lo * m + add, p1 = hi * m + add;
        if (std::llabs(add) > LIM || std::llabs(p0) > LIM || std::llabs(p1) > LIM) return false;
        if (x_bound * m + std::llabs(add) > LIM) *need_clamp = true;   // an unclamped product could overflow
        out[(size_t)0 * cpad + c] = (int32_t)lo;
        out[(size_t)1 * cpad + c] = (int32_t)hi;
        out[(size_t)2 * cpad + c] = (int32_t)m;
        out[(size_t)3 * cpad + c] = (int32_t)add;
        out[(size_t)4 * cpad + c] = (int32_t)s;
    }
    return true;
}

// The constants of a rescale without a residual, in the first form proved exact for |x| <= x_bound: 0 (32-bit, with valid
// clamps), EF_FLOAT, EF_WIDE; -1 when only the exact 64-bit evaluation is.
static int build_rescale(const QuantHost& q, int cpad, long long x_bound, std::vector<int32_t>& words)
{
    int lo = 0, hi = 0;
    bool need_clamp = false;
    if (build_fast_quant(q, cpad, x_bound, words, &lo, &hi, &need_clamp)) return 0;
    if (build_float_quant(q, cpad, x_bound, words, &need_clamp)) return EF_FLOAT;
    const bool integer = q.mode == SC_SINGLE_SHIFT || q.mode == SC_DOUBLE_SHIFT || q.mode == SC_FIXED_MULT16 || q.mode == SC_FIXED_MULT32;
    if (integer && q.out_bits == 8 && x_bound < (1ll << 30) && build_wide_quant(q, cpad, x_bound, words)) return EF_WIDE;
    return -1;
}

// w4: the cell's weights are 4-bit values (|w| <= 8), which tightens the accumulator bound
static int upload_fast(CellRec& c, const TensorRec& tout, bool residual_dtype_i8 = false, int residual_unsigned = 0,
                       bool w4 = false)
{
    c.fast = FastQuant{};
    if (tout.dtype != DT_I8) return 0;
    const int C = c.q.nb_channels;
    const int cpad = ((C + 255) / 256) * 256;
    std::vector<int32_t> f1, f2;
    int lo1, hi1, lo2 = 0, hi2 = 0;
    // |accumulator| <= K * 255 * 128 (4-bit weights: K * 255 * 8; they enter the tensor core times 16 and the
    // epilogue divides the sum by 16 again before anything else); the residual stage adds two 8-bit values
    const long long acc_bound = (long long)c.geom.kH * c.geom.kW * c.geom.Cg * 255ll * (w4 ? 8ll : 128ll);
    if (acc_bound * (w4 ? 16 : 1) > (1ll << 30)) return 0;
    bool need_clamp = false, wide = false, wide_clamps = false;
    const bool with_res = c.residual >= 0;
    const bool flt = c.q.mode == SC_FLOAT_MULT;
    if (flt) {
        // both stages of a residual cell share one form
        if (!build_float_quant(c.q, cpad, acc_bound, f1, &need_clamp)) return 0;
        if (with_res && !build_float_quant(c.q2, cpad, 512, f2, &need_clamp)) return 0;
        lo1 = c.q.out_unsigned ? 0 : (c.q.act == ACT_RECTIFIER ? 0 : -128);
        hi1 = c.q.out_unsigned ? 255 : 127;
    } else if (!build_fast_quant(c.q, cpad, acc_bound, f1, &lo1, &hi1, &need_clamp)) {
        // eff range etc. were set before the failing channel; retry in 64 bits
        need_clamp = false;
        if (c.q.out_bits != 8 || c.q.act == ACT_SATURATION
            || (c.q.mode != SC_SINGLE_SHIFT && c.q.mode != SC_DOUBLE_SHIFT && c.q.mode != SC_FIXED_MULT16
                && c.q.mode != SC_FIXED_MULT32)
            || !build_wide_quant(c.q, cpad, acc_bound, f1, &wide_clamps))
            return 0;
        wide = true;
        need_clamp = wide_clamps;
        lo1 = c.q.out_unsigned ? 0 : -128;
        hi1 = c.q.out_unsigned ? 255 : 127;
        if (c.q.act == ACT_RECTIFIER && lo1 < 0) lo1 = 0;
    }
    if (with_res && !flt && !build_fast_quant(c.q2, cpad, 512, f2, &lo2, &hi2, &need_clamp)) return 0;
    if (wide && need_clamp && !wide_clamps) return 0;   // the 64-bit form has the clamp at 0 or none
    // Dot-product form of the residual stage (see perm_block): every multiplier of the sum's scaling fits a byte,
    // both operands have a native 8-bit range and no clamp is needed.  The four bytes [t, t', r, r'] of a dot
    // product share one signedness: when the cell's own output is signed and the residual unsigned, the first
    // rescale produces t + 128 instead (its addend grows by 128 << shift, a multiple of 2^shift, so the shifted
    // value is exactly 128 larger and the unsigned saturating pack clamps at the same places) and the second
    // addend drops 128 * m2.
    bool dp4a = false, dp_t_unsigned = false;
    int dp_a_signed = 1;
    if (with_res && !need_clamp && !wide && !flt && residual_dtype_i8) {
        const bool t_uns = (lo1 == 0 && hi1 == 255), t_sig = (lo1 == -128 && hi1 == 127);
        const bool r_uns = residual_unsigned != 0;
        bool ok = t_uns || t_sig;
        for (int ch = 0; ch < C; ++ch) ok = ok && f2[(size_t)2 * cpad + ch] >= 0 && f2[(size_t)2 * cpad + ch] <= 255;
        if (ok && t_uns && !r_uns) ok = false;   // unsigned output with a signed residual: the exact two-step form
        const bool shift_t = ok && t_sig && r_uns;
        if (shift_t) {
            const long long LIM = (1ll << 31) - 1;
            for (int ch = 0; ch < C && ok; ++ch) {
                const long long m = f1[(size_t)2 * cpad + ch], add = f1[(size_t)3 * cpad + ch], sh = f1[(size_t)4 * cpad + ch];
                const long long nadd = add + (128ll << sh);
                if (acc_bound * m + std::llabs(nadd) > LIM) ok = false;
            }
        }
        if (ok) {
            dp4a = true;
            dp_t_unsigned = t_uns || shift_t;
            dp_a_signed = dp_t_unsigned ? 0 : 1;
            for (int ch = 0; ch < cpad; ++ch) {
                const long long m2 = f2[(size_t)2 * cpad + ch];
                // row 0 of the residual set: the multiplier in the byte lanes of this column (even column:
                // lanes 0 and 2 = t and r; odd column: lanes 1 and 3)
                f2[(size_t)0 * cpad + ch] = (int32_t)((ch & 1) ? (m2 << 8 | m2 << 24) : (m2 | m2 << 16));
                if (shift_t) {
                    f1[(size_t)3 * cpad + ch] += (int32_t)(128ll << f1[(size_t)4 * cpad + ch]);
                    f2[(size_t)3 * cpad + ch] -= (int32_t)(128 * m2);
                }
            }
        }
    }
    const size_t words = f1.size() + f2.size();
    CUDA_TRY(cudaMalloc((void**)&c.d_fast, words * 4 + 16));
    CUDA_TRY(cudaMemcpy(c.d_fast, f1.data(), f1.size() * 4, cudaMemcpyHostToDevice));
    if (with_res) CUDA_TRY(cudaMemcpy(c.d_fast + f1.size(), f2.data(), f2.size() * 4, cudaMemcpyHostToDevice));
    c.fast.fq = c.d_fast;
    c.fast.fq2 = with_res ? c.d_fast + f1.size() : nullptr;
    c.fast.cpad = cpad;
    c.fast.t_lo = lo1;
    c.fast.t_hi = hi1;
    c.fast.out_unsigned = with_res ? c.q2.out_unsigned : c.q.out_unsigned;
    c.fast.need_clamp = need_clamp;
    c.fast.form = wide ? EF_WIDE : (flt ? EF_FLOAT : 0);
    c.fast.dp4a = dp4a;
    c.fast.dp_t_unsigned = dp_t_unsigned;
    c.fast.dp_a_signed = dp_a_signed;
    c.fast.monotone = true;   // (row 2: a multiplier, or a factor as the bits of a float)
    for (int ch = 0; ch < C; ++ch) c.fast.monotone = c.fast.monotone && f1[(size_t)2 * cpad + ch] >= 0;
    c.fast.unit_multiplier = !wide && !flt;
    for (int ch = 0; ch < C; ++ch) c.fast.unit_multiplier = c.fast.unit_multiplier && f1[(size_t)2 * cpad + ch] == 1;
    c.fast.enabled = true;
    return 0;
}

static void unpack_weights(const void* src, int weight_bits, size_t rows, size_t row_elems, std::vector<int8_t>& dst)
{
    dst.resize(rows * row_elems);
    if (weight_bits == 8) {
        memcpy(dst.data(), src, rows * row_elems);
        return;
    }
    // Packed sub-byte weights as the reference's export stores them (data<N>, export/CPP_Quantization/include/
    // typedefs.hpp:359-517): 8 / N values per byte, the first one in the highest bits, every row starting on a byte;
    // two's complement in N bits, except N = 1 where the bit 0 stands for -1 and 1 for +1.
    const size_t per_byte = 8 / (size_t)weight_bits;
    const size_t row_bytes = (row_elems + per_byte - 1) / per_byte;
    const int mask = (1 << weight_bits) - 1, sign = 1 << (weight_bits - 1);
    const uint8_t* p = (const uint8_t*)src;
    for (size_t r = 0; r < rows; ++r)
        for (size_t i = 0; i < row_elems; ++i) {
            const uint8_t byte = p[r * row_bytes + i / per_byte];
            const int shift = 8 - weight_bits * (int)(i % per_byte + 1);
            int v = (byte >> shift) & mask;
            if (weight_bits == 1) v = v ? 1 : -1;
            else if (v & sign) v -= 1 << weight_bits;
            dst[r * row_elems + i] = (int8_t)v;
        }
}

// ---- helpers exported to the other translation units (host_internal.h) -------------------------
namespace n2d2b {
int set_error(int code, const char* fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

int prepare_fast_constants(const n2d2b_quant* quant, int channels, const int32_t* bias, long long acc_bound,
                           std::vector<int32_t>& consts, int* cpad, int* out_unsigned, bool* need_clamp)
{
    QuantHost q;
    if (int rc = validate_quant(quant, channels, true, q, bias)) return rc;
    *cpad = ((channels + 255) / 256) * 256;
    int lo = 0, hi = 0;
    *need_clamp = false;
    if (q.mode == SC_NONE || !build_fast_quant(q, *cpad, acc_bound, consts, &lo, &hi, need_clamp)) return 1;
    *out_unsigned = q.out_unsigned;
    return 0;
}
}  // namespace n2d2b

// One CTA waits, with the given limit, on a barrier that nobody ever arrives at: the bounded wait of the
// tensor-core kernels running out, on purpose and harmlessly (no fault, no trap; the kernel returns).
__global__ void wait_timeout_selftest_kernel(int* status, unsigned long long limit_ns)
{
    __shared__ unsigned long long bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) mbar_wait_for(smem_u32(&bar), 0, &abort_flag, status, 9, limit_ns);
    __syncthreads();
}

namespace n2d2b {
int wait_timeout_selftest(int* status, unsigned limit_us, cudaStream_t s)
{
    if (limit_us < 1 || limit_us > 100000) return fail(N2D2B_ERR_INVALID, "limit_us must be in 1..100000");
    wait_timeout_selftest_kernel<<<1, 32, 0, s>>>(status, (unsigned long long)limit_us * 1000ull);
    CUDA_TRY(cudaGetLastError());
    return 0;
}
}  // namespace n2d2b

// ------------------------------------------------------------------------------------ C ABI
extern "C" {

const char* n2d2b_last_error(void) { return g_err; }
int n2d2b_version(void) { return 100; }

int n2d2b_device_count(void)
{
    int n = 0;
    CUDA_TRY(cudaGetDeviceCount(&n));
    return n;
}

int n2d2b_net_create(int device, n2d2b_net** net)
{
    if (!net) return fail(N2D2B_ERR_INVALID, "net must not be NULL");
    *net = nullptr;
    int n = 0;
    CUDA_TRY(cudaGetDeviceCount(&n));
    if (device < 0 || device >= n) return fail(N2D2B_ERR_INVALID, "device %d out of range (%d devices)", device, n);
    CUDA_TRY(cudaSetDevice(device));
    cudaDeviceProp prop;
    CUDA_TRY(cudaGetDeviceProperties(&prop, device));
    if (prop.major != 10)
        return fail(N2D2B_ERR_INVALID, "device %d is sm_%d%d; this library is built for sm_100a only", device, prop.major,
                    prop.minor);
    n2d2b_net* p = new n2d2b_net();
    p->device = device;
    p->num_sms = prop.multiProcessorCount;
    *net = p;
    return 0;
}

void n2d2b_net_destroy(n2d2b_net* net)
{
    if (!net) return;
    cudaSetDevice(net->device);
    for (void* b : net->buffers) cudaFree(b);
    for (CellRec& c : net->cells) {
        cudaFree(c.d_weights);
        cudaFree(c.q.d_blob);
        cudaFree(c.q2.d_blob);
        cudaFree(c.d_fast);
        cudaFree(c.d_pad4);
        cudaFree(c.d_colpad);
        cudaFree(c.d_w8_out);
    }
    cudaFree(net->d_w8);
    cudaFree(net->d_status);
    cudaFree(net->d_small);
    cudaFree(net->d_labels_scratch);
    cudaFree(net->d_stage_in);
    cudaFree(net->d_stage_out);
    if (net->copy_stream) cudaStreamDestroy(net->copy_stream);
    for (cudaEvent_t e : net->slice_ready)
        if (e) cudaEventDestroy(e);
    if (net->stage_free) cudaEventDestroy(net->stage_free);
    for (int k = 0; k < 2; ++k) {
        cudaFree(net->d_pipe_in[k]);
        cudaFree(net->d_pipe_out[k]);
        if (net->pipe_uploaded[k]) cudaEventDestroy(net->pipe_uploaded[k]);
        if (net->pipe_computed[k]) cudaEventDestroy(net->pipe_computed[k]);
        if (net->pipe_done[k]) cudaEventDestroy(net->pipe_done[k]);
    }
    if (net->download_stream) cudaStreamDestroy(net->download_stream);
    delete net;
}

int n2d2b_net_set_input(n2d2b_net* net, int channels, int height, int width, int is_unsigned, int* tensor_id)
{
    if (!net) return fail(N2D2B_ERR_INVALID, "net must not be NULL");
    if (net->finalized || !net->tensors.empty()) return fail(N2D2B_ERR_STATE, "input already set");
    if (channels < 1 || height < 1 || width < 1) return fail(N2D2B_ERR_INVALID, "input dimensions must be positive");
    TensorRec t;
    t.C = channels; t.H = height; t.W = width; t.dtype = DT_I8; t.is_unsigned = is_unsigned ? 1 : 0;
    net->tensors.push_back(t);
    if (tensor_id) *tensor_id = 0;
    return 0;
}

static int check_tensor(const n2d2b_net* net, int id)
{
    if (!net) return fail(N2D2B_ERR_INVALID, "net must not be NULL");
    if (net->finalized) return fail(N2D2B_ERR_STATE, "the network is already finalized");
    if (id < 0 || id >= (int)net->tensors.size()) return fail(N2D2B_ERR_INVALID, "unknown tensor id %d", id);
    return 0;
}

static int conv_out(int in, int k, int stride, int pad0, int pad1, int dil)
{
    // ConvCell_Frame_Kernels.cpp:37-45
    return (int)((in + pad0 + pad1 - dil * (k - 1) - 1 + stride) / (double)stride);
}

int n2d2b_net_add_conv(n2d2b_net* net, const n2d2b_conv_desc* d, const void* weights, const int32_t* bias,
                       const n2d2b_quant* quant, int* tensor_id)
{
    if (!d || !weights) return fail(N2D2B_ERR_INVALID, "desc and weights must not be NULL");
    if (int rc = check_tensor(net, d->input)) return rc;
    const TensorRec in = net->tensors[d->input];
    if (in.dtype != DT_I8) return fail(N2D2B_ERR_INVALID, "a convolution needs an 8-bit input tensor");
    if (d->nb_outputs < 1 || d->kernel_h < 1 || d->kernel_w < 1 || d->stride_y < 1 || d->stride_x < 1
        || d->dilation_y < 1 || d->dilation_x < 1 || d->groups < 1 || d->pad_top < 0 || d->pad_left < 0
        || d->pad_bottom < 0 || d->pad_right < 0)
        return fail(N2D2B_ERR_INVALID, "invalid convolution geometry");
    if (in.C % d->groups || d->nb_outputs % d->groups)
        return fail(N2D2B_ERR_INVALID, "groups (%d) must divide channels (%d) and outputs (%d)", d->groups, in.C,
                    d->nb_outputs);
    if (d->weight_bits != 8 && d->weight_bits != 4 && d->weight_bits != 2 && d->weight_bits != 1)
        return fail(N2D2B_ERR_INVALID, "weight_bits must be 8, 4, 2 or 1");
    CellRec c;
    c.type = CELL_CONV;
    c.inputs = {d->input};
    c.conv = *d;
    ConvGeom& g = c.geom;
    g.H = in.H; g.W = in.W; g.C = in.C;
    g.O = d->nb_outputs;
    g.kH = d->kernel_h; g.kW = d->kernel_w; g.sY = d->stride_y; g.sX = d->stride_x;
    g.pT = d->pad_top; g.pL = d->pad_left; g.dY = d->dilation_y; g.dX = d->dilation_x;
    g.groups = d->groups; g.Cg = in.C / d->groups; g.Og = d->nb_outputs / d->groups;
    g.oH = conv_out(in.H, g.kH, g.sY, d->pad_top, d->pad_bottom, g.dY);
    g.oW = conv_out(in.W, g.kW, g.sX, d->pad_left, d->pad_right, g.dX);
    if (g.oH < 1 || g.oW < 1) return fail(N2D2B_ERR_INVALID, "convolution output would be empty");
    if (int rc = validate_quant(quant, g.O, true, c.q, bias)) return rc;
    unpack_weights(weights, d->weight_bits, (size_t)g.O, (size_t)g.kH * g.kW * g.Cg, c.weights);
    c.wbits = d->weight_bits;
    TensorRec t;
    t.C = g.O; t.H = g.oH; t.W = g.oW;
    quant_output_type(c.q, &t.dtype, &t.is_unsigned);
    t.producer = (int)net->cells.size();
    c.output = (int)net->tensors.size();
    net->tensors.push_back(t);
    net->cells.push_back(std::move(c));
    if (tensor_id) *tensor_id = net->cells.back().output;
    return 0;
}

int n2d2b_net_add_fc(n2d2b_net* net, int input, int nb_outputs, int weight_bits, const void* weights,
                     const int32_t* bias, const n2d2b_quant* quant, int* tensor_id)
{
    if (!weights) return fail(N2D2B_ERR_INVALID, "weights must not be NULL");
    if (int rc = check_tensor(net, input)) return rc;
    const TensorRec in = net->tensors[input];
    if (in.dtype != DT_I8) return fail(N2D2B_ERR_INVALID, "a fully-connected cell needs an 8-bit input tensor");
    if (nb_outputs < 1) return fail(N2D2B_ERR_INVALID, "nb_outputs must be positive");
    if (weight_bits != 8 && weight_bits != 4 && weight_bits != 2 && weight_bits != 1)
        return fail(N2D2B_ERR_INVALID, "weight_bits must be 8, 4, 2 or 1");
    CellRec c;
    c.type = CELL_FC;
    c.inputs = {input};
    // a fully-connected cell is a 1x1 convolution over the flattened input
    ConvGeom& g = c.geom;
    g.H = 1; g.W = 1; g.C = (int)in.elems();
    g.O = nb_outputs; g.kH = g.kW = 1; g.sY = g.sX = 1; g.pT = g.pL = 0; g.dY = g.dX = 1;
    g.groups = 1; g.Cg = g.C; g.Og = g.O; g.oH = g.oW = 1;
    if (int rc = validate_quant(quant, g.O, true, c.q, bias)) return rc;
    unpack_weights(weights, weight_bits, (size_t)g.O, (size_t)g.C, c.weights);
    c.wbits = weight_bits;
    TensorRec t;
    t.C = g.O; t.H = 1; t.W = 1;
    quant_output_type(c.q, &t.dtype, &t.is_unsigned);
    t.producer = (int)net->cells.size();
    c.output = (int)net->tensors.size();
    net->tensors.push_back(t);
    net->cells.push_back(std::move(c));
    if (tensor_id) *tensor_id = net->cells.back().output;
    return 0;
}

int n2d2b_net_add_pool(n2d2b_net* net, const n2d2b_pool_desc* d, int* tensor_id)
{
    if (!d) return fail(N2D2B_ERR_INVALID, "desc must not be NULL");
    if (int rc = check_tensor(net, d->input)) return rc;
    const TensorRec in = net->tensors[d->input];
    if (d->pool_h < 1 || d->pool_w < 1 || d->stride_y < 1 || d->stride_x < 1 || d->pad_y < 0 || d->pad_x < 0
        || (d->pooling != N2D2B_POOL_MAX && d->pooling != N2D2B_POOL_AVERAGE))
        return fail(N2D2B_ERR_INVALID, "invalid pooling geometry");
    CellRec c;
    c.type = CELL_POOL;
    c.inputs = {d->input};
    c.pool = *d;
    PoolGeom& g = c.pgeom;
    g.H = in.H; g.W = in.W; g.C = in.C;
    g.pH = d->pool_h; g.pW = d->pool_w; g.sY = d->stride_y; g.sX = d->stride_x; g.padY = d->pad_y; g.padX = d->pad_x;
    g.is_max = (d->pooling == N2D2B_POOL_MAX);
    // PoolCell.cpp:233-239
    g.oH = (int)((in.H + 2 * d->pad_y - d->pool_h + d->stride_y) / (double)d->stride_y);
    g.oW = (int)((in.W + 2 * d->pad_x - d->pool_w + d->stride_x) / (double)d->stride_x);
    if (g.oH < 1 || g.oW < 1) return fail(N2D2B_ERR_INVALID, "pooling output would be empty");
    TensorRec t;
    t.C = in.C; t.H = g.oH; t.W = g.oW; t.dtype = in.dtype; t.is_unsigned = in.is_unsigned;
    t.producer = (int)net->cells.size();
    c.output = (int)net->tensors.size();
    net->tensors.push_back(t);
    net->cells.push_back(std::move(c));
    if (tensor_id) *tensor_id = net->cells.back().output;
    return 0;
}

int n2d2b_net_add_elemwise_sum(n2d2b_net* net, const int* inputs, int nb_inputs, const n2d2b_quant* quant,
                               int* tensor_id)
{
    if (!inputs || nb_inputs < 1 || nb_inputs > 4)
        return fail(N2D2B_ERR_INVALID, "an element-wise sum takes 1 to 4 inputs");
    for (int k = 0; k < nb_inputs; ++k)
        if (int rc = check_tensor(net, inputs[k])) return rc;
    const TensorRec a = net->tensors[inputs[0]];
    for (int k = 1; k < nb_inputs; ++k) {
        const TensorRec& b = net->tensors[inputs[k]];
        if (b.C != a.C || b.H != a.H || b.W != a.W)
            return fail(N2D2B_ERR_INVALID, "element-wise inputs differ in shape");
    }
    CellRec c;
    c.type = CELL_SUM;
    c.inputs.assign(inputs, inputs + nb_inputs);
    if (int rc = validate_quant(quant, a.C, false, c.q, nullptr)) return rc;
    TensorRec t;
    t.C = a.C; t.H = a.H; t.W = a.W;
    quant_output_type(c.q, &t.dtype, &t.is_unsigned);
    t.producer = (int)net->cells.size();
    c.output = (int)net->tensors.size();
    net->tensors.push_back(t);
    net->cells.push_back(std::move(c));
    if (tensor_id) *tensor_id = net->cells.back().output;
    return 0;
}

int n2d2b_net_add_scaling(n2d2b_net* net, int input, const n2d2b_quant* quant, int* tensor_id)
{
    const int ids[1] = {input};
    int rc = n2d2b_net_add_elemwise_sum(net, ids, 1, quant, tensor_id);
    if (rc == 0) net->cells.back().type = CELL_SCALING;
    return rc;
}

// ---- finalize -------------------------------------------------------------------------------
static void fuse_residuals(n2d2b_net* net)
{
    const int nc = (int)net->cells.size();
    std::vector<int> consumers(net->tensors.size(), 0);
    for (const CellRec& c : net->cells)
        for (int i : c.inputs) consumers[i]++;
    for (int si = 0; si < nc; ++si) {
        CellRec& s = net->cells[si];
        if (s.type != CELL_SUM || s.inputs.size() != 2) continue;
        if (s.q.mode == SC_NONE) continue;
        int best = -1;
        for (int k = 0; k < 2; ++k) {
            const int t = s.inputs[k], other = s.inputs[1 - k];
            const TensorRec& tt = net->tensors[t];
            const TensorRec& ot = net->tensors[other];
            if (tt.producer < 0 || consumers[t] != 1) continue;
            CellRec& p = net->cells[tt.producer];
            if (p.type != CELL_CONV || p.geom.groups != 1 || p.residual >= 0 || p.skipped) continue;
            if (tt.dtype != DT_I8 || ot.dtype != DT_I8) continue;
            if (ot.producer >= tt.producer) continue;  // the other operand must exist when p runs
            if (best < 0 || tt.producer > net->tensors[s.inputs[best]].producer) best = k;
        }
        if (best < 0) continue;
        const int t = s.inputs[best], other = s.inputs[1 - best];
        CellRec& p = net->cells[net->tensors[t].producer];
        p.residual = other;
        p.q2 = s.q;
        p.has_q2 = true;
        p.inputs.push_back(other);  // keeps the operand alive for the buffer planner
        net->tensors[t].readable = false;
        net->tensors[t].buffer = -2;  // never materialised
        p.output = s.output;
        net->tensors[s.output].producer = net->tensors[t].producer;
        s.skipped = true;
        s.engine = ENG_FUSED;
    }
}

// Which cells share a kernel is settled before the buffers are planned, because it decides which tensors are stored and how long others live; the same
// functions then make the plans over the real addresses (plan_duals, plan_chains).
static int settle_duals(n2d2b_net* net);
static int settle_chains(n2d2b_net* net);

// Cells [0, n) that the host-buffer entry point may run slice by slice (a structural rule, applied before the
// kernels are chosen; the engine-based rule in finalize can only shorten it): image-wise cells with large
// per-image tensors, up to the first fully-connected cell or stand-alone sum.
static int head_candidate_prefix(const n2d2b_net* net)
{
    int n = 0;
    for (size_t ci = 0; ci < net->cells.size(); ++ci) {
        const CellRec& c = net->cells[ci];
        if (!c.skipped) {
            if (c.type == CELL_FC || c.type == CELL_SUM || c.type == CELL_SCALING) break;
            const TensorRec& t = net->tensors[c.output];
            if ((long long)t.H * t.W < 2048) break;
        }
        n = (int)ci + 1;
    }
    return n;
}

// A stride-2 first layer whose only reader is a max pooling writes the pooled tensor directly (stem_pool_tcgen05.cu, or on request
// the POOL variant of the space-to-depth kernel): the convolution's output, the largest tensor of such a network, is never stored.
static int fuse_stem_pool(n2d2b_net* net);

// A 3x3 depthwise cell whose only reader is a 1x1 cell becomes part of it (dwpw_tcgen05.cu): its output is never stored.
static int fuse_depthwise(n2d2b_net* net);

// Buffers are shared by lifetime.  Cells of the head run once per batch slice at an image offset, so slice k of
// a head tensor may be written while slices < k of every other head tensor are complete and still needed: two
// head tensors share a buffer only when they have the same bytes per image (slice k of one then lies exactly
// over slice k of the other, which the per-slice order of the cells has already retired).
static int plan_buffers(n2d2b_net* net)
{
    const bool keep_all = (net->flags & N2D2B_KEEP_ALL_OUTPUTS) != 0;
    std::vector<size_t> head_bpi;   // per buffer: bytes per image of the head tensors it has held (0 = none)
    const int nt = (int)net->tensors.size();
    std::vector<int> last_use(nt, -1);
    for (int ci = 0; ci < (int)net->cells.size(); ++ci) {
        const CellRec& c = net->cells[ci];
        if (c.skipped) continue;
        for (int i : c.inputs) last_use[i] = std::max(last_use[i], ci);
    }
    int final_tensor = -1;
    for (int ci = (int)net->cells.size() - 1; ci >= 0; --ci)
        if (!net->cells[ci].skipped) { final_tensor = net->cells[ci].output; break; }
    std::vector<size_t> sizes;
    std::vector<int> free_list;
    for (int ci = 0; ci < (int)net->cells.size(); ++ci) {
        CellRec& c = net->cells[ci];
        if (c.skipped) continue;
        auto take = [&](TensorRec& t, bool in_head) {
            const size_t need = ((t.bytes_per_image() * (size_t)net->max_batch + 255) / 256) * 256 + 256;
            int pick = -1;
            if (!keep_all) {
                for (size_t f = 0; f < free_list.size(); ++f) {
                    const int b = free_list[f];
                    if (in_head && head_bpi[b] != t.bytes_per_image()) continue;
                    if (sizes[b] >= need && (pick < 0 || sizes[b] < sizes[free_list[pick]])) pick = (int)f;
                }
            }
            if (pick >= 0) {
                t.buffer = free_list[pick];
                free_list.erase(free_list.begin() + pick);
            } else {
                t.buffer = (int)sizes.size();
                sizes.push_back(need);
                head_bpi.push_back(in_head ? t.bytes_per_image() : 0);
            }
        };
        TensorRec& t = net->tensors[c.output];
        if (c.dual_sum >= 0 && net->cells[c.dual_sum].dual_always) {   // its output stays on chip, its input lives until the sum
            t.readable = false;
            t.buffer = -2;
            continue;
        }
        if (c.chain_prev < 0) take(t, ci < net->head_limit);   // (else it was taken with the cell in front)
        if (c.chain_next >= 0) take(net->tensors[net->cells[c.chain_next].output], c.chain_next < net->head_limit);
        if (!keep_all) {
            // release the inputs that die with this cell (never the network input or the final output)
            for (int i : c.inputs) {
                if (i == 0 || i == final_tensor) continue;
                if (last_use[i] == ci && net->tensors[i].buffer >= 0) {
                    if (std::find(free_list.begin(), free_list.end(), net->tensors[i].buffer) == free_list.end())
                        free_list.push_back(net->tensors[i].buffer);
                }
            }
            // a tensor nobody reads (other than the final one) can be reused at once
            if (last_use[c.output] < 0 && c.output != final_tensor) free_list.push_back(t.buffer);
        }
    }
    if (!keep_all)
        for (int i = 1; i < nt; ++i)
            if (net->tensors[i].buffer >= 0 && i != final_tensor) net->tensors[i].readable = false;
    net->buffers.assign(sizes.size(), nullptr);
    net->buffer_bytes = sizes;
    for (size_t b = 0; b < sizes.size(); ++b) {
        CUDA_TRY(cudaMalloc(&net->buffers[b], sizes[b]));
        CUDA_TRY(cudaMemset(net->buffers[b], 0, sizes[b]));
    }
    return 0;
}

static void* tensor_ptr(const n2d2b_net* net, int id, const void* d_input)
{
    if (id == 0) return (void*)d_input;
    const TensorRec& t = net->tensors[id];
    return t.buffer >= 0 ? net->buffers[t.buffer] : nullptr;
}

// What a plan is made over where a tensor has no address: the network's input before a forward pass (encoded anew then), an output that is never
// stored, and every tensor while cells that share a kernel are settled
static void* placeholder()
{
    static char bytes[16] __attribute__((aligned(16)));
    return bytes;
}

static void* tensor_or_placeholder(const n2d2b_net* net, int id)
{
    void* p = tensor_ptr(net, id, nullptr);
    return p ? p : placeholder();
}

static int final_tensor_of(const n2d2b_net* net)
{
    for (int ci = (int)net->cells.size() - 1; ci >= 0; --ci)
        if (!net->cells[ci].skipped) return net->cells[ci].output;
    return -1;
}

// Whether a cell whose columns are padded stores the wanted ones from the registers: classifiers (one pixel per image) of launches that store that way
static bool stores_rows(const CellRec& c, const IgemmPlan& p) { return c.geom.oH * c.geom.oW == 1 && igemm_writes_rows(p, c.geom.O); }

// Whether a patch cell whose weights stream (128 channels) runs as an implicit GEMM in a call of `batch` images: up to one tile per SM.  A band then has few
// tiles to share the stream of all its weights, which the implicit GEMM loads ahead, tile by tile (3x3, 128 channels of 28 x 28 in ResNet-50, the
// whole network: one image 240 us -> 233, 8 images 301 / 298, 16 images 344 / 340; 32 images, two tiles per SM, 424 / 427).
static bool patch_as_gemm(const n2d2b_net* net, const CellRec& c, int batch)
{
    if (c.engine != ENG_PATCH || c.inputs[0] == 0 || c.residual >= 0 || c.geom.groups != 1 || !c.patch.b_stream || c.plan.perm != 32) return false;
    const long long m_tiles = ((long long)batch * c.geom.oH * c.geom.oW + 127) / 128;
    return m_tiles * ((c.geom.O + c.plan.BN - 1) / c.plan.BN) <= net->num_sms;
}

// Whether a call of `call` images widens packed weights at its start, in one launch of 3 to 4 us.  The line is drawn where a call is large enough to pay
// for it (ResNet-18 at 224 x 224, 1.7 G multiply-accumulates an image: four images 217 us with the expansion in the kernels, 182 widened cell by cell, 162 in
// one launch; 128 images 656 / 460 / 421: the expansion warps' shared-memory stores bound every layer of long K, and the classifier, which has no
// 32-bit epilogue in that form, took 38 to 110 us).
static bool widens_all(long long macs, int call) { return macs * call >= (1ll << 29); }
static bool widen_all(const n2d2b_net* net, int call) { return widens_all(net->w8_macs, call); }

static long long packed_tiles(const CellRec& c, int batch)
{
    return ((long long)batch * c.geom.oH * c.geom.oW + 127) / 128 * ((c.geom.O + c.plan.BN - 1) / c.plan.BN);
}

// In a smaller call a cell is widened by itself where a CTA has more than two tiles, whose in-kernel expansions would repeat
static bool widens_alone(const n2d2b_net* net, const CellRec& c, int batch) { return packed_tiles(c, batch) > 2ll * net->num_sms; }

// Which cells a large call widens.  The expansion costs a CTA about 0.14 us per K block and tile; widening moves 2.5 bytes a weight, 0.05 us per K block
// and 1024 outputs.  So wide layers of a tile per CTA keep their packed weights, unless their epilogue is not the 32-bit one in that form.
static bool worth_widening(const n2d2b_net* net, const CellRec& c, int call)
{
    const long long per_cta = (packed_tiles(c, call) + net->num_sms - 1) / net->num_sms;
    return c.geom.O < 1024 * per_cta || widens_alone(net, c, call) || !igemm_uses_fast_epilogue(c.plan, c.fast, c.residual >= 0, DT_I8);
}

// Whether a packed cell takes the widened form in a call of `call` images, `batch` of them at once; macs: of the network's packed cells, per image
static bool widens_in(const n2d2b_net* net, const CellRec& c, long long macs, int batch, int call)
{
    return (widens_all(macs, call) && worth_widening(net, c, call)) || widens_alone(net, c, batch);
}

static bool use_widened(const n2d2b_net* net, const CellRec& c, int batch, int call)
{
    return c.w8 != CellRec::W8_NONE && widens_in(net, c, net->w8_macs, batch, call);
}

// The implicit-GEMM plan of a dense cell
static int plan_dense(n2d2b_net* net, CellRec& c, const ConvGeom& g, bool w4, const void* in, const int8_t* w, const void* out, const void* res, const char** why)
{
    ConvGeom gb = g;
    gb.B = net->max_batch;
    return igemm_make_plan(&c.plan, in, w, out, res, gb, net->tensors[c.inputs[0]].is_unsigned, (net->flags & N2D2B_FORCE_IM2COL) ? 1 : 0, 0, net->num_sms, why,
                           (net->flags & N2D2B_FORCE_PAIR) ? 1 : 0, w4 ? 1 : 0);
}

// The kernel of a dense cell whose implicit-GEMM plan is made: its 32-bit constants, the patch kernel where that is the faster one, and the order of its
// weight rows (plan.perm)
static int choose_dense(n2d2b_net* net, CellRec& c, bool w4, const void* in, const int8_t* w)
{
    ConvGeom g = c.geom;
    g.B = net->max_batch;
    const TensorRec& tout = net->tensors[c.output];
    const bool exact = (net->flags & N2D2B_EXACT64_EPILOGUE) != 0, with_res = c.residual >= 0;
    const char* why = "";
    c.engine = ENG_TCGEN05;
    if (!exact && !c.pad_O && !c.d_fast) {
        // (the patch kernel's residual stage is not the dot-product form, nor is its sum with a projection)
        const bool res_i8 = with_res && net->tensors[c.residual].dtype == DT_I8 && (w4 || !patch_takes_residual(g))
                            && !(c.dual_branch >= 0 && patch_takes_projection(net->cells[c.dual_branch].geom, g));
        if (int rc = upload_fast(c, tout, res_i8, with_res ? net->tensors[c.residual].is_unsigned : 0, w4)) return rc;
    }
    // small-channel stride-1 layers read their input once, from a shared-memory patch
    if (!w4 && !c.pad_O && c.fast.enabled && (!with_res || (patch_takes_residual(g) && net->tensors[c.residual].dtype == DT_I8)) && tout.dtype == DT_I8
        && !exact && !(net->flags & N2D2B_FORCE_IM2COL) && patch_eligible(g)
        && patch_make_plan(&c.patch, in, w, g, net->tensors[c.inputs[0]].is_unsigned, net->num_sms, &why) == 0)
        c.engine = ENG_PATCH;
    // (a patch cell's rows are in the order of the implicit GEMM, which small calls may take: patch_as_gemm)
    if (igemm_uses_fast_epilogue(c.plan, c.fast, with_res, tout.dtype) && (c.engine == ENG_TCGEN05 || igemm_perm_block(c.plan) == 32))
        c.plan.perm = igemm_perm_block(c.plan);
    return 0;
}

// Bytes of widened weights of a packed cell, rounded so that another one's may follow
static size_t widened_bytes(const CellRec& c)
{
    const size_t n = (size_t)((c.geom.O + 31) & ~31) * c.geom.kH * c.geom.kW * c.geom.C;
    return (n + 255) & ~(size_t)255;
}

// Whether a packed cell has a widened form, whose plans are made over the given addresses (out: a matrix of padded rows where the outputs are no whole
// blocks of 32 columns)
static int plan_widened_cell(n2d2b_net* net, CellRec& c, const void* in, const int8_t* w, void* out, const void* res)
{
    ConvGeom g = c.geom;
    g.B = net->max_batch;
    const int in_u = net->tensors[c.inputs[0]].is_unsigned;
    const char* why = "";
    c.w8_ng_src = c.plan.perm / 8;
    c.w8_rows = g.O;
    if ((!res || (patch_takes_residual(g) && !c.fast.dp4a)) && patch_eligible(g) && patch_make_plan(&c.patch8, in, w, g, in_u, net->num_sms, &why) == 0) {
        c.patch8.late_weights = 1;
        c.w8_ng_dst = 4;
        c.w8 = CellRec::W8_PATCH;
        return 0;
    }
    g.O = c.w8_rows = (g.O + 31) & ~31;
    if (igemm_make_plan(&c.plan8, in, w, out, res, g, in_u, 0, 0, net->num_sms, &why) || !igemm_uses_fast_epilogue(c.plan8, c.fast, res != nullptr, DT_I8)) return 0;
    c.plan8.late_weights = 1;
    c.plan8.perm = igemm_perm_block(c.plan8);
    c.w8_ng_dst = c.plan8.perm / 8;
    c.w8 = CellRec::W8_IGEMM;
    return 0;
}

static long long cell_macs(const CellRec& c) { return (long long)c.geom.oH * c.geom.oW * c.geom.O * c.geom.kH * c.geom.kW * c.geom.C; }

// Plans the widened form of the packed cells that some call widens.  The weights stay packed in HBM; a scratch block of twice their size holds the int8
// weights of the call that is running.
static int plan_widened(n2d2b_net* net)
{
    auto plan = [&](CellRec& c, const int8_t* w, void* out) {
        const void* res = c.residual >= 0 ? tensor_or_placeholder(net, c.residual) : nullptr;
        return plan_widened_cell(net, c, c.plan_input, w, out, res);
    };
    for (CellRec& c : net->cells) {
        c.w8 = CellRec::W8_NONE;
        // (not where the input or the residual is the caller's buffer, whose address only the forward pass knows)
        if (c.skipped || c.engine != ENG_TCGEN05 || !c.plan.w4 || !c.fast.enabled || c.inputs[0] == 0 || c.residual == 0) continue;
        if (net->tensors[c.output].dtype != DT_I8 || (c.geom.O % 32 != 0 && c.residual >= 0)) continue;
        if (int rc = plan(c, (const int8_t*)placeholder(), placeholder())) return rc;
        if (c.w8 != CellRec::W8_NONE) net->w8_macs += cell_macs(c);
    }
    size_t total = 0;
    for (CellRec& c : net->cells) {
        if (!use_widened(net, c, net->max_batch, net->max_batch)) c.w8 = CellRec::W8_NONE;   // nor in a smaller call
        if (c.w8 == CellRec::W8_NONE) continue;
        c.w8_offset = total;
        total += widened_bytes(c);
    }
    if (!total) return 0;
    CUDA_TRY(cudaMalloc(&net->d_w8, total + 256));
    const bool all = widen_all(net, net->max_batch);
    if (all) net->launches++;
    for (CellRec& c : net->cells) {
        if (c.w8 == CellRec::W8_NONE) continue;
        void* out = tensor_or_placeholder(net, c.output);
        if (c.geom.O % 32 != 0) {
            CUDA_TRY(cudaMalloc(&c.d_w8_out, (size_t)net->max_batch * c.geom.oH * c.geom.oW * ((c.geom.O + 31) & ~31) + 256));
            out = c.d_w8_out;
        }
        if (int rc = plan(c, (const int8_t*)net->d_w8 + c.w8_offset, out)) return rc;
        if (c.w8 == CellRec::W8_NONE) return fail(N2D2B_ERR_STATE, "internal: a packed cell lost its widened form");
        net->launches += (all ? 0 : 1) + (c.d_w8_out && !stores_rows(c, c.plan8) ? 1 : 0);
    }
    return 0;
}

// Whether the pair of convolutions that ends in cell `b` runs as one kernel in a call of `batch` images: packed weights only where both are widened
static bool use_dual(const n2d2b_net* net, const CellRec& b, int batch, int call)
{
    if (!b.dual_on) return false;
    const CellRec& a = net->cells[b.dual_branch];
    return !a.plan.w4 || (use_widened(net, a, batch, call) && use_widened(net, b, batch, call));
}

// The pair of cell `b`, which carries the sum, and its branch as one kernel, planned over the given addresses; false where they stay two
static bool make_dual(n2d2b_net* net, CellRec& b, const void* in_a, const int8_t* w_a, const void* in_b, const int8_t* w_b, const void* out)
{
    CellRec& a = net->cells[b.dual_branch];
    const bool packed = a.plan.w4 && b.plan.w4;
    if (b.engine != ENG_TCGEN05 || (a.engine != ENG_TCGEN05 && a.engine != ENG_PATCH) || a.plan.w4 != b.plan.w4) return false;
    if (!a.fast.enabled || !b.fast.enabled || !b.fast.fq2 || net->tensors[b.output].dtype != DT_I8 || net->tensors[a.output].dtype != DT_I8) return false;
    // one order of weight rows for both: blocks of 32 channels
    if (packed ? (a.w8 == CellRec::W8_NONE || b.w8 == CellRec::W8_NONE || a.w8_ng_dst != 4 || b.w8_ng_dst != 4)
               : (b.plan.perm != 32 || (a.engine == ENG_TCGEN05 && a.plan.perm != 32)))
        return false;
    // A branch of few tiles and long K runs on clusters that share a tile when it is a kernel of its own: 3x3, 512 channels of 7 x 7 beside a projection of 256, one
    // and two images 16.6 us as two kernels, 17.9 and 18.5 as one; three images, no clusters, 20.0 / 18.7
    if (packed ? a.w8 == CellRec::W8_IGEMM && igemm_takes_clusters(a.plan8) : a.engine == ENG_TCGEN05 && igemm_takes_clusters(a.plan)) return false;
    ConvGeom ga = a.geom, gb = b.geom;
    ga.B = gb.B = net->max_batch;
    const char* why = "";
    // The patch kernel reads a 64-channel branch's input once, an im2col map nine times: 64 -> 64 channels of 55 x 55 with its projection at 2048 images
    // 596 us as two kernels, 718 as one of im2col loads; 128 channels of 28 x 28 400 / 290
    if ((a.engine == ENG_PATCH || a.w8 == CellRec::W8_PATCH) && ga.C <= 64) {
        // (a wide form's clamp is one at 0: both rescales have it or neither)
        if (!patch_takes_projection(ga, gb) || b.fast.dp4a || a.fast.form != b.fast.form || (a.fast.form == EF_WIDE && a.fast.need_clamp != b.fast.need_clamp)) return false;
        if (patch_make_plan(&b.dual_patch, in_a, w_a, ga, net->tensors[a.inputs[0]].is_unsigned, net->num_sms, &why)
            || patch_add_projection(&b.dual_patch, in_b, w_b, ga, net->tensors[b.inputs[0]].is_unsigned, &why)) {
            b.dual_patch.proj_in = nullptr;
            return false;
        }
        b.dual_patch.late_weights = packed ? 1 : 0;
        return true;
    }
    return dual_make_plan(&b.dual, in_a, w_a, ga, net->tensors[a.inputs[0]].is_unsigned, in_b, w_b, gb, net->tensors[b.inputs[0]].is_unsigned, out, net->num_sms, &why) == 0;
}

// The same for cell `c`, an expansion with its residual sum, and the 1x1 cell behind it
static bool make_chain(n2d2b_net* net, CellRec& c, const void* in, const int8_t* w, const void* out, const void* res, const int8_t* w_next)
{
    const CellRec& p = net->cells[c.chain_next];
    if (c.engine != ENG_TCGEN05 || p.engine != ENG_TCGEN05 || !c.fast.enabled || !c.fast.fq2 || !p.fast.enabled || c.plan.perm != 32 || p.plan.perm != 32
        || net->tensors[c.output].dtype != DT_I8)
        return false;
    ConvGeom g = c.geom;
    g.B = net->max_batch;
    const char* why = "";
    return chain_make_plan(&c.chain, in, w, out, res, g, net->tensors[c.inputs[0]].is_unsigned, w_next, p.geom, net->tensors[c.output].is_unsigned, net->num_sms, &why) == 0;
}

// Kernel and constants of a cell that may share a kernel with another one, ahead of its buffers; false where it is not a dense cell of whole blocks of columns.
// (The constants are kept, the plans are made again over the real addresses.)
static int probe_dense(n2d2b_net* net, CellRec& c, bool* dense)
{
    *dense = c.probed;
    if (c.probed) return 0;
    const ConvGeom& g = c.geom;
    if (c.dw_cell >= 0 || g.groups != 1 || g.C % 16 != 0 || g.O % 32 != 0) return 0;
    const char* why = "";
    void* const at = placeholder();
    const void* const out = net->tensors[c.output].dtype == DT_I8 ? at : nullptr;
    const void* const res = c.residual >= 0 ? at : nullptr;
    bool w4 = c.wbits == 4;
    int planned = plan_dense(net, c, g, w4, at, (const int8_t*)at, out, res, &why);
    if (planned != 0 && w4) {
        w4 = false;
        planned = plan_dense(net, c, g, w4, at, (const int8_t*)at, out, res, &why);
    }
    if (planned != 0) return 0;
    if (int rc = choose_dense(net, c, w4, at, (const int8_t*)at)) return rc;
    if (w4 && c.engine == ENG_TCGEN05 && c.fast.enabled && c.inputs[0] != 0 && c.residual != 0 && out)
        if (int rc = plan_widened_cell(net, c, at, (const int8_t*)at, at, res)) return rc;
    *dense = c.probed = true;
    return 0;
}

// What probe_dense found for a cell does not hold any more
static void forget_probe(CellRec& c)
{
    cudaFree(c.d_fast);
    c.d_fast = nullptr;
    c.fast = FastQuant{};
    c.probed = false;
    c.w8 = CellRec::W8_NONE;
}

// Pairs of convolutions whose outputs only meet in a sum, the branch and the projection of a residual block's first unit: the branch is computed by the
// kernel of the later one, so its input lives until then and its output is not stored
static int settle_duals(n2d2b_net* net)
{
    std::vector<int> consumers(net->tensors.size(), 0);
    for (const CellRec& c : net->cells)
        if (!c.skipped)
            for (int i : c.inputs) consumers[i]++;
    const void* const at = placeholder();
    const int8_t* const w = (const int8_t*)at;
    bool packed = false;
    for (size_t bi = 0; bi < net->cells.size(); ++bi) {
        CellRec& b = net->cells[bi];
        if (b.skipped || b.type != CELL_CONV || b.residual <= 0 || b.inputs[0] == 0) continue;
        const int ai = net->tensors[b.residual].producer;
        if (ai < 0 || ai >= (int)bi || consumers[b.residual] != 1) continue;
        CellRec& a = net->cells[ai];
        if (a.skipped || a.type != CELL_CONV || a.residual >= 0 || a.output != b.residual || a.inputs[0] == 0 || a.geom.groups != 1) continue;
        b.dual_branch = ai;
        bool both = false;
        if (int rc = probe_dense(net, a, &both)) return rc;
        if (both)
            if (int rc = probe_dense(net, b, &both)) return rc;
        if (!both || !make_dual(net, b, at, w, at, w, at)) {
            b.dual_branch = -1;
            forget_probe(b);   // (its constants may be those of the shared kernel)
            continue;
        }
        a.dual_sum = (int)bi;
        b.inputs.push_back(a.inputs[0]);
        b.dual_always = !b.plan.w4;
        packed = packed || b.plan.w4;
    }
    if (!packed) return 0;
    // packed weights share a kernel where they are widened: in every call, if a single image is enough for that
    long long macs = 0;
    for (CellRec& c : net->cells) {
        bool dense = false;
        if (c.skipped || (c.type != CELL_CONV && c.type != CELL_FC) || c.wbits != 4) continue;
        if (int rc = probe_dense(net, c, &dense)) return rc;
        if (c.w8 != CellRec::W8_NONE) macs += cell_macs(c);
    }
    for (CellRec& b : net->cells) {
        if (b.dual_branch < 0 || !b.plan.w4) continue;
        CellRec& a = net->cells[b.dual_branch];
        auto both = [&](int call) { return widens_in(net, a, macs, call, call) && widens_in(net, b, macs, call, call); };
        if (both(1)) {
            b.dual_always = true;
        } else if (!both(net->max_batch)) {
            a.dual_sum = b.dual_branch = -1;   // they never share a kernel: the branch's input dies with the branch
            b.inputs.pop_back();
            forget_probe(b);
        }
    }
    return 0;
}

// Expansions with a residual sum whose reader is the next cell, a 1x1 one: the kernel of the first writes the output of both, so the second's buffer
// is taken while the first's operands still have theirs
static int settle_chains(n2d2b_net* net)
{
    const void* const at = placeholder();
    const int8_t* const w = (const int8_t*)at;
    for (size_t i = 0; i < net->cells.size(); ++i) {
        CellRec& c = net->cells[i];
        if (c.skipped || c.type != CELL_CONV || c.residual <= 0 || c.inputs[0] == 0 || c.wbits != 8 || c.dual_branch >= 0) continue;
        size_t j = i + 1;
        while (j < net->cells.size() && net->cells[j].skipped) ++j;
        if (j == net->cells.size()) continue;
        CellRec& p = net->cells[j];
        if (p.type != CELL_CONV || p.residual >= 0 || p.inputs.size() != 1 || p.inputs[0] != c.output || p.wbits != 8 || p.dual_sum >= 0) continue;
        if (!chain_eligible(c.geom, p.geom) || net->tensors[p.output].dtype != DT_I8) continue;
        // (few row tiles: by themselves the two cells spread their columns over more multiprocessors.  64 -> 256 -> 64 channels with the sum behind them, 7 tiles 16.1
        // us as two kernels, 17.3 as one; 13 16.0 / 17.5; 25 16.8 / 16.9, to 128 channels 18.8 / 17.2; 49 20.0 / 18.9)
        if (((long long)net->max_batch * c.geom.oH * c.geom.oW + 127) / 128 * 7 < net->num_sms) continue;
        c.chain_next = (int)j;
        bool both = false;
        if (int rc = probe_dense(net, c, &both)) return rc;
        if (both)
            if (int rc = probe_dense(net, p, &both)) return rc;
        if (!both || !make_chain(net, c, at, w, at, at, w)) {
            c.chain_next = -1;
            continue;
        }
        p.chain_prev = (int)i;
    }
    return 0;
}

static int plan_duals(n2d2b_net* net)
{
    for (CellRec& b : net->cells) {
        if (b.dual_branch < 0) continue;
        CellRec& a = net->cells[b.dual_branch];
        const bool packed = a.plan.w4;
        if (!make_dual(net, b, tensor_ptr(net, a.inputs[0], nullptr), packed ? (const int8_t*)net->d_w8 + a.w8_offset : a.d_weights, tensor_ptr(net, b.inputs[0], nullptr),
                       packed ? (const int8_t*)net->d_w8 + b.w8_offset : b.d_weights, tensor_ptr(net, b.output, nullptr)))
            return fail(N2D2B_ERR_STATE, "internal: a branch and its projection without a plan");
        b.dual_on = true;
        if (use_dual(net, b, net->max_batch, net->max_batch)) net->launches--;
        else if (b.dual_always) return fail(N2D2B_ERR_STATE, "internal: a branch without a buffer");
    }
    return 0;
}

static int plan_chains(n2d2b_net* net)
{
    for (CellRec& c : net->cells) {
        if (c.chain_next < 0) continue;
        if (!make_chain(net, c, tensor_ptr(net, c.inputs[0], nullptr), c.d_weights, tensor_ptr(net, c.output, nullptr), tensor_ptr(net, c.residual, nullptr),
                        net->cells[c.chain_next].d_weights))
            return fail(N2D2B_ERR_STATE, "internal: an expansion and the cell behind it without a plan");
        net->launches--;
    }
    return 0;
}

// A chain of convolutions, poolings and fully-connected cells whose weights fit one SM's shared memory runs as one kernel
// (small_net.cu).  The bound on the arithmetic keeps out what the tensor cores do better: 2^20 multiply-accumulates
// take an SM about 8 us there, and a batch of b images b / 148 times that.
static int plan_small_net(n2d2b_net* net)
{
    if (net->flags & (N2D2B_KEEP_ALL_OUTPUTS | N2D2B_NO_FUSION | N2D2B_FORCE_SIMT | N2D2B_FORCE_IM2COL | N2D2B_EXACT64_EPILOGUE
                      | N2D2B_FORCE_PAIR))
        return 0;
    long long macs = 0, weights = 0;
    int tensor = 0;
    for (const CellRec& c : net->cells) {
        if (c.skipped || c.residual >= 0 || c.inputs.size() != 1 || c.inputs[0] != tensor) return 0;
        if (c.type != CELL_CONV && c.type != CELL_FC && c.type != CELL_POOL) return 0;
        if (net->tensors[tensor].dtype != DT_I8 || net->tensors[c.output].dtype != DT_I8) return 0;
        if (c.type != CELL_POOL) {
            if (c.geom.groups != 1 || c.geom.dX != 1) return 0;
            macs += (long long)c.geom.oH * c.geom.oW * c.geom.O * c.geom.kH * c.geom.kW * c.geom.C;
            weights += (long long)c.weights.size();
        }
        if ((long long)net->tensors[c.output].elems() * net->tensors[c.output].C >= (1ll << 32)) return 0;   // exact quotients
        tensor = c.output;
    }
    if (macs > (1 << 20) || weights > 160 * 1024 || net->cells.size() > SMALL_NET_CELLS) return 0;
    SmallNetPlan p;
    for (const CellRec& c : net->cells) {
        const int in_u = net->tensors[c.inputs[0]].is_unsigned, out_u = net->tensors[c.output].is_unsigned;
        if (c.type == CELL_POOL) {
            small_net_add_pool(&p, c.pgeom, in_u);
            continue;
        }
        std::vector<int32_t> words;
        const int form = build_rescale(c.q, c.geom.O, (long long)c.geom.kH * c.geom.kW * c.geom.C * 255ll * 128ll, words);
        small_net_add_conv(&p, c.geom, in_u, out_u, c.weights.data(), form, words.data(), c.geom.O, c.q.dev);
    }
    if (!small_net_finish(&p, (int)net->tensors[tensor].bytes_per_image())) return 0;
    CUDA_TRY(cudaMalloc(&net->d_small, p.blob.size()));
    CUDA_TRY(cudaMemcpy(net->d_small, p.blob.data(), p.blob.size(), cudaMemcpyHostToDevice));
    p.blob.shrink_to_fit();
    net->small = std::move(p);
    return 0;
}

// Whether the dot-product kernel is the faster one for a 3x3 depthwise layer in a call of `batch` images.  The block-diagonal form on
// the tensor cores moves whole bands of large maps at a time: it is even or ahead where there are many pixels of few channels (256
// images: 56 x 56 x 128 70 us against 74, 112 x 112 x 32 73 / 74), behind on deep maps (14 x 14 x 512 31 / 24, 7 x 7 x 1024 30 / 17) and
// in small calls, whose bands leave SMs idle (33 images: 112 x 112 x 32 23 / 16, 14 x 14 x 512 12.4 / 10.3).
static bool dw3x3_faster(const ConvGeom& g, int batch)
{
    return g.C >= 256 || (long long)batch * g.oH * g.oW * g.C < (1ll << 24);
}

// Whether a cell that has both forms runs on the dot-product kernel in a call of `batch` images (a cell for which that holds up to
// max_batch has no other form, see finalize)
static bool use_dw3x3(const CellRec& c, int batch) { return c.d_dw3x3 && dw3x3_faster(c.geom, batch); }

static int plan_dwpw(n2d2b_net* net, CellRec& c);
int n2d2b_net_finalize(n2d2b_net* net, int max_batch, unsigned flags)
{
    if (!net) return fail(N2D2B_ERR_INVALID, "net must not be NULL");
    if (net->finalized) return fail(N2D2B_ERR_STATE, "the network is already finalized");
    if (net->cells.empty()) return fail(N2D2B_ERR_STATE, "the network has no cells");
    if (max_batch < 1) return fail(N2D2B_ERR_INVALID, "max_batch must be positive");
    CUDA_TRY(cudaSetDevice(net->device));
    net->max_batch = max_batch;
    net->flags = flags;
    if (!(flags & N2D2B_NO_FUSION)) fuse_residuals(net);
    if (!(flags & (N2D2B_NO_FUSION | N2D2B_KEEP_ALL_OUTPUTS | N2D2B_FORCE_SIMT | N2D2B_EXACT64_EPILOGUE)))
        if (int rc = fuse_stem_pool(net)) return rc;
    if (!(flags & (N2D2B_NO_FUSION | N2D2B_KEEP_ALL_OUTPUTS | N2D2B_FORCE_SIMT | N2D2B_EXACT64_EPILOGUE | N2D2B_FORCE_DEPTHWISE_TENSOR | N2D2B_FORCE_IM2COL
                   | N2D2B_FORCE_PAIR)))
        if (int rc = fuse_depthwise(net)) return rc;
    if (!(flags & (N2D2B_NO_FUSION | N2D2B_KEEP_ALL_OUTPUTS | N2D2B_FORCE_SIMT | N2D2B_EXACT64_EPILOGUE | N2D2B_FORCE_IM2COL | N2D2B_FORCE_PAIR))) {
        if (int rc = settle_duals(net)) return rc;
        if (int rc = settle_chains(net)) return rc;
    }
    net->head_limit = head_candidate_prefix(net);
    if (int rc = plan_buffers(net)) return rc;
    CUDA_TRY(cudaMalloc(&net->d_status, 64));
    CUDA_TRY(cudaMemset(net->d_status, 0, 64));
    net->launches = 0;
    for (CellRec& c : net->cells) {
        if (c.skipped) continue;
        net->launches++;
        if (c.type == CELL_POOL) { c.engine = ENG_POOL; continue; }
        if (int rc = upload_quant(c.q)) return rc;
        if (c.has_q2)
            if (int rc = upload_quant(c.q2)) return rc;
        if (c.type == CELL_SUM || c.type == CELL_SCALING) { c.engine = ENG_SUM; continue; }
        // conv / fc: choose the kernel family and lay the weights out for it
        const ConvGeom& g = c.geom;
        if (c.dw_cell >= 0) {
            if (int rc = plan_dwpw(net, c)) return rc;
            continue;
        }
        const bool depthwise = (c.type == CELL_CONV && g.groups == g.C && g.Cg == 1 && g.Og == 1 && g.C % 16 == 0
                                && g.groups > 1 && c.residual < 0
                                && net->tensors[c.output].dtype == DT_I8);
        std::vector<int8_t> laid = c.weights;
        const bool stem = !depthwise && c.type == CELL_CONV && !(flags & N2D2B_FORCE_SIMT) && c.residual < 0
                          && stem_eligible(g) && net->tensors[c.output].dtype == DT_I8 && !(flags & N2D2B_EXACT64_EPILOGUE);
        if (stem) {
            if (!c.d_fast)
                if (int rc = upload_fast(c, net->tensors[c.output])) return rc;
            if (c.fast.enabled && stem_s2d_eligible(g)) {
                // stride 2: space-to-depth image, no gather
                std::vector<int8_t> arranged(c.pool_first ? stem_pool_weight_bytes(g) : stem_s2d_weight_bytes(g));
                if (c.pool_first) stem_pool_arrange_weights(g, c.weights.data(), arranged.data());
                else stem_s2d_arrange_weights(g, c.weights.data(), arranged.data());
                CUDA_TRY(cudaMalloc((void**)&c.d_weights, arranged.size() + 256));
                CUDA_TRY(cudaMemcpy(c.d_weights, arranged.data(), arranged.size(), cudaMemcpyHostToDevice));
                c.d_weight_bytes = arranged.size();
                int Hs = 0, Ws = 0;
                stem_s2d_dims(g, &Hs, &Ws);
                CUDA_TRY(cudaMalloc(&c.d_pad4, (size_t)max_batch * Hs * Ws * 16 + 256));
                const char* why = "";
                const int uns = net->tensors[c.inputs[0]].is_unsigned;
                if ((c.pool_first ? stem_pool_make_plan(&c.stem_pool, c.d_pad4, c.d_weights, g, c.fused_pool, max_batch, uns, net->num_sms, &why)
                                  : stem_s2d_make_plan(&c.stem2, c.d_pad4, c.d_weights, g, max_batch, uns, net->num_sms, &why,
                                                       c.pool_fused ? &c.fused_pool : nullptr)) == 0) {
                    ConvGeom gb = g;
                    gb.B = max_batch;
                    if (!c.pool_first || !stem_pool_takes_image(c.stem_pool, gb, nullptr)) net->launches++;   // (of an aligned image)
                    c.engine = ENG_STEM_S2D;
                    continue;
                }
                if (c.pool_fused) return fail(N2D2B_ERR_STATE, "internal: the fused first layer has no plan (%s)", why);
                cudaFree(c.d_weights);
                c.d_weights = nullptr;
                cudaFree(c.d_pad4);
                c.d_pad4 = nullptr;
            }
            if (c.fast.enabled) {
                std::vector<int8_t> arranged(stem_weight_bytes(g));
                stem_arrange_weights(g, c.weights.data(), arranged.data());
                CUDA_TRY(cudaMalloc((void**)&c.d_weights, arranged.size() + 256));
                CUDA_TRY(cudaMemcpy(c.d_weights, arranged.data(), arranged.size(), cudaMemcpyHostToDevice));
                c.d_weight_bytes = arranged.size();
                const char* why = "";
                if (stem_make_plan(&c.stem, c.d_weights, g, net->tensors[c.inputs[0]].is_unsigned, net->num_sms, &why) == 0) {
                    int Hp = 0, Wp = 0;
                    stem_padded_dims(g, &Hp, &Wp);
                    CUDA_TRY(cudaMalloc(&c.d_pad4, (size_t)max_batch * Hp * Wp * 4 + 256));
                    net->launches++;
                    c.engine = ENG_STEM;
                    continue;
                }
                cudaFree(c.d_weights);
                c.d_weights = nullptr;
            }
            cudaFree(c.d_fast);
            c.d_fast = nullptr;
            c.fast = FastQuant{};
        }
        if (depthwise) {
            c.engine = ENG_DEPTHWISE;
            if (!(flags & N2D2B_EXACT64_EPILOGUE))
                if (int rc = upload_fast(c, net->tensors[c.output])) return rc;
            // [C][kH][kW] -> [kH][kW][C]: four or sixteen channels of a tap are one load
            const int taps = g.kH * g.kW;
            for (int ch = 0; ch < g.C; ++ch)
                for (int t = 0; t < taps; ++t) laid[(size_t)t * g.C + ch] = c.weights[(size_t)ch * taps + t];
            // The block-diagonal form is made only where a call within max_batch can take it (the dot-product kernel's rule holds for
            // every smaller call where it holds for max_batch); the dot-product weights then follow it in the same block.
            const bool dot = c.fast.enabled && !(flags & (N2D2B_FORCE_SIMT | N2D2B_FORCE_DEPTHWISE_TENSOR)) && depthwise3x3_eligible(g);
            const bool tensor = c.fast.enabled && !(flags & N2D2B_FORCE_SIMT) && !(dot && dw3x3_faster(g, max_batch));
            auto alloc_blocks = [&](size_t bytes) -> int {
                c.d_weight_bytes = bytes + (dot ? laid.size() : 0);
                CUDA_TRY(cudaMalloc((void**)&c.d_weights, c.d_weight_bytes + 256));
                return 0;
            };
            auto upload_blocks = [&](std::vector<int8_t>& rows) -> int {
                if (dot) {
                    c.d_dw3x3 = c.d_weights + rows.size();
                    rows.insert(rows.end(), laid.begin(), laid.end());
                }
                CUDA_TRY(cudaMemcpy(c.d_weights, rows.data(), rows.size(), cudaMemcpyHostToDevice));
                return 0;
            };
            auto drop_blocks = [&] {
                cudaFree(c.d_weights);
                c.d_weights = nullptr;
                c.d_weight_bytes = 0;
            };
            // Stride-1 layers whose channels come in whole groups of 32 run on the tensor cores as block-diagonal
            // groups (patch kernel); it needs the 32-bit epilogue
            ConvGeom gb = g;
            gb.B = max_batch;
            const char* why = "";
            const void* in_ptr = tensor_ptr(net, c.inputs[0], nullptr);
            const void* enc_ptr = in_ptr ? in_ptr : placeholder();
            if (tensor && patch_eligible(gb)) {
                std::vector<int8_t> arranged(patch_dw_weight_bytes(g));
                if (int rc = alloc_blocks(arranged.size())) return rc;
                if (patch_make_plan(&c.patch, enc_ptr, c.d_weights, gb, net->tensors[c.inputs[0]].is_unsigned, net->num_sms, &why) == 0) {
                    patch_dw_arrange_weights(g, c.weights.data(), arranged.data());
                    if (int rc = upload_blocks(arranged)) return rc;
                    c.engine = ENG_PATCH;
                    c.plan_input = in_ptr;   // nullptr = re-encoded with the real input at the first forward pass
                    continue;
                }
                drop_blocks();
            }
            // Strided ones (and whatever else the patch kernel leaves) take the implicit-GEMM kernel the same way: one
            // 64-column tile per group of 64 channels, im2col loads of the group's channel slice
            if (tensor && igemm_dw_group(gb)) {
                std::vector<int8_t> arranged(igemm_dw_weight_bytes(g));
                if (int rc = alloc_blocks(arranged.size())) return rc;
                if (igemm_make_plan(&c.plan, enc_ptr, c.d_weights, tensor_ptr(net, c.output, nullptr), nullptr, gb,
                                    net->tensors[c.inputs[0]].is_unsigned, 1, 0, net->num_sms, &why, 0, 0) == 0
                    && igemm_uses_fast_epilogue(c.plan, c.fast, false, DT_I8)) {
                    igemm_dw_arrange_weights(g, c.weights.data(), arranged.data());
                    const int pb = igemm_perm_block(c.plan);
                    std::vector<int8_t> rows(arranged.size());
                    igemm_permute_weights(arranged.data(), rows.data(), g.C, arranged.size() / (size_t)g.C, pb);
                    c.plan.perm = pb;
                    if (int rc = upload_blocks(rows)) return rc;
                    c.engine = ENG_TCGEN05;
                    c.plan_input = in_ptr;
                    continue;
                }
                drop_blocks();
            }
        } else {
            c.engine = ENG_SIMT;
        }
        // Packed 4-bit weights stay packed in HBM when the cell runs on the implicit-GEMM kernel, whose expansion
        // warps unpack them tile by tile; every other kernel takes them widened to int8.
        const bool igemm_shape = !depthwise && !(flags & N2D2B_FORCE_SIMT) && g.groups == 1 && g.C % 16 == 0;
        bool w4 = c.wbits == 4 && igemm_shape;
        auto pack4 = [](const std::vector<int8_t>& w) {
            std::vector<int8_t> p(w.size() / 2);
            for (size_t i = 0; i < p.size(); ++i) p[i] = (int8_t)(((w[2 * i] & 0xF) << 4) | (w[2 * i + 1] & 0xF));
            return p;
        };
        // Output channels that are not a multiple of 32: take the 32-bit epilogue on a padded copy (see pad_O)
        ConvGeom gplan = g;
        if (igemm_shape && !w4 && g.O % 32 != 0 && c.residual < 0 && net->tensors[c.output].dtype == DT_I8
            && !(flags & N2D2B_EXACT64_EPILOGUE)) {
            if (int rc = upload_fast(c, net->tensors[c.output])) return rc;
            if (c.fast.enabled) {
                c.pad_O = (g.O + 63) & ~63;
                gplan.O = c.pad_O;
                laid.resize((size_t)c.pad_O * g.kH * g.kW * g.Cg, 0);
                CUDA_TRY(cudaMalloc(&c.d_colpad, (size_t)max_batch * g.oH * g.oW * c.pad_O + 256));
            }
        }
        c.d_weight_bytes = w4 ? laid.size() / 2 : laid.size();
        CUDA_TRY(cudaMalloc((void**)&c.d_weights, c.d_weight_bytes + 256));
        CUDA_TRY(cudaMemset(c.d_weights, 0, c.d_weight_bytes + 256));
        if (!w4) CUDA_TRY(cudaMemcpy(c.d_weights, laid.data(), laid.size(), cudaMemcpyHostToDevice));
        if (igemm_shape) {
            const char* why = "";
            // the network input pointer is only known at forward time; its map is encoded again on first use
            const void* in_ptr = tensor_ptr(net, c.inputs[0], nullptr);
            const void* enc_ptr = in_ptr ? in_ptr : placeholder();
            const void* out_ptr = c.pad_O ? c.d_colpad : net->tensors[c.output].dtype == DT_I8 ? tensor_or_placeholder(net, c.output) : nullptr;
            const void* res_ptr = c.residual >= 0 ? tensor_or_placeholder(net, c.residual) : nullptr;
            int planned = plan_dense(net, c, gplan, w4, enc_ptr, c.d_weights, out_ptr, res_ptr, &why);
            if (planned != 0 && w4) {
                // no room for the packed variant: widen the weights after all
                w4 = false;
                cudaFree(c.d_weights);
                c.d_weights = nullptr;
                c.d_weight_bytes = laid.size();
                CUDA_TRY(cudaMalloc((void**)&c.d_weights, laid.size() + 256));
                CUDA_TRY(cudaMemset(c.d_weights, 0, laid.size() + 256));
                CUDA_TRY(cudaMemcpy(c.d_weights, laid.data(), laid.size(), cudaMemcpyHostToDevice));
                planned = plan_dense(net, c, gplan, w4, enc_ptr, c.d_weights, out_ptr, res_ptr, &why);
            }
            if (planned == 0) {
                if (int rc = choose_dense(net, c, w4, enc_ptr, c.d_weights)) return rc;
                c.plan_input = in_ptr;  // nullptr = must be re-encoded with the real input
                // weight rows in the permuted order that the 32-bit epilogue reads (see perm_block)
                if (c.engine == ENG_PATCH) {
                    std::vector<int8_t> rows(laid.size());
                    patch_permute_weights(laid.data(), rows.data(), g.O, (size_t)g.kH * g.kW * g.Cg);
                    CUDA_TRY(cudaMemcpy(c.d_weights, rows.data(), rows.size(), cudaMemcpyHostToDevice));
                } else if (c.plan.perm || w4) {
                    std::vector<int8_t> rows = laid;
                    if (c.plan.perm) igemm_permute_weights(laid.data(), rows.data(), gplan.O, (size_t)g.kH * g.kW * g.Cg, c.plan.perm);
                    if (c.pad_O && !stores_rows(c, c.plan)) net->launches++;   // the copy that drops the padding
                    if (w4) rows = pack4(rows);
                    CUDA_TRY(cudaMemcpy(c.d_weights, rows.data(), rows.size(), cudaMemcpyHostToDevice));
                }
            } else if (w4 || c.pad_O) {
                return fail(N2D2B_ERR_STATE, "internal: a packed or padded cell without a plan (%s)", why);
            }
        }
    }
    if (int rc = plan_widened(net)) return rc;
    if (int rc = plan_small_net(net)) return rc;
    if (net->d_small) net->launches = 1;
    CUDA_TRY(cudaMalloc(&net->d_stage_in, net->tensors[0].bytes_per_image() * (size_t)max_batch + 256));
    CUDA_TRY(cudaMalloc(&net->d_stage_out,
                        net->tensors[final_tensor_of(net)].bytes_per_image() * (size_t)max_batch + 256));
    CUDA_TRY(cudaStreamCreateWithFlags(&net->copy_stream, cudaStreamNonBlocking));
    for (cudaEvent_t& e : net->slice_ready) CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    CUDA_TRY(cudaEventCreateWithFlags(&net->stage_free, cudaEventDisableTiming));
    // Leading cells that the host-buffer entry point runs slice by slice while later slices of the batch
    // are still being uploaded: every cell works image by image, so a slice is an offset (in images for the
    // pointer-based kernels, in rows of the tensor maps for the tensor-core ones).  The head ends where the
    // per-image tensors get small (after the first stage of a ResNet): from there on a launch per slice would
    // cost more in fixed launch time than the overlap gains.
    net->head_cells = 0;
    for (size_t ci = 0; ci < net->cells.size(); ++ci) {
        const CellRec& c = net->cells[ci];
        bool sliceable = true;
        if (!c.skipped) {
            const bool mapped = c.engine == ENG_TCGEN05 || c.engine == ENG_PATCH || c.engine == ENG_DWPW;
            const bool pointer_based = (c.engine == ENG_STEM || c.engine == ENG_STEM_S2D || c.engine == ENG_POOL
                                        || c.engine == ENG_DEPTHWISE || c.engine == ENG_SIMT)
                                       && c.residual < 0 && c.inputs.size() == 1;
            sliceable = c.type != CELL_FC && (mapped || pointer_based);
            const TensorRec& t = net->tensors[c.output];
            if ((long long)t.H * t.W < 2048) sliceable = false;
        }
        if (!sliceable || (int)ci >= net->head_limit) break;
        net->head_cells = (int)ci + 1;
    }
    // cells that share a kernel are in the head together or not at all
    for (int ci = net->head_cells - 1; ci >= 0; --ci) {
        const CellRec& c = net->cells[ci];
        if (c.dual_sum >= net->head_cells || c.chain_next >= net->head_cells) net->head_cells = ci;
    }
    if (int rc = plan_duals(net)) return rc;
    if (int rc = plan_chains(net)) return rc;
    for (int k = 0; k < 2; ++k) {
        CUDA_TRY(cudaEventCreateWithFlags(&net->pipe_uploaded[k], cudaEventDisableTiming));
        CUDA_TRY(cudaEventCreateWithFlags(&net->pipe_computed[k], cudaEventDisableTiming));
        CUDA_TRY(cudaEventCreateWithFlags(&net->pipe_done[k], cudaEventDisableTiming));
    }
    CUDA_TRY(cudaStreamCreateWithFlags(&net->download_stream, cudaStreamNonBlocking));
    net->finalized = true;
    return 0;
}

static int fuse_stem_pool(n2d2b_net* net)
{
    std::vector<int> consumers(net->tensors.size(), 0);
    for (const CellRec& c : net->cells)
        if (!c.skipped)
            for (int i : c.inputs) consumers[i]++;
    for (size_t ci = 0; ci < net->cells.size(); ++ci) {
        CellRec& c = net->cells[ci];
        if (c.skipped || c.type != CELL_CONV || c.residual >= 0 || c.inputs[0] != 0) continue;
        if (!stem_eligible(c.geom) || !stem_s2d_eligible(c.geom)) continue;
        const int t = c.output;
        if (consumers[t] != 1 || net->tensors[t].dtype != DT_I8) continue;
        int pj = -1;
        for (size_t cj = ci + 1; cj < net->cells.size(); ++cj)
            if (!net->cells[cj].skipped && net->cells[cj].inputs.size() == 1 && net->cells[cj].inputs[0] == t) { pj = (int)cj; break; }
        if (pj < 0 || net->cells[pj].type != CELL_POOL) continue;
        CellRec& p = net->cells[pj];
        const bool first = stem_pool_eligible(c.geom, p.pgeom), bytes = (net->flags & N2D2B_FUSE_FIRST_POOL) && stem_s2d_pool_eligible(c.geom, p.pgeom);
        if (!first && !bytes) continue;
        // the first-layer kernels need the 32-bit epilogue
        if (int rc = upload_fast(c, net->tensors[t])) return rc;
        c.pool_first = first && c.fast.enabled && c.fast.monotone;
        if (!c.fast.enabled || !(c.pool_first || bytes)) continue;
        c.pool_fused = true;
        c.fused_pool = p.pgeom;
        net->tensors[t].readable = false;
        net->tensors[t].buffer = -2;   // never materialised
        c.output = p.output;
        net->tensors[p.output].producer = (int)ci;
        p.skipped = true;
        p.engine = ENG_FUSED;
    }
    return 0;
}

static int fuse_depthwise(n2d2b_net* net)
{
    std::vector<int> consumers(net->tensors.size(), 0);
    for (const CellRec& c : net->cells)
        if (!c.skipped)
            for (int i : c.inputs) consumers[i]++;
    for (size_t ci = 0; ci < net->cells.size(); ++ci) {
        CellRec& c = net->cells[ci];
        // (the maps of the input want its address, which of the caller's buffer only the forward pass knows)
        if (c.skipped || c.type != CELL_CONV || c.residual >= 0 || c.inputs.size() != 1 || c.inputs[0] == 0) continue;
        const int t = c.output;
        const TensorRec &tin = net->tensors[c.inputs[0]], &tmid = net->tensors[t];
        if (consumers[t] != 1 || tin.dtype != DT_I8 || tmid.dtype != DT_I8 || !tin.is_unsigned || !tmid.is_unsigned || c.wbits != 8) continue;
        int pj = -1;
        for (size_t cj = ci + 1; cj < net->cells.size(); ++cj)
            if (!net->cells[cj].skipped && net->cells[cj].inputs.size() == 1 && net->cells[cj].inputs[0] == t) { pj = (int)cj; break; }
        if (pj < 0) continue;
        CellRec& p = net->cells[pj];
        if (p.type != CELL_CONV || p.residual >= 0 || p.wbits != 8 || net->tensors[p.output].dtype != DT_I8 || !dwpw_eligible(c.geom, p.geom)) continue;
        if (!dwpw_faster(c.geom, p.geom.O, net->max_batch, net->num_sms)) continue;
        ConvGeom g = c.geom;
        g.B = net->max_batch;
        DwPwPlan probe{};
        probe.d = g;
        probe.N = p.geom.O;
        probe.num_sms = net->num_sms;
        if (dwpw_set_batch(&probe, net->max_batch)) continue;
        if (int rc = upload_fast(c, tmid)) return rc;
        if (int rc = upload_fast(p, net->tensors[p.output])) return rc;
        if (!dwpw_takes_forms(c.fast, p.fast)) {
            for (CellRec* x : {&c, &p}) {
                cudaFree(x->d_fast);
                x->d_fast = nullptr;
                x->fast = FastQuant{};
            }
            continue;
        }
        p.dw_cell = (int)ci;
        p.inputs[0] = c.inputs[0];
        net->tensors[t].readable = false;
        net->tensors[t].buffer = -2;   // never materialised
        c.skipped = true;
        c.engine = ENG_FUSED;
    }
    return 0;
}

// Weights and plan of a 1x1 cell that computes the depthwise cell in front of it
static int plan_dwpw(n2d2b_net* net, CellRec& c)
{
    CellRec& d = net->cells[c.dw_cell];
    std::vector<uint32_t> words(dwpw_depthwise_words(d.geom));
    dwpw_arrange_depthwise(d.geom, d.weights.data(), words.data());
    d.d_weight_bytes = words.size() * 4;
    CUDA_TRY(cudaMalloc((void**)&d.d_weights, d.d_weight_bytes));
    CUDA_TRY(cudaMemcpy(d.d_weights, words.data(), d.d_weight_bytes, cudaMemcpyHostToDevice));
    std::vector<int8_t> rows(c.weights.size());
    igemm_permute_weights(c.weights.data(), rows.data(), c.geom.O, (size_t)c.geom.C, 32);
    c.d_weight_bytes = rows.size();
    CUDA_TRY(cudaMalloc((void**)&c.d_weights, rows.size() + 256));
    CUDA_TRY(cudaMemcpy(c.d_weights, rows.data(), rows.size(), cudaMemcpyHostToDevice));
    const char* why = "";
    if (dwpw_make_plan(&c.dwpw, tensor_ptr(net, c.inputs[0], nullptr), d.d_weights, c.d_weights, d.geom, c.geom.O, net->max_batch, net->num_sms, &why))
        return fail(N2D2B_ERR_STATE, "internal: a depthwise and 1x1 cell without a plan (%s)", why);
    c.engine = ENG_DWPW;
    return 0;
}

// ---- forward --------------------------------------------------------------------------------
// Whether a depthwise cell can read from `in`, which only the caller's own buffer may fail.  A cell that has the block-diagonal form
// takes what that form's tensor maps take, whichever kernel runs it; the others what the loads of their kernel do.
static bool depthwise_takes(const n2d2b_net* net, const CellRec& c, int batch, const void* in)
{
    if (((uintptr_t)in & 15) == 0) return true;
    ConvGeom g = c.geom;
    g.B = batch;
    const bool block_form = c.fast.enabled && !(net->flags & N2D2B_FORCE_SIMT) && (patch_eligible(g) || igemm_dw_group(g));
    return !block_form && (uintptr_t)in % depthwise_alignment(g, c.fast) == 0;
}

// Widens the packed weights of cell `c` into the scratch block, or in a large call those of every cell that takes the form, once
static int widen_weights(n2d2b_net* net, const CellRec& c, cudaStream_t s)
{
    const bool all = widen_all(net, net->call_batch);
    if (all && net->call_widened) return 0;
    std::vector<WidenJob> jobs;
    for (const CellRec& x : net->cells) {
        if (x.w8 == CellRec::W8_NONE || (all ? !worth_widening(net, x, net->call_batch) : &x != &c)) continue;
        WidenJob j;
        j.packed = (const uint8_t*)x.d_weights;
        j.dst = (int8_t*)net->d_w8 + x.w8_offset;
        j.rows_src = x.geom.O;
        j.ng_src = x.w8_ng_src;
        j.rows = x.w8_rows;
        j.ng_dst = x.w8_ng_dst;
        j.words = (unsigned)((size_t)x.geom.kH * x.geom.kW * x.geom.C / 8);
        jobs.push_back(j);
    }
    CUDA_TRY(launch_widen_int4(jobs.data(), (int)jobs.size(), s));
    net->call_widened = all;
    return 0;
}

// The implicit GEMM of a cell, and where its columns were padded (into `padded`) its output in place: short launches of a classifier store the wanted
// columns from the registers, others leave them to a copy kernel
static int run_igemm(n2d2b_net* net, const CellRec& c, IgemmPlan p, const Residual& r, void* padded, void* out, int out_dtype, int batch, int img0, cudaStream_t s)
{
    const ConvGeom& g = c.geom;
    p.M = batch * g.oH * g.oW;
    const size_t row0 = (size_t)img0 * g.oH * g.oW;
    if (padded && !img0 && stores_rows(c, p)) {
        CUDA_TRY(launch_igemm(p, c.q.dev, r, c.fast, padded, out_dtype, 0, net->d_status, s, out, g.O));
        return 0;
    }
    CUDA_TRY(launch_igemm(p, c.q.dev, r, c.fast, padded ? padded : out, out_dtype, (int)row0, net->d_status, s));
    if (padded) CUDA_TRY(launch_drop_padded_columns((const uint8_t*)padded + row0 * p.N, p.N, (uint8_t*)out + row0 * g.O, g.O, (size_t)p.M, s));
    return 0;
}

// Runs one cell on images [img0, img0 + batch) of the batch (img0 != 0 only for cells without tensor maps).
static int run_cell(n2d2b_net* net, CellRec& c, const void* d_input, int batch, cudaStream_t s, int img0 = 0)
{
    if (c.dual_sum >= 0 && use_dual(net, net->cells[c.dual_sum], batch, net->call_batch)) return 0;   // computed by the cell that carries the sum
    if (c.chain_prev >= 0) return 0;   // written by the cell in front
    const void* in0 = tensor_ptr(net, c.inputs[0], d_input);
    void* out = tensor_ptr(net, c.output, d_input);
    const TensorRec& tin = net->tensors[c.inputs[0]];
    const TensorRec& tout = net->tensors[c.output];
    if (!in0 || !out) return fail(N2D2B_ERR_STATE, "internal: tensor without a buffer");
    // the tensor-core cells address their tensors through maps encoded over the whole buffers: a batch slice
    // is an offset in rows / images there; every other cell takes offset pointers
    const bool mapped = c.engine == ENG_TCGEN05 || c.engine == ENG_PATCH || c.engine == ENG_DWPW;
    if (img0 && !mapped) {
        if (c.engine == ENG_SUM || c.residual >= 0)
            return fail(N2D2B_ERR_STATE, "internal: this cell cannot run on a slice");
        in0 = (const uint8_t*)in0 + (size_t)img0 * tin.bytes_per_image();
        out = (uint8_t*)out + (size_t)img0 * tout.bytes_per_image();
    }
    Residual r{};
    if (c.residual >= 0) {
        r.ptr = tensor_ptr(net, c.residual, d_input);
        r.is_unsigned = net->tensors[c.residual].is_unsigned;
        r.q2 = c.q2.dev;
    }
    // the maps and the loads of a residual start on 16 bytes; the network's input is the caller's buffer
    if (c.residual == 0 && mapped && ((uintptr_t)r.ptr & 15))
        return fail(N2D2B_ERR_INVALID, "a residual sum cannot read an input at %p: operands must be 16-byte aligned", r.ptr);
    if (c.chain_next >= 0) {
        const CellRec& p = net->cells[c.chain_next];
        const int pixels = c.geom.oH * c.geom.oW;
        CUDA_TRY(launch_chain(c.chain, batch * pixels, c.fast, r.is_unsigned, p.fast, tensor_ptr(net, p.output, d_input), img0 * pixels, net->d_status, s));
        return 0;
    }
    const bool dual = c.dual_branch >= 0 && use_dual(net, c, batch, net->call_batch), widened = use_widened(net, c, batch, net->call_batch);
    if (widened) {
        if (dual)
            if (int rc = widen_weights(net, net->cells[c.dual_branch], s)) return rc;
        if (int rc = widen_weights(net, c, s)) return rc;
    }
    if (dual) {
        const CellRec& a = net->cells[c.dual_branch];
        ConvGeom g = c.geom;
        g.B = batch;
        if (c.dual_patch.proj_in) {
            Residual branch{};
            branch.is_unsigned = net->tensors[a.output].is_unsigned;
            ConvGeom ga = a.geom;
            ga.B = batch;
            if (patch_set_batch(&c.dual_patch, a.geom, batch)) return fail(N2D2B_ERR_INVALID, "patch plan failed for %d images", batch);
            CUDA_TRY(launch_patch(c.dual_patch, ga, img0, branch, c.fast, out, net->d_status, s, &a.fast));
            return 0;
        }
        CUDA_TRY(launch_dual(c.dual, g, a.fast, c.fast, net->tensors[a.output].is_unsigned, img0 * g.oH * g.oW, a.plan.w4, net->d_status, s));
        return 0;
    }
    if (widened) {
        ConvGeom g = c.geom;
        g.B = batch;
        if (c.w8 == CellRec::W8_PATCH) {
            if (patch_set_batch(&c.patch8, c.geom, batch)) return fail(N2D2B_ERR_INVALID, "patch plan failed for %d images", batch);
            CUDA_TRY(launch_patch(c.patch8, g, img0, r, c.fast, out, net->d_status, s));
            return 0;
        }
        return run_igemm(net, c, c.plan8, r, c.d_w8_out, out, DT_I8, batch, img0, s);
    }
    if ((c.engine == ENG_DEPTHWISE || c.d_dw3x3) && !depthwise_takes(net, c, batch, in0))
        return fail(N2D2B_ERR_INVALID, "a depthwise cell cannot read an input at %p: operands must be 16-byte aligned", in0);
    if (use_dw3x3(c, batch)) {
        ConvGeom g = c.geom;
        g.B = batch;
        const size_t in_off = mapped ? (size_t)img0 * tin.bytes_per_image() : 0, out_off = mapped ? (size_t)img0 * tout.bytes_per_image() : 0;
        CUDA_TRY(launch_depthwise3x3((const uint8_t*)in0 + in_off, tin.is_unsigned, c.d_dw3x3, g, c.fast, (uint8_t*)out + out_off, net->num_sms, s));
        return 0;
    }
    switch (c.engine) {
    case ENG_TCGEN05: {
        // tensors of the caller: their address and the images of this call
        const void* const caller_in = c.inputs[0] == 0 ? in0 : nullptr;
        const void* const caller_res = c.residual == 0 ? r.ptr : nullptr;
        if (c.plan_input != in0 || c.plan_res != caller_res || ((caller_in || caller_res) && c.plan_images != img0 + batch)) {
            ConvGeom gb = c.geom;
            gb.B = img0 + batch;
            if (c.pad_O) gb.O = c.pad_O;
            const char* why = "";
            c.plan_images = 0;
            if (igemm_bind_buffers(&c.plan, caller_in, caller_res, gb, &why)) return fail(N2D2B_ERR_INVALID, "tensor-core plan failed: %s", why);
            c.plan_input = in0;
            c.plan_res = caller_res;
            c.plan_images = gb.B;
        }
        return run_igemm(net, c, c.plan, r, c.d_colpad, out, tout.dtype, batch, img0, s);
    }
    case ENG_PATCH: {
        if (patch_as_gemm(net, c, batch)) return run_igemm(net, c, c.plan, r, nullptr, out, tout.dtype, batch, img0, s);
        if (c.plan_input != in0) {
            ConvGeom gb = c.geom;
            gb.B = net->max_batch;
            const char* why = "";
            if (patch_make_plan(&c.patch, in0, c.d_weights, gb, tin.is_unsigned, net->num_sms, &why))
                return fail(N2D2B_ERR_INVALID, "patch plan failed: %s", why);
            c.plan_input = in0;
        }
        if (patch_set_batch(&c.patch, c.geom, batch)) return fail(N2D2B_ERR_INVALID, "patch plan failed for %d images", batch);
        ConvGeom g = c.geom;
        g.B = batch;
        CUDA_TRY(launch_patch(c.patch, g, img0, r, c.fast, out, net->d_status, s));
        break;
    }
    case ENG_DWPW:
        if (dwpw_set_batch(&c.dwpw, batch)) return fail(N2D2B_ERR_INVALID, "depthwise plan failed for %d images", batch);
        CUDA_TRY(launch_dwpw(c.dwpw, img0, net->cells[c.dw_cell].fast, c.fast, out, net->d_status, s));
        break;
    case ENG_STEM_S2D: {
        ConvGeom g = c.geom;
        g.B = batch;
        int Hs = 0, Ws = 0;
        stem_s2d_dims(g, &Hs, &Ws);
        if (c.pool_first) {
            const bool raw = stem_pool_takes_image(c.stem_pool, g, in0);
            if (!raw) CUDA_TRY(launch_s2d_image(in0, g, batch, (uint8_t*)c.d_pad4 + (size_t)img0 * Hs * Ws * 16, s));
            CUDA_TRY(launch_stem_pool(c.stem_pool, g, img0, raw ? in0 : nullptr, c.fast, out, net->d_status, s));
            break;
        }
        if (stem_s2d_set_batch(&c.stem2, c.geom, batch)) return fail(N2D2B_ERR_INVALID, "first-layer plan failed for %d images", batch);
        CUDA_TRY(launch_s2d_image(in0, g, batch, (uint8_t*)c.d_pad4 + (size_t)img0 * Hs * Ws * 16, s));
        CUDA_TRY(launch_stem_s2d(c.stem2, g, img0, c.fast, out, net->d_status, s));
        break;
    }
    case ENG_STEM: {
        ConvGeom g = c.geom;
        g.B = batch;
        int Hp = 0, Wp = 0;
        stem_padded_dims(g, &Hp, &Wp);
        void* in4 = (uint8_t*)c.d_pad4 + (size_t)img0 * Hp * Wp * 4;
        CUDA_TRY(launch_pad_image(in0, g, batch, in4, s));
        CUDA_TRY(launch_stem(c.stem, in4, g, c.fast, out, net->d_status, s));
        break;
    }
    case ENG_SIMT: {
        ConvGeom g = c.geom;
        g.B = batch;
        if (c.type == CELL_FC && c.residual < 0)
            CUDA_TRY(launch_fc_direct(in0, tin.is_unsigned, c.d_weights, batch, g.C, g.O, c.q.dev, out, tout.dtype, s));
        else
            CUDA_TRY(launch_conv_direct(in0, tin.is_unsigned, c.d_weights, g, c.q.dev, r, out, tout.dtype, s));
        break;
    }
    case ENG_DEPTHWISE: {
        ConvGeom g = c.geom;
        g.B = batch;
        CUDA_TRY(launch_conv_depthwise(in0, tin.is_unsigned, c.d_weights, g, c.q.dev, c.fast, out, s));
        break;
    }
    case ENG_POOL: {
        PoolGeom g = c.pgeom;
        g.B = batch;
        if (tin.dtype == DT_I32) CUDA_TRY(launch_pool_i32(in0, g, out, s));
        else CUDA_TRY(launch_pool(in0, tin.is_unsigned, g, out, s));
        break;
    }
    case ENG_SUM: {
        SumInputs ins{};
        ins.n = (int)c.inputs.size();
        for (int k = 0; k < ins.n; ++k) {
            ins.ptr[k] = tensor_ptr(net, c.inputs[k], d_input);
            ins.dtype[k] = net->tensors[c.inputs[k]].dtype;
            ins.is_unsigned[k] = net->tensors[c.inputs[k]].is_unsigned;
        }
        CUDA_TRY(launch_elemwise_sum(ins, (size_t)batch * tout.H * tout.W, tout.C, c.q.dev, out, tout.dtype, s));
        break;
    }
    case ENG_FUSED:
        break;
    }
    return 0;
}

static int forward_impl(n2d2b_net* net, const void* d_input, int batch, void* d_output, cudaStream_t s, float* ms,
                        int nb_cells, int first_cell = 0)
{
    if (!net) return fail(N2D2B_ERR_INVALID, "net must not be NULL");
    if (!net->finalized) return fail(N2D2B_ERR_STATE, "forward before finalize");
    if (batch < 0 || batch > net->max_batch)
        return fail(N2D2B_ERR_TOO_LARGE, "batch %d exceeds the finalized maximum %d", batch, net->max_batch);
    if (batch == 0) return 0;
    if (!d_input) return fail(N2D2B_ERR_INVALID, "d_input must not be NULL");
    CUDA_TRY(cudaSetDevice(net->device));
    const bool one_kernel = net->d_small && first_cell == 0;
    if (first_cell == 0) {   // (else the leading cells of the same call have run)
        net->call_batch = batch;
        net->call_widened = false;
    }
    std::vector<cudaEvent_t> ev;
    if (ms) {
        if (nb_cells != (int)net->cells.size())
            return fail(N2D2B_ERR_INVALID, "ms must have one entry per cell (%d)", (int)net->cells.size());
        ev.resize((one_kernel ? 1 : net->cells.size()) + 1);
        for (auto& e : ev) CUDA_TRY(cudaEventCreate(&e));
        CUDA_TRY(cudaEventRecord(ev[0], s));
    }
    if (one_kernel) {
        CUDA_TRY(launch_small_net(net->small, net->d_small, d_input, batch, tensor_ptr(net, final_tensor_of(net), d_input), d_output,
                                  net->num_sms, s));
        net->last_input = d_input;
        if (!ms) return 0;
        CUDA_TRY(cudaEventRecord(ev[1], s));
        CUDA_TRY(cudaStreamSynchronize(s));
        std::fill(ms, ms + nb_cells, 0.0f);   // the whole network is the first entry
        CUDA_TRY(cudaEventElapsedTime(&ms[0], ev[0], ev[1]));
        for (auto& e : ev) cudaEventDestroy(e);
        return 0;
    }
    for (size_t ci = (size_t)first_cell; ci < net->cells.size(); ++ci) {
        CellRec& c = net->cells[ci];
        if (!c.skipped)
            if (int rc = run_cell(net, c, d_input, batch, s)) return rc;
        if (ms) CUDA_TRY(cudaEventRecord(ev[ci + 1], s));
    }
    const int ft = final_tensor_of(net);
    if (d_output) {
        const TensorRec& t = net->tensors[ft];
        CUDA_TRY(cudaMemcpyAsync(d_output, tensor_ptr(net, ft, d_input), t.bytes_per_image() * (size_t)batch,
                                 cudaMemcpyDeviceToDevice, s));
    }
    net->last_input = d_input;
    if (ms) {
        CUDA_TRY(cudaStreamSynchronize(s));
        for (size_t ci = 0; ci < net->cells.size(); ++ci) CUDA_TRY(cudaEventElapsedTime(&ms[ci], ev[ci], ev[ci + 1]));
        for (auto& e : ev) cudaEventDestroy(e);
    }
    return 0;
}

static int check_status(n2d2b_net* net)
{
    int st = 0;
    CUDA_TRY(cudaMemcpy(&st, net->d_status, sizeof(int), cudaMemcpyDeviceToHost));
    if (st != 0) {
        cudaMemset(net->d_status, 0, sizeof(int));
        return fail(N2D2B_ERR_TIMEOUT, "a tensor-core kernel gave up waiting on a pipeline barrier (role %d)", st);
    }
    return 0;
}

int n2d2b_net_forward(n2d2b_net* net, const void* d_input, int batch, void* d_output, n2d2b_stream stream)
{
    return forward_impl(net, d_input, batch, d_output, (cudaStream_t)stream, nullptr, 0);
}

int n2d2b_net_check(n2d2b_net* net, n2d2b_stream stream)
{
    if (!net) return fail(N2D2B_ERR_INVALID, "net must not be NULL");
    if (!net->finalized) return fail(N2D2B_ERR_STATE, "check before finalize");
    CUDA_TRY(cudaSetDevice(net->device));
    CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
    return check_status(net);
}

int n2d2b_net_selftest_wait_timeout(n2d2b_net* net, unsigned limit_us, n2d2b_stream stream)
{
    if (!net) return fail(N2D2B_ERR_INVALID, "net must not be NULL");
    if (!net->finalized) return fail(N2D2B_ERR_STATE, "selftest before finalize");
    CUDA_TRY(cudaSetDevice(net->device));
    return wait_timeout_selftest(net->d_status, limit_us, (cudaStream_t)stream);
}

int n2d2b_net_profile(n2d2b_net* net, const void* d_input, int batch, void* d_output, float* ms, int nb_cells,
                      n2d2b_stream stream)
{
    if (!ms) return fail(N2D2B_ERR_INVALID, "ms must not be NULL");
    if (int rc = forward_impl(net, d_input, batch, d_output, (cudaStream_t)stream, ms, nb_cells)) return rc;
    return check_status(net);
}

int n2d2b_net_set_slices(n2d2b_net* net, int nb_slices)
{
    if (!net) return fail(N2D2B_ERR_INVALID, "net must not be NULL");
    if (nb_slices < 0 || nb_slices > 8) return fail(N2D2B_ERR_INVALID, "nb_slices must be in 0..8 (0 = automatic)");
    net->forced_slices = nb_slices;
    return 0;
}

static int host_call_checks(n2d2b_net* net, const void* h_input, int batch, void* h_output)
{
    if (!net) return fail(N2D2B_ERR_INVALID, "net must not be NULL");
    if (!net->finalized) return fail(N2D2B_ERR_STATE, "forward before finalize");
    if (batch < 0 || batch > net->max_batch)
        return fail(N2D2B_ERR_TOO_LARGE, "batch %d exceeds the finalized maximum %d", batch, net->max_batch);
    if (batch > 0 && (!h_input || !h_output)) return fail(N2D2B_ERR_INVALID, "host buffers must not be NULL");
    return 0;
}

int n2d2b_net_forward_host(n2d2b_net* net, const void* h_input, int batch, void* h_output, n2d2b_stream stream)
{
    if (int rc = host_call_checks(net, h_input, batch, h_output)) return rc;
    if (batch == 0) return 0;
    CUDA_TRY(cudaSetDevice(net->device));
    cudaStream_t s = (cudaStream_t)stream;
    const size_t in_bytes = net->tensors[0].bytes_per_image() * (size_t)batch;
    const int ft = final_tensor_of(net);
    const size_t out_bytes = net->tensors[ft].bytes_per_image() * (size_t)batch;
    void* d_in = net->d_stage_in;
    void* d_out = net->d_stage_out;
    // Slices of about 128 images, at most 8.  The upload is slower than the leading cells, so what the caller
    // waits for is the upload, then the leading cells of the LAST slice, then the rest of the network: the last
    // slice is half as large as the others.
    int nslices = (net->head_cells > 0 && batch >= 256) ? (batch / 128 > 8 ? 8 : batch / 128) : 1;
    if (net->forced_slices > 0 && net->head_cells > 0) nslices = net->forced_slices;
    while (nslices > 1 && batch < 2 * nslices - 1) --nslices;   // every slice holds at least one image
    const int wsum = 2 * nslices - 1;   // weights 2, 2, ..., 2, 1
    if (nslices == 1) {
        CUDA_TRY(cudaMemcpyAsync(d_in, h_input, in_bytes, cudaMemcpyHostToDevice, s));
        if (int rc = forward_impl(net, d_in, batch, d_out, s, nullptr, 0)) return rc;
    } else {
        // the staging buffer may still be read by work queued on `s` by an earlier call
        CUDA_TRY(cudaEventRecord(net->stage_free, s));
        CUDA_TRY(cudaStreamWaitEvent(net->copy_stream, net->stage_free, 0));
        const size_t img_bytes = net->tensors[0].bytes_per_image();
        net->call_batch = batch;
        net->call_widened = false;
        for (int k = 0; k < nslices; ++k) {
            const int b0 = (int)((long long)batch * (2 * k) / wsum);
            const int b1 = k + 1 == nslices ? batch : (int)((long long)batch * (2 * k + 2) / wsum);
            if (b1 <= b0) continue;
            CUDA_TRY(cudaMemcpyAsync((uint8_t*)d_in + (size_t)b0 * img_bytes, (const uint8_t*)h_input + (size_t)b0 * img_bytes,
                                     (size_t)(b1 - b0) * img_bytes, cudaMemcpyHostToDevice, net->copy_stream));
            CUDA_TRY(cudaEventRecord(net->slice_ready[k], net->copy_stream));
            CUDA_TRY(cudaStreamWaitEvent(s, net->slice_ready[k], 0));
            for (int ci = 0; ci < net->head_cells; ++ci)
                if (!net->cells[ci].skipped)
                    if (int rc = run_cell(net, net->cells[ci], d_in, b1 - b0, s, b0)) return rc;
        }
        if (int rc = forward_impl(net, d_in, batch, d_out, s, nullptr, 0, net->head_cells)) return rc;
    }
    CUDA_TRY(cudaMemcpyAsync(h_output, d_out, out_bytes, cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaStreamSynchronize(s));
    return check_status(net);
}

// Streaming form of the host-buffer entry point.  The reference overlaps the preparation of the next batch with
// the inference of the current one on a second host thread (src/utils/Helper.cpp:428-454); here the overlap is on
// the device: the upload of batch k + 1 runs on the copy stream, into the second staging buffer, under the
// forward pass of batch k.
int n2d2b_net_submit_host(n2d2b_net* net, const void* h_input, int batch, void* h_output, n2d2b_stream stream)
{
    if (int rc = host_call_checks(net, h_input, batch, h_output)) return rc;
    if (batch == 0) return 0;
    CUDA_TRY(cudaSetDevice(net->device));
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned slot = net->pipe_next & 1u;
    const size_t in_cap = net->tensors[0].bytes_per_image() * (size_t)net->max_batch + 256;
    const int ft = final_tensor_of(net);
    const size_t out_cap = net->tensors[ft].bytes_per_image() * (size_t)net->max_batch + 256;
    if (!net->d_pipe_in[slot]) {
        // the staging sets of this entry point are allocated on first use (callers of the blocking form never pay for them)
        CUDA_TRY(cudaMalloc(&net->d_pipe_in[slot], in_cap));
        CUDA_TRY(cudaMalloc(&net->d_pipe_out[slot], out_cap));
    }
    // the slot's previous batch (two submissions ago) must have left its staging buffers: its forward pass has
    // read the input (the upload waits for that) and its download has read the output (the forward pass, which
    // writes the output buffer last, waits for that)
    if (net->pipe_busy[slot]) {
        CUDA_TRY(cudaStreamWaitEvent(net->copy_stream, net->pipe_computed[slot], 0));
        CUDA_TRY(cudaStreamWaitEvent(s, net->pipe_done[slot], 0));
    }
    const size_t in_bytes = net->tensors[0].bytes_per_image() * (size_t)batch;
    const size_t out_bytes = net->tensors[ft].bytes_per_image() * (size_t)batch;
    CUDA_TRY(cudaMemcpyAsync(net->d_pipe_in[slot], h_input, in_bytes, cudaMemcpyHostToDevice, net->copy_stream));
    CUDA_TRY(cudaEventRecord(net->pipe_uploaded[slot], net->copy_stream));
    CUDA_TRY(cudaStreamWaitEvent(s, net->pipe_uploaded[slot], 0));
    if (int rc = forward_impl(net, net->d_pipe_in[slot], batch, net->d_pipe_out[slot], s, nullptr, 0)) return rc;
    // the download leaves on a stream of its own, so that `s` holds nothing but forward passes back to back
    CUDA_TRY(cudaEventRecord(net->pipe_computed[slot], s));
    CUDA_TRY(cudaStreamWaitEvent(net->download_stream, net->pipe_computed[slot], 0));
    CUDA_TRY(cudaMemcpyAsync(h_output, net->d_pipe_out[slot], out_bytes, cudaMemcpyDeviceToHost, net->download_stream));
    CUDA_TRY(cudaEventRecord(net->pipe_done[slot], net->download_stream));
    net->pipe_busy[slot] = true;
    net->pipe_stream[slot] = s;
    net->pipe_next++;
    return 0;
}

int n2d2b_net_wait(n2d2b_net* net)
{
    if (!net) return fail(N2D2B_ERR_INVALID, "net must not be NULL");
    if (!net->finalized) return fail(N2D2B_ERR_STATE, "wait before finalize");
    CUDA_TRY(cudaSetDevice(net->device));
    for (int k = 0; k < 2; ++k)
        if (net->pipe_busy[k]) {
            CUDA_TRY(cudaEventSynchronize(net->pipe_done[k]));
            net->pipe_busy[k] = false;
        }
    return check_status(net);
}

int n2d2b_net_estimated_labels(n2d2b_net* net, int batch, int32_t* d_labels, int32_t* d_values, n2d2b_stream stream)
{
    if (!net || !d_labels) return fail(N2D2B_ERR_INVALID, "net and d_labels must not be NULL");
    if (!net->finalized) return fail(N2D2B_ERR_STATE, "estimated labels before finalize");
    if (!net->last_input) return fail(N2D2B_ERR_STATE, "estimated labels before a forward pass");
    if (batch < 0 || batch > net->max_batch) return fail(N2D2B_ERR_TOO_LARGE, "batch out of range");
    CUDA_TRY(cudaSetDevice(net->device));
    const int ft = final_tensor_of(net);
    const TensorRec& t = net->tensors[ft];
    CUDA_TRY(launch_argmax(tensor_ptr(net, ft, net->last_input), t.dtype, t.is_unsigned, (size_t)batch * t.H * t.W, t.C, d_labels,
                           d_values, (cudaStream_t)stream));
    return 0;
}

int n2d2b_net_estimated_labels_topn(n2d2b_net* net, int batch, int top_n, int32_t* d_labels, int32_t* d_values, n2d2b_stream stream)
{
    if (!net || !d_labels) return fail(N2D2B_ERR_INVALID, "net and d_labels must not be NULL");
    if (!net->finalized) return fail(N2D2B_ERR_STATE, "estimated labels before finalize");
    if (!net->last_input) return fail(N2D2B_ERR_STATE, "estimated labels before a forward pass");
    if (batch < 0 || batch > net->max_batch) return fail(N2D2B_ERR_TOO_LARGE, "batch out of range");
    const int ft = final_tensor_of(net);
    const TensorRec& t = net->tensors[ft];
    if (top_n < 1 || top_n > t.C) return fail(N2D2B_ERR_INVALID, "top_n must be in 1..%d (the number of classes)", t.C);
    if (t.C > 16384) return fail(N2D2B_ERR_TOO_LARGE, "top-N handles up to 16384 classes");
    CUDA_TRY(cudaSetDevice(net->device));
    const void* scores = tensor_ptr(net, ft, net->last_input);
    if (top_n == 1)   // the reference's top-1 branch: first maximum; the layouts coincide
        CUDA_TRY(launch_argmax(scores, t.dtype, t.is_unsigned, (size_t)batch * t.H * t.W, t.C, d_labels, d_values, (cudaStream_t)stream));
    else
        CUDA_TRY(launch_topn(scores, t.dtype, t.is_unsigned, (size_t)batch * t.H * t.W, (size_t)t.H * t.W, t.C, top_n, d_labels,
                             d_values, (cudaStream_t)stream));
    return 0;
}

int n2d2b_net_estimated_labels_topn_host(n2d2b_net* net, int batch, int top_n, int32_t* h_labels, int32_t* h_values)
{
    if (!net || !h_labels) return fail(N2D2B_ERR_INVALID, "net and h_labels must not be NULL");
    if (!net->finalized) return fail(N2D2B_ERR_STATE, "estimated labels before finalize");
    if (batch < 0 || batch > net->max_batch) return fail(N2D2B_ERR_TOO_LARGE, "batch out of range");
    const TensorRec& t = net->tensors[final_tensor_of(net)];
    if (top_n < 1 || top_n > t.C) return fail(N2D2B_ERR_INVALID, "top_n must be in 1..%d (the number of classes)", t.C);
    CUDA_TRY(cudaSetDevice(net->device));
    const size_t n = (size_t)batch * top_n * t.H * t.W;
    if (n == 0) return 0;
    if (net->labels_scratch_bytes < 2 * n * sizeof(int32_t)) {
        cudaFree(net->d_labels_scratch);
        net->d_labels_scratch = nullptr;
        net->labels_scratch_bytes = 0;
        CUDA_TRY(cudaMalloc(&net->d_labels_scratch, 2 * n * sizeof(int32_t)));
        net->labels_scratch_bytes = 2 * n * sizeof(int32_t);
    }
    int32_t* d_labels = (int32_t*)net->d_labels_scratch;
    int32_t* d_values = d_labels + n;
    // the legacy stream orders this after the forward pass on any blocking stream
    if (int rc = n2d2b_net_estimated_labels_topn(net, batch, top_n, d_labels, d_values, nullptr)) return rc;
    CUDA_TRY(cudaMemcpy(h_labels, d_labels, n * sizeof(int32_t), cudaMemcpyDeviceToHost));
    if (h_values) CUDA_TRY(cudaMemcpy(h_values, d_values, n * sizeof(int32_t), cudaMemcpyDeviceToHost));
    return 0;
}

int n2d2b_quantize_stimuli(int device, const float* d_in, int batch, int channels, int height, int width, int nb_bits,
                           int env_unsigned, void* d_out, n2d2b_stream stream)
{
    if (!d_in || !d_out) return fail(N2D2B_ERR_INVALID, "device buffers must not be NULL");
    if (batch < 0 || channels < 1 || height < 1 || width < 1) return fail(N2D2B_ERR_INVALID, "invalid stimuli dimensions");
    if (nb_bits < 2 || nb_bits > 8) return fail(N2D2B_ERR_INVALID, "nb_bits must be in 2..8 (the path carries 8-bit stimuli)");
    CUDA_TRY(cudaSetDevice(device));
    const int hi = env_unsigned ? (1 << nb_bits) - 1 : (1 << (nb_bits - 1)) - 1;
    const int lo = env_unsigned ? 0 : -(1 << (nb_bits - 1));
    CUDA_TRY(launch_quantize_stimuli(d_in, batch, channels, height, width, (float)hi, lo, hi, d_out, (cudaStream_t)stream));
    return 0;
}

int n2d2b_net_num_tensors(const n2d2b_net* net) { return net ? (int)net->tensors.size() : fail(N2D2B_ERR_INVALID, "net must not be NULL"); }

int n2d2b_net_tensor_info(const n2d2b_net* net, int id, n2d2b_tensor_info* info)
{
    if (!net || !info) return fail(N2D2B_ERR_INVALID, "net and info must not be NULL");
    if (id < 0 || id >= (int)net->tensors.size()) return fail(N2D2B_ERR_INVALID, "unknown tensor id %d", id);
    const TensorRec& t = net->tensors[id];
    info->channels = t.C; info->height = t.H; info->width = t.W;
    info->dtype = t.dtype; info->is_unsigned = t.is_unsigned; info->producer = t.producer;
    info->readable = (t.readable && (id == 0 || t.buffer >= 0 || !net->finalized)) ? 1 : 0;
    return 0;
}

int n2d2b_net_read_tensor(n2d2b_net* net, int id, int batch, void* host_dst, size_t bytes)
{
    if (!net || !host_dst) return fail(N2D2B_ERR_INVALID, "net and host_dst must not be NULL");
    if (!net->finalized) return fail(N2D2B_ERR_STATE, "read before finalize");
    if (id < 0 || id >= (int)net->tensors.size()) return fail(N2D2B_ERR_INVALID, "unknown tensor id %d", id);
    const TensorRec& t = net->tensors[id];
    if (batch < 0 || batch > net->max_batch) return fail(N2D2B_ERR_TOO_LARGE, "batch out of range");
    const size_t need = t.bytes_per_image() * (size_t)batch;
    if (bytes < need) return fail(N2D2B_ERR_INVALID, "destination holds %zu bytes, the tensor needs %zu", bytes, need);
    const void* src = tensor_ptr(net, id, net->last_input);
    if (!src || !t.readable) return fail(N2D2B_ERR_STATE, "tensor %d is not kept (finalize with N2D2B_KEEP_ALL_OUTPUTS)", id);
    CUDA_TRY(cudaSetDevice(net->device));
    CUDA_TRY(cudaDeviceSynchronize());
    CUDA_TRY(cudaMemcpy(host_dst, src, need, cudaMemcpyDeviceToHost));
    return check_status(net);
}

int n2d2b_net_weight_bytes(const n2d2b_net* net, size_t* total_bytes, size_t* packed4_bytes)
{
    if (!net || !net->finalized) return fail(N2D2B_ERR_STATE, "the network is not finalized");
    size_t total = 0, packed = 0;
    for (const CellRec& c : net->cells) {
        total += c.d_weight_bytes;
        if (c.engine == ENG_TCGEN05 && c.plan.w4) packed += c.d_weight_bytes;
    }
    if (net->d_small) total += net->small.blob.size();
    if (total_bytes) *total_bytes = total;
    if (packed4_bytes) *packed4_bytes = packed;
    return 0;
}

int n2d2b_net_launches_per_forward(const n2d2b_net* net)
{
    if (!net || !net->finalized) return fail(N2D2B_ERR_STATE, "the network is not finalized");
    return net->launches;
}

// (decided by the same rules as a forward pass of max_batch images)
const char* n2d2b_net_cell_engine(const n2d2b_net* net, int cell)
{
    if (!net || cell < 0 || cell >= (int)net->cells.size()) return "";
    if (net->d_small) return "small-net";
    const CellRec& c = net->cells[cell];
    if (c.dual_sum >= 0 && use_dual(net, net->cells[c.dual_sum], net->max_batch, net->max_batch)) return "fused";
    if (c.dual_branch >= 0 && use_dual(net, c, net->max_batch, net->max_batch)) return c.dual_patch.proj_in ? "patch-tcgen05-dual" : "tcgen05-dual";
    if (c.chain_prev >= 0) return "fused";
    if (c.chain_next >= 0) return "tcgen05-chain";
    if (use_dw3x3(c, net->max_batch)) return "depthwise";
    if (use_widened(net, c, net->max_batch, net->max_batch)) return c.w8 == CellRec::W8_PATCH ? "patch-tcgen05-widened" : "tcgen05-widened";
    switch (c.engine) {
    case ENG_TCGEN05: {
        const bool pair = c.plan.pair && c.fast.enabled && c.residual < 0
                          && net->tensors[c.output].dtype == DT_I8 && c.geom.O % 32 == 0;
        if (c.geom.groups > 1) return "depthwise-tcgen05";
        return pair ? "tcgen05-pair" : (c.plan.w4 ? "tcgen05-w4" : "tcgen05");
    }
    case ENG_SIMT: return "simt";
    case ENG_DEPTHWISE: return "depthwise";
    case ENG_POOL: return "pool";
    case ENG_SUM: return "sum";
    case ENG_FUSED: return "fused";
    case ENG_STEM: return "stem-tcgen05";
    case ENG_STEM_S2D: return c.pool_fused ? "stem-pool-tcgen05" : "stem-tcgen05";
    case ENG_DWPW: return "depthwise-1x1-tcgen05";
    case ENG_PATCH:
        if (patch_as_gemm(net, c, net->max_batch)) return "tcgen05";
        return c.geom.groups > 1 ? "depthwise-tcgen05" : "patch-tcgen05";
    }
    return "";
}

int n2d2b_scaling_propagate(int device, const int32_t* d_in, void* d_out, size_t nb_pixels, const n2d2b_quant* quant,
                            n2d2b_stream stream)
{
    if (!quant) return fail(N2D2B_ERR_INVALID, "quant must not be NULL");
    if (!d_in || !d_out) return fail(N2D2B_ERR_INVALID, "device buffers must not be NULL");
    if (quant->scaling.mode == SC_NONE) return fail(N2D2B_ERR_INVALID, "a NONE scaling has nothing to do");
    if (quant->scaling.nb_channels < 0) return fail(N2D2B_ERR_INVALID, "nb_channels must not be negative (got %d)", quant->scaling.nb_channels);
    CUDA_TRY(cudaSetDevice(device));
    QuantHost q;
    if (int rc = validate_quant(quant, quant->scaling.nb_channels, false, q, nullptr)) return rc;
    // the 32-bit or floating-point form where it is proved exact for every 32-bit input, the 64-bit one otherwise
    std::vector<int32_t> words;
    const int proved = build_rescale(q, q.nb_channels, (1ll << 31) - 1, words);
    const int form = proved == 0 ? 0 : (proved == EF_FLOAT ? 1 : 2);
    if (form == 2) words = exact_words(q);
    QuantDev scalars{};
    fill_quant_scalars(q, scalars);
    cudaError_t e = launch_rescale_i32(d_in, d_out, nb_pixels, q.nb_channels, form, words.data(), scalars, (cudaStream_t)stream);
    cudaError_t e2 = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) return fail(N2D2B_ERR_CUDA, "scaling kernel launch failed: %s", cudaGetErrorString(e));
    if (e2 != cudaSuccess) return fail(N2D2B_ERR_CUDA, "scaling kernel failed: %s", cudaGetErrorString(e2));
    return 0;
}

}  // extern "C"
