// Resize (bilinear / nearest neighbour) of the H and W axes, the reference's arithmetic operation for operation
// (src/backends/reference/workloads/Resize.cpp:25-216): coordinates and weights in fp32, Lerp as two rounded products
// and a rounded sum, samples through Decoder / Encoder.  8-bit tensors take resize_rows_kernel; resize_kernel (one output
// element per thread) serves the other types.
#include "common.cuh"

namespace b200k {

struct ResizeArgs {
    QView x, y;
    int N, C, IH, IW, OH, OW;
    int method, align, half, nchw;
    float scale_y, scale_x;
    long long count;
};

// Lerp(a, b, w) = w * b + (1 - w) * a with every operation rounded (Resize.cpp:17-20)
__device__ __forceinline__ float lerp_ref(float a, float b, float w)
{
    return __fadd_rn(__fmul_rn(w, b), __fmul_rn(__fsub_rn(1.f, w), a));
}

// armnn::roundf (include/armnn/Utils.hpp:43-47)
__device__ __forceinline__ float round_ref(float v)
{
    return v < 0.f ? floorf(__fsub_rn(v, 0.5f)) : floorf(__fadd_rn(v, 0.5f));
}

// PixelScaler (Resize.cpp:36-56)
__device__ __forceinline__ float pixel_scaler(int pixel, float scale, bool half, int method)
{
    if (half && method == 0) return __fsub_rn(__fmul_rn(__fadd_rn((float)pixel, 0.5f), scale), 0.5f);
    if (half && method == 1) return __fmul_rn(__fadd_rn((float)pixel, 0.5f), scale);
    return __fmul_rn((float)pixel, scale);
}

__global__ void __launch_bounds__(256) resize_kernel(const ResizeArgs a)
{
    pdl_enter();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.count) return;
    int n, c, oy, ox;
    long long t = i;
    if (a.nchw) { ox = (int)(t % a.OW); t /= a.OW; oy = (int)(t % a.OH); t /= a.OH; c = (int)(t % a.C); n = (int)(t / a.C); }
    else        { c = (int)(t % a.C); t /= a.C; ox = (int)(t % a.OW); t /= a.OW; oy = (int)(t % a.OH); n = (int)(t / a.OH); }
    const bool half = a.half != 0, nn_round = a.method == 1 && a.align != 0;
    const float iy = pixel_scaler(oy, a.scale_y, half, a.method);
    const float fiy = nn_round ? round_ref(iy) : floorf(iy);
    int y0 = (int)fmaxf(fiy, 0.f);
    const float yw = __fsub_rn(iy, fiy);
    const float ix = pixel_scaler(ox, a.scale_x, half, a.method);
    const float fix = nn_round ? round_ref(ix) : floorf(ix);
    int x0 = (int)fmaxf(fix, 0.f);
    const float xw = __fsub_rn(ix, fix);
    // (the reference reads past the row for coordinates a rounded scale pushes to the input size; here they are clamped)
    y0 = min(y0, a.IH - 1); x0 = min(x0, a.IW - 1);
    int x1, y1;
    if (half) {
        x1 = min((int)fmaxf(ceilf(ix), 0.f), a.IW - 1);
        y1 = min((int)fmaxf(ceilf(iy), 0.f), a.IH - 1);
    } else {
        x1 = min(x0 + 1, a.IW - 1);
        y1 = min(y0 + 1, a.IH - 1);
    }
    auto at = [&](int yy, int xx) -> long long {
        return a.nchw ? (((long long)n * a.C + c) * a.IH + yy) * a.IW + xx : (((long long)n * a.IH + yy) * a.IW + xx) * a.C + c;
    };
    float v;
    if (a.method == 0) {
        const float ly0 = lerp_ref(a.x.get(at(y0, x0)), a.x.get(at(y0, x1)), xw);
        const float ly1 = lerp_ref(a.x.get(at(y1, x0)), a.x.get(at(y1, x1)), xw);
        v = lerp_ref(ly0, ly1, yw);
    } else {
        // the neighbour at distance 0 from (fix, fiy) is (x0, y0): the scaled coordinates are never negative
        v = a.x.get(at(y0, x0));
    }
    a.y.set(i, v);
}

// Where an output index samples the input along one axis, and with what weight.
struct AxisSample { int i0, i1; float w; };
__device__ __forceinline__ AxisSample axis_sample(int o, float scale, bool half, int method, bool align, int extent)
{
    AxisSample s;
    const float f = pixel_scaler(o, scale, half, method);
    const float fi = (method == 1 && align) ? round_ref(f) : floorf(f);
    s.w = __fsub_rn(f, fi);
    s.i0 = min((int)fmaxf(fi, 0.f), extent - 1);
    s.i1 = half ? min((int)fmaxf(ceilf(f), 0.f), extent - 1) : min(s.i0 + 1, extent - 1);
    return s;
}

// 8-bit tensors.  A thread owns four neighbouring bytes of the output row (pixel and channel run together in NHWC; NCHW
// is the same with one channel and N * C images) and walks RZ_ROWS output rows: its horizontal sample positions and
// weights are worked out once, and the two horizontally interpolated input rows are kept while the output rows stay
// between them, so an enlarged row costs the vertical interpolation and the requantisation only.  Instruction-bound:
// 8 x 64 x 64 x 21 -> 256 x 256 took 117 us with one element per thread (64-bit index divisions, coordinates and four
// samples for every element), 13.8 with a division and a coordinate per byte in the set-up and roundf for exact halves, about 11 now.
constexpr int RZ_ROWS = 16, RZ_THREADS = 128;

template <bool BILINEAR>
__global__ void __launch_bounds__(RZ_THREADS) resize_rows_kernel(const ResizeArgs a, const Quant4 quant)
{
    __shared__ AxisSample s_row[RZ_ROWS];
    pdl_enter();
    const int width = a.OW * a.C;                            // bytes of an output row (NCHW: C == 1 here)
    const int j0 = (blockIdx.x * RZ_THREADS + threadIdx.x) * 4;
    const int n = blockIdx.z, oy0 = blockIdx.y * RZ_ROWS, nrows = min(RZ_ROWS, a.OH - oy0);
    const bool half = a.half != 0, align = a.align != 0;
    if ((int)threadIdx.x < nrows) s_row[threadIdx.x] = axis_sample(oy0 + (int)threadIdx.x, a.scale_y, half, a.method, align, a.IH);
    __syncthreads();
    if (j0 >= width) return;
    const uint8_t* x = (const uint8_t*)a.x.data + (long long)n * a.IH * a.IW * a.C;
    uint8_t* y = (uint8_t*)a.y.data + ((long long)n * a.OH + oy0) * width + j0;
    int off0[4], off1[4];
    float xw[4];
    if (a.C >= 4) {                                          // four bytes of at most two neighbouring pixels
        const int ox = j0 / a.C, c0 = j0 - ox * a.C;
        const AxisSample s0 = axis_sample(ox, a.scale_x, half, a.method, align, a.IW), s1 = axis_sample(min(ox + 1, a.OW - 1), a.scale_x, half, a.method, align, a.IW);
        #pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool second = c0 + k >= a.C;
            const int c = second ? c0 + k - a.C : c0 + k;    // (bytes beyond the row: any of the row's samples)
            off0[k] = (second ? s1.i0 : s0.i0) * a.C + c; off1[k] = (second ? s1.i1 : s0.i1) * a.C + c;
            xw[k] = second ? s1.w : s0.w;
        }
    } else {
        #pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int j = min(j0 + k, width - 1), ox = j / a.C, c = j - ox * a.C;
            const AxisSample s = axis_sample(ox, a.scale_x, half, a.method, align, a.IW);
            off0[k] = s.i0 * a.C + c; off1[k] = s.i1 * a.C + c;
            xw[k] = s.w;
        }
    }
    // a byte as a float: 2^23 + byte (int8: + 128), minus 2^23 and the zero point (see bytes_minus_zp)
    const bool su = a.x.dtype == B200K_U8;
    const uint32_t expo = su ? 0x4b000000u : 0x4b000080u;
    const float zoff = 8388608.0f + (float)(a.x.zp + (su ? 0 : 128)), sx = a.x.scale;
    auto sample = [&](const uint8_t* row, int o) -> float { return __fmul_rn(__fsub_rn(__uint_as_float((uint32_t)row[o] ^ expo), zoff), sx); };
    f32x2 top[2], bot[2];
    const f32x2 zero2 = pack2(0.f, 0.f);
    auto line = [&](int iy, f32x2* out) {                    // the input row interpolated at this thread's columns
        const uint8_t* row = x + (long long)iy * a.IW * a.C;
        float v[4];
        #pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (BILINEAR) v[k] = __fadd_rn(__fmul_rn(xw[k], sample(row, off1[k])), __fmul_rn(__fsub_rn(1.f, xw[k]), sample(row, off0[k])));
            else          v[k] = sample(row, off0[k]);
        }
        out[0] = pack2(v[0], v[1]); out[1] = pack2(v[2], v[3]);
    };
    const bool word = ((width & 3) == 0) && (((uintptr_t)y & 3) == 0), s8 = a.y.dtype == B200K_S8;
    int top_y = -1, bot_y = -1;
    for (int r = 0; r < nrows; ++r, y += width) {
        const AxisSample s = s_row[r];
        f32x2 v[2];
        if (BILINEAR) {
            if (s.i0 != top_y) {
                if (s.i0 == bot_y) { top[0] = bot[0]; top[1] = bot[1]; }
                else line(s.i0, top);
                top_y = s.i0;
            }
            if (s.i1 != bot_y) {
                if (s.i1 == top_y) { bot[0] = top[0]; bot[1] = top[1]; }
                else line(s.i1, bot);
                bot_y = s.i1;
            }
            const float w1 = __fsub_rn(1.f, s.w);
            const f32x2 w2 = pack2(s.w, s.w), w12 = pack2(w1, w1);
            #pragma unroll
            for (int k = 0; k < 2; ++k) v[k] = add2(fma2(w2, bot[k], zero2), fma2(w12, top[k], zero2));
        } else {
            if (s.i0 != top_y) { line(s.i0, top); top_y = s.i0; }
            v[0] = top[0]; v[1] = top[1];
        }
        float z[4];
        quant(v[0], v[1], z);
        const uint32_t packed = sat_pack4(z, s8);
        if (word) *(uint32_t*)y = packed;
        else {
            #pragma unroll
            for (int k = 0; k < 4; ++k)
                if (j0 + k < width) y[k] = (uint8_t)(packed >> (8 * k));
        }
    }
}

}  // namespace b200k

using namespace b200k;

extern "C" int b200k_resize_q(const b200k_resize_params* p, void* stream)
{
    B200K_REQUIRE(p, B200K_E_INVALID, "resize_q: null params");
    B200K_REQUIRE(p->x.data && p->y.data, B200K_E_INVALID, "resize_q: null tensor pointer");
    B200K_REQUIRE(p->n > 0 && p->c > 0 && p->in_h > 0 && p->in_w > 0 && p->out_h > 0 && p->out_w > 0, B200K_E_INVALID,
                  "resize_q: bad geometry");
    B200K_REQUIRE(p->method == 0 || p->method == 1, B200K_E_INVALID, "resize_q: method %d is neither Bilinear (0) nor NearestNeighbor (1)", p->method);
    B200K_REQUIRE(!(p->align_corners && p->half_pixel_centers), B200K_E_INVALID,
                  "resize_q: align_corners and half_pixel_centers cannot both be set");
    B200K_REQUIRE(p->x.dtype != B200K_S32 && p->y.dtype != B200K_S32, B200K_E_UNSUPPORTED, "resize_q: Signed32 not supported");
    ResizeArgs a;
    a.x = make_view(p->x); a.y = make_view(p->y);
    a.N = p->n; a.C = p->c; a.IH = p->in_h; a.IW = p->in_w; a.OH = p->out_h; a.OW = p->out_w;
    a.method = p->method; a.align = p->align_corners; a.half = p->half_pixel_centers; a.nchw = p->nchw;
    // CalculateResizeScale (Resize.cpp:27-34), in fp32 like the reference
    a.scale_y = (p->align_corners && p->out_h > 1) ? (float)(p->in_h - 1) / (float)(p->out_h - 1) : (float)p->in_h / (float)p->out_h;
    a.scale_x = (p->align_corners && p->out_w > 1) ? (float)(p->in_w - 1) / (float)(p->out_w - 1) : (float)p->in_w / (float)p->out_w;
    a.count = (long long)p->n * p->c * p->out_h * p->out_w;
    // 8-bit tensors: rows of bytes; NCHW is N * C one-channel images
    const long long images = p->nchw ? (long long)p->n * p->c : p->n;
    const long long width = (long long)p->out_w * (p->nchw ? 1 : p->c), in_width = (long long)p->in_w * (p->nchw ? 1 : p->c);
    const unsigned row_blocks = div_up(p->out_h, RZ_ROWS);
    if (is_q8(p->x.dtype) && is_q8(p->y.dtype) && ordinary_quant(p->x) && quotient_holds(2.0 * value_bound(p->x), p->y) && images <= 65535 && row_blocks <= 65535 &&
        width < (1ll << 30) && in_width < (1ll << 30)) {
        ResizeArgs r = a;
        if (p->nchw) { r.N = (int)images; r.C = 1; r.nchw = 0; }
        const dim3 grid(div_up(div_up(width, 4), RZ_THREADS), row_blocks, (unsigned)images);
        Quant4 quant;
        quant.sy = p->y.scale; quant.inv_sy = rn_reciprocal(p->y.scale); quant.zy = (float)p->y.zero_point;
        if (p->method == 0) launch_pdl(resize_rows_kernel<true>, grid, dim3(RZ_THREADS), 0, (cudaStream_t)stream, r, quant);
        else                launch_pdl(resize_rows_kernel<false>, grid, dim3(RZ_THREADS), 0, (cudaStream_t)stream, r, quant);
        return check_launch("resize_rows_kernel");
    }
    launch_pdl(resize_kernel, dim3(div_up(a.count, 256)), dim3(256), 0, (cudaStream_t)stream, a);
    return check_launch("resize_kernel");
}
