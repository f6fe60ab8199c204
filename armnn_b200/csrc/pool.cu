// Pooling2d (Max / Average / L2, both padding methods) and Mean over H,W for quantised NHWC tensors.
// Bandwidth-bound: each thread owns VEC consecutive channels of one output pixel, consecutive threads
// walk the channel axis, every tap is one coalesced vector load.  The arithmetic is CpuRef's own:
// dequantise to fp32, accumulate in CpuRef's (y, x) visiting order with unfused fp32 adds, divide,
// re-quantise — so the results equal CpuRef's bit for bit (Pooling2d.cpp:142-303, Reduce.cpp:68-173 of
// the Arm NN tree).
#include <type_traits>
#include "common.cuh"

namespace b200k {

struct PoolArgs {
    QView x, y;
    int N, H, W, C, OH, OW;
    int ph, pw, sh, sw, pt, pb, pl, pr;
    int type, exclude;
    long long total;
};

__device__ __forceinline__ bool clamp_range(int& s, int& e, int maxr)
{
    if (s < 0 || e > maxr) {
        s = min(max(s, 0), maxr);
        e = min(max(e, 0), maxr);
        return true;
    }
    return false;
}

// VEC consecutive elements as they lie in memory (8-bit types; VEC == 1: any type, dequantised at once)
template <int VEC> struct RawVec;
template <> struct RawVec<1>  { typedef float type; };
template <> struct RawVec<4>  { typedef unsigned type; };
template <> struct RawVec<16> { typedef uint4 type; };

template <int VEC>
__device__ __forceinline__ typename RawVec<VEC>::type load_raw(const QView& t, long long i)
{
    if constexpr (VEC == 1) return t.get(i);
    else return *(const typename RawVec<VEC>::type*)((const uint8_t*)t.data + i);
}

template <int VEC>
__device__ __forceinline__ void raw_to_f(const QView& t, const typename RawVec<VEC>::type& v, float* out)
{
    if constexpr (VEC == 1) {
        out[0] = v;
    } else {
        const uint8_t* raw = (const uint8_t*)&v;
        #pragma unroll
        for (int k = 0; k < VEC; ++k) {
            const int q = t.dtype == B200K_U8 ? (int)raw[k] : (int)(int8_t)raw[k];
            out[k] = dequantize_dev(q, t.scale, t.zp);
        }
    }
}

template <int VEC>
__device__ __forceinline__ void store_vec_f(const QView& t, long long i, const float* v)
{
    if (VEC == 1) { t.set(i, v[0]); return; }
    uint8_t raw[VEC];
    #pragma unroll
    for (int k = 0; k < VEC; ++k) raw[k] = (uint8_t)t.quant(v[k]);
    if (VEC == 16) *(uint4*)((uint8_t*)t.data + i) = *(const uint4*)raw;
    else           *(unsigned*)((uint8_t*)t.data + i) = *(const unsigned*)raw;
}

template <int VEC>
__global__ void __launch_bounds__(256) pool2d_kernel(const PoolArgs a)
{
    pdl_enter();
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= a.total) return;
    const int cg = a.C / VEC;
    const int c = (int)(idx % cg) * VEC;
    long long t = idx / cg;
    const int ox = (int)(t % a.OW); t /= a.OW;
    const int oy = (int)(t % a.OH);
    const int n = (int)(t / a.OH);

    int hstart = oy * a.sh - a.pt;
    int hend = min(hstart + a.ph, a.H + a.pb);
    const int height = hend - hstart;
    bool clamped = clamp_range(hstart, hend, a.H);
    int wstart = ox * a.sw - a.pl;
    int wend = min(wstart + a.pw, a.W + a.pr);
    float area = __int2float_rn(height * (wend - wstart));
    const long long oi = (((long long)n * a.OH + oy) * a.OW + ox) * a.C + c;

    float r[VEC];
    if ((hend <= 0 || hstart > a.H) || (wend <= 0 || wstart > a.W)) {
        // window lies entirely in the padding: 0 by convention (Pooling2d.cpp:216-241)
        #pragma unroll
        for (int k = 0; k < VEC; ++k) r[k] = 0.0f;
        store_vec_f<VEC>(a.y, oi, r);
        return;
    }
    clamped |= clamp_range(wstart, wend, a.W);
    if (clamped && a.exclude) area = __int2float_rn((hend - hstart) * (wend - wstart));

    #pragma unroll
    for (int k = 0; k < VEC; ++k) r[k] = a.type == 0 ? -3.402823466e+38f : 0.0f;
    // The taps in (y, x) order, BATCH of them loaded before the first is used: a window's sum is one dependent chain per
    // channel, and with one load per link the few threads of a global pooling layer wait for memory 49 times in a row
    // (7 x 7 x 1280, one image: 9.3 us).
    constexpr int BATCH = VEC == 16 ? 8 : 16;
    const int ww = wend - wstart, taps = ww > 0 && hend > hstart ? ww * (hend - hstart) : 0;
    long long at = (((long long)n * a.H + hstart) * a.W + wstart) * a.C + c;
    const long long row_skip = (long long)(a.W - ww) * a.C;
    int col = 0;
    for (int t0 = 0; t0 < taps; t0 += BATCH) {
        typename RawVec<VEC>::type raw[BATCH];
        #pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            if (t0 + j < taps) {
                raw[j] = load_raw<VEC>(a.x, at);
                at += a.C;
                if (++col == ww) { col = 0; at += row_skip; }
            }
        }
        #pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            if (t0 + j >= taps) break;
            float v[VEC];
            raw_to_f<VEC>(a.x, raw[j], v);
            #pragma unroll
            for (int k = 0; k < VEC; ++k) {
                if (a.type == 0)      { if (v[k] > r[k]) r[k] = v[k]; }
                else if (a.type == 1) r[k] = __fadd_rn(r[k], v[k]);
                else                  r[k] = __fadd_rn(r[k], __fmul_rn(v[k], v[k]));
            }
        }
    }
    #pragma unroll
    for (int k = 0; k < VEC; ++k) {
        if (a.type == 1)      r[k] = __fdiv_rn(r[k], area);
        else if (a.type == 2) r[k] = __fsqrt_rn(__fdiv_rn(r[k], area));
    }
    store_vec_f<VEC>(a.y, oi, r);
}

// Max pooling whose input and output share type, scale and offset: dequantisation is monotone and, for an ordinary scale,
// Quantize(Dequantize(q)) == q, so the result is the maximum of the quantised bytes themselves, no floating point.  A window with
// no valid tap yields Quantize(lowest float) = the type minimum, a padding-only window Quantize(0) = the zero point, as in the
// general kernel.
//
// Two 16-bit maxima take a word's odd bytes as they lie (the even byte below only breaks ties) and its even bytes shifted up:
// three instructions per four bytes, where a byte maximum is made of several.  A block of BH x BW taps is loaded before the first
// is compared; where the window ends inside a block its last tap repeats.  Bound by the loads' latency and by L2: ResNet-50's
// 112 x 112 x 64 at batch 256, 257 MB, took 84 us with byte maxima and a load per tap and trip, 68 now.
template <bool U8>
__device__ __forceinline__ uint32_t max16x2(uint32_t a, uint32_t b)
{
    uint32_t d;
    if (U8) asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    else    asm("max.s16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

template <bool U8, int BH, int BW>
__global__ void __launch_bounds__(256) maxpool_same_quant_kernel(const PoolArgs a)
{
    pdl_enter();
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= a.total) return;
    const int cg = a.C / 16;
    const int c = (int)(idx % cg) * 16;
    long long t = idx / cg;
    const int ox = (int)(t % a.OW); t /= a.OW;
    const int oy = (int)(t % a.OH);
    const int n = (int)(t / a.OH);
    int hstart = oy * a.sh - a.pt;
    int hend = min(hstart + a.ph, a.H + a.pb);
    clamp_range(hstart, hend, a.H);
    int wstart = ox * a.sw - a.pl;
    int wend = min(wstart + a.pw, a.W + a.pr);
    uint4 r;
    if ((hend <= 0 || hstart > a.H) || (wend <= 0 || wstart > a.W)) {
        const unsigned z = 0x01010101u * (unsigned)(a.x.zp & 0xff);
        r = make_uint4(z, z, z, z);
    } else {
        clamp_range(wstart, wend, a.W);
        const uint32_t lowest = U8 ? 0u : 0x80008000u;
        uint32_t odd[4], even[4];
        #pragma unroll
        for (int k = 0; k < 4; ++k) odd[k] = even[k] = lowest;
        const uint8_t* x = (const uint8_t*)a.x.data + (long long)n * a.H * a.W * a.C + c;
        for (int iy = hstart; iy < hend; iy += BH)
            for (int ix = wstart; ix < wend; ix += BW) {
                uint4 v[BH * BW];
                #pragma unroll
                for (int j = 0; j < BH * BW; ++j)
                    v[j] = *(const uint4*)(x + ((long long)min(iy + j / BW, hend - 1) * a.W + min(ix + j % BW, wend - 1)) * a.C);
                #pragma unroll
                for (int j = 0; j < BH * BW; ++j) {
                    const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
                    #pragma unroll
                    for (int k = 0; k < 4; ++k) { odd[k] = max16x2<U8>(odd[k], w[k]); even[k] = max16x2<U8>(even[k], w[k] << 8); }
                }
            }
        uint32_t o[4];
        #pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = (odd[k] & 0xff00ff00u) | ((even[k] >> 8) & 0x00ff00ffu);
        r = make_uint4(o[0], o[1], o[2], o[3]);
    }
    *(uint4*)((uint8_t*)a.y.data + (((long long)n * a.OH + oy) * a.OW + ox) * a.C + c) = r;
}

struct MeanArgs { QView x, y; int N, HW, C; };

// Mean over H x W.  The reference's sum is sequential, so a channel is one dependent chain of HW additions (784 of them
// at 28 x 28: 1.6 us), and there are few chains: what counts is that the chain never waits for memory.  A block owns 32
// lanes x VEC channels of one image; all its warps copy blocks of MEAN_ROWS pixels to shared memory, the next block's
// loads in flight during this block's sums, and the first warp adds them up.  (Float32 8 x 28 x 28 x 128: 20.4 us with
// one thread per channel group and a load per link, 7.9 us staged.)
constexpr int MEAN_ROWS = 128, MEAN_THREADS = 256;

template <int VEC>
__global__ void __launch_bounds__(MEAN_THREADS) mean_staged_kernel(const MeanArgs a)
{
    typedef typename RawVec<VEC>::type raw_t;                // one 32-bit word in both cases
    constexpr int PER = MEAN_ROWS * 32 / MEAN_THREADS;
    __shared__ raw_t s_v[2][MEAN_ROWS][32];
    pdl_enter();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = (blockIdx.x * 32 + lane) * VEC;
    const int n = blockIdx.y;
    const bool in = c < a.C;
    const long long base = (long long)n * a.HW * a.C + c;
    raw_t v[PER];
    auto load = [&](int p0) {
        #pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int p = p0 + warp + j * (MEAN_THREADS / 32);
            v[j] = in && p < a.HW ? load_raw<VEC>(a.x, base + (long long)p * a.C) : raw_t(0);
        }
    };
    float r[VEC];
    #pragma unroll
    for (int k = 0; k < VEC; ++k) r[k] = 0.0f;
    load(0);
    int buf = 0;
    for (int p0 = 0; p0 < a.HW; p0 += MEAN_ROWS, buf ^= 1) {
        #pragma unroll
        for (int j = 0; j < PER; ++j) s_v[buf][warp + j * (MEAN_THREADS / 32)][lane] = v[j];
        __syncthreads();             // (one barrier per block: the other buffer was read a whole block ago)
        if (p0 + MEAN_ROWS < a.HW) load(p0 + MEAN_ROWS);
        if (warp == 0) {
            const int rows = min(MEAN_ROWS, a.HW - p0);
            #pragma unroll 16
            for (int i = 0; i < rows; ++i) {
                float f[VEC];
                raw_to_f<VEC>(a.x, s_v[buf][i][lane], f);
                #pragma unroll
                for (int k = 0; k < VEC; ++k) r[k] = __fadd_rn(r[k], f[k]);
            }
        }
    }
    if (warp != 0 || !in) return;
    const float cnt = __int2float_rn(a.HW);
    #pragma unroll
    for (int k = 0; k < VEC; ++k) r[k] = __fdiv_rn(r[k], cnt);
    store_vec_f<VEC>(a.y, (long long)n * a.C + c, r);
}

// Taps per block along one axis of the window.  Blocks of three repeat taps in windows of one, two and four: with them for
// every window above 2 x 2, 64 x 56 x 56 x 128 took 39.5 us at 1 x 7 (26.3 with a load per tap and trip, 25.7 now), 17.8 at
// 1 x 4, stride 2 (11.6, 10.2), 15.0 at 4 x 4, stride 2 (14.5, 10.4), 13.4 at 3 x 2 (15.1, 11.2).  Longer ones gain from three: 7 x 7, stride 2
// 32.3 and 27.4, 9 x 9 162 and 82.
static int taps_per_block(int window) { return window == 1 ? 1 : (window == 2 || window == 4 ? 2 : 3); }

static int pick_vec(const b200k_qtensor& x, const b200k_qtensor& y, int C)
{
    if (!is_q8(x.dtype) || !is_q8(y.dtype)) return 1;
    const uintptr_t al = (uintptr_t)x.data | (uintptr_t)y.data;
    if ((C % 16) == 0 && (al & 15) == 0) return 16;
    if ((C % 4) == 0 && (al & 3) == 0) return 4;
    return 1;
}

}  // namespace b200k

using namespace b200k;

extern "C" int b200k_pool2d_q8(const b200k_pool2d_params* p, void* stream)
{
    B200K_REQUIRE(p, B200K_E_INVALID, "pool2d_q8: null params");
    B200K_REQUIRE(p->x.data && p->y.data, B200K_E_INVALID, "pool2d_q8: null tensor pointer");
    B200K_REQUIRE(p->pool_type >= 0 && p->pool_type <= 2, B200K_E_INVALID, "pool2d_q8: unsupported pooling algorithm %d", p->pool_type);
    B200K_REQUIRE(p->padding_method == 0 || p->padding_method == 1, B200K_E_INVALID, "pool2d_q8: unsupported padding type %d", p->padding_method);
    B200K_REQUIRE(p->n > 0 && p->h > 0 && p->wd > 0 && p->c > 0 && p->oh > 0 && p->ow > 0 && p->pool_h > 0 &&
                  p->pool_w > 0 && p->stride_h > 0 && p->stride_w > 0, B200K_E_INVALID, "pool2d_q8: bad geometry");
    B200K_REQUIRE(p->x.dtype != B200K_S32 && p->y.dtype != B200K_S32, B200K_E_UNSUPPORTED, "pool2d_q8: Signed32 not supported");
    PoolArgs a;
    a.x = make_view(p->x); a.y = make_view(p->y);
    a.N = p->n; a.H = p->h; a.W = p->wd; a.C = p->c; a.OH = p->oh; a.OW = p->ow;
    a.ph = p->pool_h; a.pw = p->pool_w; a.sh = p->stride_h; a.sw = p->stride_w;
    a.pt = p->pad_top; a.pb = p->pad_bottom; a.pl = p->pad_left; a.pr = p->pad_right;
    a.type = p->pool_type; a.exclude = p->padding_method == 1;
    int vec = pick_vec(p->x, p->y, p->c);
    // few outputs with large windows (global average pooling): narrower vectors give more threads to hide the latency
    // of the window's loads
    if (vec == 16 && (long long)p->n * p->oh * p->ow * (p->c / 16) < sm_count() * 1024ll) vec = 4;
    a.total = (long long)p->n * p->oh * p->ow * (p->c / vec);
    cudaStream_t s = (cudaStream_t)stream;
    int lo, hi;
    type_range(p->x.dtype, lo, hi);
    if (vec == 16 && p->pool_type == 0 && p->x.dtype == p->y.dtype && p->x.scale == p->y.scale &&
        p->x.zero_point == p->y.zero_point && ordinary_scale(p->x.scale) && p->x.zero_point >= lo && p->x.zero_point <= hi) {
        const bool u8 = p->x.dtype == B200K_U8;
        auto go = [&](auto kern) { launch_pdl(kern, dim3((unsigned)(div_up(a.total, 256))), dim3(256), 0, s, a); };
        auto width = [&](auto bh, auto bw) {
            constexpr int BH = decltype(bh)::value, BW = decltype(bw)::value;
            if (u8) go(maxpool_same_quant_kernel<true, BH, BW>); else go(maxpool_same_quant_kernel<false, BH, BW>);
        };
        auto height = [&](auto bh) {
            switch (taps_per_block(p->pool_w)) {
                case 1:  width(bh, std::integral_constant<int, 1>{}); break;
                case 2:  width(bh, std::integral_constant<int, 2>{}); break;
                default: width(bh, std::integral_constant<int, 3>{}); break;
            }
        };
        switch (taps_per_block(p->pool_h)) {
            case 1:  height(std::integral_constant<int, 1>{}); break;
            case 2:  height(std::integral_constant<int, 2>{}); break;
            default: height(std::integral_constant<int, 3>{}); break;
        }
        return check_launch("maxpool_same_quant_kernel");
    }
    if (vec == 16)     launch_pdl(pool2d_kernel<16>, dim3((unsigned)(div_up(a.total, 256))), dim3(256), 0, s, a);
    else if (vec == 4) launch_pdl(pool2d_kernel<4>, dim3((unsigned)(div_up(a.total, 256))), dim3(256), 0, s, a);
    else               launch_pdl(pool2d_kernel<1>, dim3((unsigned)(div_up(a.total, 256))), dim3(256), 0, s, a);
    return check_launch("pool2d_kernel");
}

extern "C" int b200k_mean_hw_q8(const b200k_mean_params* p, void* stream)
{
    B200K_REQUIRE(p, B200K_E_INVALID, "mean_hw_q8: null params");
    B200K_REQUIRE(p->x.data && p->y.data, B200K_E_INVALID, "mean_hw_q8: null tensor pointer");
    B200K_REQUIRE(p->n > 0 && p->h > 0 && p->wd > 0 && p->c > 0, B200K_E_INVALID, "mean_hw_q8: bad shape");
    B200K_REQUIRE(p->x.dtype != B200K_S32 && p->y.dtype != B200K_S32, B200K_E_UNSUPPORTED, "mean_hw_q8: Signed32 not supported");
    MeanArgs a;
    a.x = make_view(p->x); a.y = make_view(p->y);
    a.N = p->n; a.HW = p->h * p->wd; a.C = p->c;
    const bool by4 = pick_vec(p->x, p->y, p->c) >= 4;
    cudaStream_t s = (cudaStream_t)stream;
    // (images along the grid's second dimension: at most 65535 per launch)
    const size_t xw = (size_t)elem_size(p->x.dtype) * a.HW * p->c, yw = (size_t)elem_size(p->y.dtype) * p->c;
    for (int n0 = 0; n0 < p->n; n0 += 65535) {
        MeanArgs q = a;
        q.x.data = (const uint8_t*)a.x.data + n0 * xw;
        q.y.data = (const uint8_t*)a.y.data + n0 * yw;
        const unsigned images = (unsigned)(p->n - n0 < 65535 ? p->n - n0 : 65535);
        if (by4) launch_pdl(mean_staged_kernel<4>, dim3(div_up(p->c, 128), images), dim3(MEAN_THREADS), 0, s, q);
        else     launch_pdl(mean_staged_kernel<1>, dim3(div_up(p->c, 32), images), dim3(MEAN_THREADS), 0, s, q);
        const int rc = check_launch("mean_staged_kernel");
        if (rc) return rc;
    }
    return B200K_OK;
}
