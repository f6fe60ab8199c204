// Softmax, LogSoftmax, L2Normalization and ArgMinMax: independent rows along one axis of a quantised (or fp32) tensor.
//
// The denominator of a Softmax is summed in the row's index order, because CpuRef's fp32 sum is sequential
// (Softmax.cpp:40-46 of the Arm NN tree) and a tree reduction would round differently.  A row is therefore one dependent
// chain of additions, and the kernels differ in how they keep the rest of the machine busy meanwhile:
//   * softmax_kernel: one CTA per row, for few or long rows and every type and mode.  All threads compute the
//     exponentials into shared memory, one thread adds them up (128-bit reads, so that the chain itself, about four
//     cycles per element, is what it costs), all threads divide and re-quantise.
//   * softmax_rows_kernel: many 8-bit rows, four per warp, one LANE per row running the chains.
#include "common.cuh"

namespace b200k {

struct SoftmaxArgs { QView x, y; int outer, axis, inner; float beta; };

constexpr int SM_THREADS = 256;
constexpr int SM_MAX_AXIS = (48 * 1024 - 64) / 4;        // dynamic floats + the static words below stay within 48 KiB

enum { ROW_SOFTMAX = 0, ROW_LOG_SOFTMAX = 1, ROW_L2_NORM = 2 };

// v[0] + v[1] + ... + v[n - 1] in that order.  v: 16-byte aligned shared memory, CHAIN_SLACK floats longer than n: the
// reads run one block of sixteen ahead of the additions, unconditionally, into values that are never added.
constexpr int CHAIN_SLACK = 48;
__device__ __forceinline__ float chain_sum(const float* v, int n)
{
    float sum = 0.0f;
    const float4* q = (const float4*)v;
    auto add16 = [&](const float4* b) {
        #pragma unroll
        for (int j = 0; j < 4; ++j) {
            sum = __fadd_rn(sum, b[j].x); sum = __fadd_rn(sum, b[j].y); sum = __fadd_rn(sum, b[j].z); sum = __fadd_rn(sum, b[j].w);
        }
    };
    float4 b[4], c[4];
    #pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = q[j];
    int i = 0;
    #pragma unroll 1
    for (; i + 32 <= n; i += 32, q += 8) {
        #pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = q[4 + j];
        add16(b);
        #pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = q[8 + j];
        add16(c);
    }
    if (i + 16 <= n) { add16(b); i += 16; }
    #pragma unroll 1
    for (; i < n; ++i) sum = __fadd_rn(sum, v[i]);
    return sum;
}

// MODE ROW_SOFTMAX / ROW_LOG_SOFTMAX: beta as in the descriptor.  ROW_L2_NORM: beta is eps; the parked values are the
// squares, summed in index order like the reference's `reduction += value * value`
// (RefL2NormalizationWorkload.cpp:73-80), and every element is multiplied by 1 / sqrt(max(sum, eps)).
template <int MODE>
__global__ void __launch_bounds__(SM_THREADS) softmax_kernel(const SoftmaxArgs a)
{
    pdl_enter();
    extern __shared__ __align__(16) float ex[];            // [axis + CHAIN_SLACK]
    __shared__ float red[SM_THREADS / 32];
    __shared__ float s_sum;
    const int row = blockIdx.x;
    const int o = row / a.inner, in = row - o * a.inner;
    const long long base = (long long)o * a.axis * a.inner + in;
    const int tid = threadIdx.x;

    // the row's values are parked in shared memory on the first read
    float mx = 0.f;
    if (MODE != ROW_L2_NORM) {
        mx = -3.402823466e+38f;
        for (int i = tid; i < a.axis; i += SM_THREADS) {
            const float v = a.x.get(base + (long long)i * a.inner);
            ex[i] = v;
            mx = fmaxf(mx, v);
        }
        #pragma unroll
        for (int s = 16; s > 0; s >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, s));
        if ((tid & 31) == 0) red[tid >> 5] = mx;
        __syncthreads();
        mx = red[0];
        #pragma unroll
        for (int w = 1; w < SM_THREADS / 32; ++w) mx = fmaxf(mx, red[w]);
        for (int i = tid; i < a.axis; i += SM_THREADS) ex[i] = expf(__fmul_rn(__fsub_rn(ex[i], mx), a.beta));
    } else {
        for (int i = tid; i < a.axis; i += SM_THREADS) {
            const float v = a.x.get(base + (long long)i * a.inner);
            ex[i] = __fmul_rn(v, v);
        }
    }
    __syncthreads();
    if (tid == 0) s_sum = chain_sum(ex, a.axis);
    __syncthreads();
    const float sum = s_sum;
    if (MODE == ROW_SOFTMAX) {
        for (int i = tid; i < a.axis; i += SM_THREADS)
            a.y.set(base + (long long)i * a.inner, __fdiv_rn(ex[i], sum));
    } else if (MODE == ROW_LOG_SOFTMAX) {
        const float log_sum = logf(sum);
        for (int i = tid; i < a.axis; i += SM_THREADS) {
            const long long at = base + (long long)i * a.inner;
            a.y.set(at, __fsub_rn(__fmul_rn(__fsub_rn(a.x.get(at), mx), a.beta), log_sum));
        }
    } else {
        const float scale = __fdiv_rn(1.0f, __fsqrt_rn(sum < a.beta ? a.beta : sum));
        for (int i = tid; i < a.axis; i += SM_THREADS) {
            const long long at = base + (long long)i * a.inner;
            a.y.set(at, __fmul_rn(a.x.get(at), scale));
        }
    }
}

// ---- many 8-bit rows (attention scores) -----------------------------------------------------------------------------
//
// Every warp keeps the bytes of its four rows in registers, finds each row's maximum on 16-bit pairs and writes the
// exponentials to shared memory; one warp of the block then runs all the block's chains, a row per lane (a pitch of 4 mod
// 32 words makes eight lanes' 128-bit reads one conflict-free wavefront), while the SM's other blocks compute; finally
// every warp divides and re-quantises its rows.
// The division and the re-quantisation are one multiplication by 1 / (sum * output scale) and a test that its error cannot matter
// (rows_sure); a value that fails it, one in 3500, takes the reference's divisions with its group of four, and so does its warp.
// Bound by instruction issue, about 16 per element, eight of them expf; a chain of 512 takes about 2300 cycles, while the SM's
// other blocks compute: with four warps a block six of them, and whatever phase one is in, others are in the other two.
// 32768 rows of 512: 101.9 us with one CTA and one summing thread per row; 28.7 with a margin of 1e-3 in the test (a group in a
// hundred, but one warp in three) and eight warps per block, 25.5 now (both alone, with cold caches).
constexpr int SMR_ROWS = 4, SMR_MAX_AXIS = 2048;             // rows per warp

struct RowsArgs {
    const uint8_t* x; uint8_t* y;
    uint32_t flip;                               // 0x80 for int8 input: bytes are compared and converted as byte + 128
    float off_x, sx, beta, sy, zy, tlo, thi, sure;
    int axis, pitch;
    long long rows;
};
// How far e / (s sy) + zy, evaluated as fma(e, 1 / (s sy), zy), may lie from an integer for the reference's value, two rounded
// divisions and a rounding, to be that integer.  With u = 2^-24 the product differs from the quotient by 2 u, the reference's
// by another 2 u, relative to a quotient of at most 257 + |zy| where the result does not saturate; the sum is rounded once more.
static float rows_sure(int zp)
{
    const double error = 1.1 * 5.9604645e-8 * (4.01 * (257.0 + fabs((double)zp)) + 257.0);
    return error < 0.25 ? (float)(0.5 - error) : -1.0f;      // (-1: nothing is sure)
}

// WPL: 4-byte words per lane and row (axis <= 128 WPL).  WORDS: rows are whole 4-byte words; otherwise every lane handles
// single bytes, 32 apart.
template <int WPL, bool WORDS, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) softmax_rows_kernel(const RowsArgs a)
{
    extern __shared__ __align__(16) float ex[];              // [block's rows][pitch] + CHAIN_SLACK
    constexpr int BATCH = WPL >= 16 ? 1 : (WPL >= 4 ? 16 / WPL : 4);    // rows whose bytes are in flight at once
    constexpr int BLOCK_ROWS = WARPS * SMR_ROWS;             // 32, 16 or 8
    __shared__ float s_sum[BLOCK_ROWS];
    pdl_enter();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long block0 = (long long)blockIdx.x * BLOCK_ROWS, row0 = block0 + warp * SMR_ROWS;
    const int rows = (int)max(0ll, min((long long)SMR_ROWS, a.rows - row0));
    float* mine = ex + warp * SMR_ROWS * a.pitch;
    const int words = a.axis >> 2;
    const f32x2 off2 = pack2(a.off_x, a.off_x), sx2 = pack2(a.sx, a.sx), beta2 = pack2(a.beta, a.beta), zero2 = pack2(0.f, 0.f);
    const uint32_t flip4 = a.flip * 0x01010101u;
    for (int r0 = 0; r0 < rows; r0 += BATCH) {
        uint32_t w[BATCH][WPL];
        #pragma unroll
        for (int b = 0; b < BATCH; ++b) {
            const uint8_t* x = a.x + (row0 + min(r0 + b, rows - 1)) * a.axis;
            #pragma unroll
            for (int k = 0; k < WPL; ++k) {
                if (WORDS) {
                    const int i = lane + 32 * k;
                    w[b][k] = i < words ? ((const uint32_t*)x)[i] ^ flip4 : 0u;
                } else {
                    w[b][k] = 0u;
                    #pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int i = lane + 32 * (4 * k + e);
                        if (i < a.axis) w[b][k] |= ((uint32_t)x[i] ^ a.flip) << (8 * e);
                    }
                }
            }
        }
        #pragma unroll
        for (int b = 0; b < BATCH; ++b) {
            if (r0 + b >= rows) break;
            uint32_t m2 = 0;                                 // maxima of the even and the odd bytes
            #pragma unroll
            for (int k = 0; k < WPL; ++k) m2 = __vmaxu2(m2, __vmaxu2(w[b][k] & 0x00ff00ffu, (w[b][k] >> 8) & 0x00ff00ffu));
            const uint32_t m = __reduce_max_sync(0xffffffffu, max(m2 & 0xffffu, m2 >> 16));
            // dequantisation is monotone: the largest byte has the largest value
            const float mx = __fmul_rn(__fsub_rn(__uint_as_float(0x4b000000u | m), a.off_x), a.sx);
            const f32x2 mx2 = pack2(mx, mx);
            float* e = mine + (r0 + b) * a.pitch;
            #pragma unroll
            for (int k = 0; k < WPL; ++k) {
                if (WORDS ? lane + 32 * k >= words : 128 * k >= a.axis) break;
                f32x2 q[2];
                float v[4];
                bytes_minus_zp(w[b][k], 0u, off2, q[0], q[1]);
                #pragma unroll
                for (int h = 0; h < 2; ++h) unpack2(mul2(sub2(fma2(q[h], sx2, zero2), mx2), beta2), v[h * 2], v[h * 2 + 1]);   // (value - maximum) * beta
                #pragma unroll
                for (int h = 0; h < 4; ++h) v[h] = expf(v[h]);
                if (WORDS) {
                    *(float4*)(e + (lane + 32 * k) * 4) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
                    #pragma unroll
                    for (int h = 0; h < 4; ++h)
                        if (lane + 32 * (4 * k + h) < a.axis) e[lane + 32 * (4 * k + h)] = v[h];
                }
            }
        }
    }
    __syncthreads();
    // (the chain warp changes from block to block, so that neighbours on an SM use different schedulers)
    if (warp == (int)(blockIdx.x % WARPS) && lane < BLOCK_ROWS && block0 + lane < a.rows) s_sum[lane] = chain_sum(ex + lane * a.pitch, a.axis);
    __syncthreads();
    auto exact = [&](float e, float s) -> float {            // the reference's chain
        return fminf(fmaxf(__fadd_rn(a.zy, roundf(__fdiv_rn(__fdiv_rn(e, s), a.sy))), a.tlo), a.thi);
    };
    const f32x2 magic2 = pack2(12582912.0f, 12582912.0f), zy2 = pack2(a.zy, a.zy);
    const bool s8 = a.tlo < 0.f;
    for (int r = 0; r < rows; ++r) {
        const float* e = mine + r * a.pitch;
        uint8_t* y = a.y + (row0 + r) * a.axis;
        const float s = s_sum[warp * SMR_ROWS + r], inv = __fdiv_rn(1.0f, __fmul_rn(s, a.sy));
        const f32x2 inv2 = pack2(inv, inv);
        if (WORDS) {
            #pragma unroll 4
            for (int i = lane; i < words; i += 32) {
                const float4 v = *(const float4*)(e + i * 4);
                const f32x2 q01 = fma2(pack2(v.x, v.y), inv2, zy2), q23 = fma2(pack2(v.z, v.w), inv2, zy2);
                const f32x2 z01 = sub2(add2(q01, magic2), magic2), z23 = sub2(add2(q23, magic2), magic2);
                float z[4], d[4];
                unpack2(z01, z[0], z[1]); unpack2(z23, z[2], z[3]);
                unpack2(sub2(q01, z01), d[0], d[1]); unpack2(sub2(q23, z23), d[2], d[3]);
                // (an exponential that overflowed, as with a negative beta, leaves NaN)
                if (!(max4_nan(fabsf(d[0]), fabsf(d[1]), fabsf(d[2]), fabsf(d[3])) < a.sure)) {
                    z[0] = exact(v.x, s); z[1] = exact(v.y, s); z[2] = exact(v.z, s); z[3] = exact(v.w, s);
                }
                ((uint32_t*)y)[i] = sat_pack4(z, s8);
            }
        } else {
            for (int i = lane; i < a.axis; i += 32) {
                const float q = __fmaf_rn(e[i], inv, a.zy), z = __fsub_rn(__fadd_rn(q, 12582912.0f), 12582912.0f);
                const bool fine = fabsf(__fsub_rn(q, z)) < a.sure;
                y[i] = (uint8_t)(int)(fine ? fminf(fmaxf(z, a.tlo), a.thi) : exact(e[i], s));
            }
        }
    }
}

struct ArgArgs { QView x; void* y; int outer, axis, inner, want_max, out64; long long rows; };

// One row per warp when the axis is contiguous (inner == 1: lanes stride the axis, then a shuffle reduction that keeps
// the lower index among equals), else one row per thread (neighbouring threads read neighbouring `inner` positions).
template <bool WARP>
__global__ void __launch_bounds__(256) arg_min_max_kernel(const ArgArgs a)
{
    pdl_enter();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long row = WARP ? t >> 5 : t;
    if (row >= a.rows) return;
    const int lane = WARP ? (int)(t & 31) : 0, step = WARP ? 32 : 1;
    const long long o = row / a.inner, in = row - o * a.inner;
    const long long base = o * a.axis * a.inner + in;
    // the reference starts from element 0 and replaces on a strict comparison: the first of equal elements wins
    float best = 0.f;
    int idx = 0x7fffffff;
    for (int i = lane; i < a.axis; i += step) {
        const float v = a.x.get(base + (long long)i * a.inner);
        if (idx == 0x7fffffff || (a.want_max ? v > best : v < best)) { best = v; idx = i; }
    }
    if (WARP) {
        #pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, s);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, s);
            const bool better = oi != 0x7fffffff && (idx == 0x7fffffff || (a.want_max ? ov > best : ov < best) || (ov == best && oi < idx));
            if (better) { best = ov; idx = oi; }
        }
        if (lane != 0) return;
    }
    if (a.out64) ((long long*)a.y)[row] = idx; else ((int*)a.y)[row] = idx;
}

// Short contiguous 8-bit rows (class scores per pixel): a block copies ARG_ROWS rows to shared memory in 128-bit pieces
// and every thread scans one of them there.  Dequantisation is monotone and keeps equal bytes equal, so the bytes
// themselves are compared.  (524288 rows of 21: 9.9 us with one thread
// per row straight from memory, 5.6 us now.)
constexpr int ARG_ROWS = 256;

__global__ void __launch_bounds__(ARG_ROWS) arg_min_max_bytes_kernel(const ArgArgs a)
{
    extern __shared__ __align__(16) uint8_t s_rows[];
    pdl_enter();
    const long long row0 = (long long)blockIdx.x * ARG_ROWS;
    const int rows = (int)min((long long)ARG_ROWS, a.rows - row0);
    const uint8_t* src = (const uint8_t*)a.x.data + row0 * a.axis;       // 16-byte aligned: ARG_ROWS is a multiple of 16
    const int bytes = rows * a.axis, v16 = bytes >> 4;
    for (int i = threadIdx.x; i < v16; i += ARG_ROWS) ((uint4*)s_rows)[i] = ((const uint4*)src)[i];
    for (int i = v16 * 16 + threadIdx.x; i < bytes; i += ARG_ROWS) s_rows[i] = src[i];
    __syncthreads();
    if ((int)threadIdx.x >= rows) return;
    const uint8_t* p = s_rows + threadIdx.x * a.axis;
    // order-preserving key: larger is better, whatever the type and the function
    const uint32_t flip = (a.x.dtype == B200K_S8 ? 0x80u : 0u) ^ (a.want_max ? 0u : 0xffu);
    uint32_t best = p[0] ^ flip;
    int idx = 0;
    #pragma unroll 4
    for (int i = 1; i < a.axis; ++i) {
        const uint32_t v = p[i] ^ flip;
        if (v > best) { best = v; idx = i; }
    }
    if (a.out64) ((long long*)a.y)[row0 + threadIdx.x] = idx; else ((int*)a.y)[row0 + threadIdx.x] = idx;
}

}  // namespace b200k

using namespace b200k;

static int launch_rows(const b200k_softmax_params* p, void* stream, int mode, const char* what)
{
    B200K_REQUIRE(p, B200K_E_INVALID, "%s: null params", what);
    B200K_REQUIRE(p->x.data && p->y.data, B200K_E_INVALID, "%s: null tensor pointer", what);
    B200K_REQUIRE(p->outer > 0 && p->axis_size > 0 && p->inner > 0, B200K_E_INVALID, "%s: bad shape", what);
    B200K_REQUIRE(p->x.dtype != B200K_S32 && p->y.dtype != B200K_S32, B200K_E_UNSUPPORTED, "%s: Signed32 not supported", what);
    // one float per element of the axis in dynamic shared memory, next to the kernel's few static words, within the
    // 48 KiB every launch may use without opting in
    B200K_REQUIRE(p->axis_size <= SM_MAX_AXIS, B200K_E_TOOBIG, "%s: axis length %d exceeds the %d this kernel stages in shared memory",
                  what, p->axis_size, SM_MAX_AXIS);
    SoftmaxArgs a;
    a.x = make_view(p->x); a.y = make_view(p->y);
    a.outer = p->outer; a.axis = p->axis_size; a.inner = p->inner; a.beta = p->beta;
    const long long rows = (long long)p->outer * p->inner;
    B200K_REQUIRE(rows < (1ll << 31), B200K_E_TOOBIG, "%s: too many rows", what);
    const size_t smem = ((size_t)p->axis_size + CHAIN_SLACK) * sizeof(float);
    cudaStream_t s = (cudaStream_t)stream;
    // From about one warp per scheduler on, four rows per warp; fewer or longer rows take a CTA each.
    if (mode == ROW_SOFTMAX && p->inner == 1 && rows >= 2048 && p->axis_size <= SMR_MAX_AXIS && is_q8(p->x.dtype) && is_q8(p->y.dtype) &&
        ordinary_quant(p->x) && ordinary_quant(p->y)) {
        RowsArgs r;
        r.x = (const uint8_t*)p->x.data; r.y = (uint8_t*)p->y.data;
        r.flip = p->x.dtype == B200K_S8 ? 0x80u : 0u;
        r.off_x = 8388608.0f + (float)(p->x.zero_point + (int)r.flip);
        r.sx = p->x.scale; r.beta = p->beta; r.sy = p->y.scale; r.zy = (float)p->y.zero_point;
        r.tlo = a.y.tlo; r.thi = a.y.thi;
        r.sure = rows_sure(p->y.zero_point);
        r.axis = p->axis_size; r.pitch = (p->axis_size + 27) / 32 * 32 + 4; r.rows = rows;
        const bool words = (p->axis_size & 3) == 0 && (((uintptr_t)p->x.data | (uintptr_t)p->y.data) & 3) == 0;
        auto go = [&](auto tag, int warps) -> int {
            const size_t bytes = ((size_t)warps * SMR_ROWS * r.pitch + CHAIN_SLACK) * sizeof(float);
            if (const int rc = allow_shared<decltype(tag)::kernel>(bytes)) return rc;
            launch_pdl(tag.kernel, dim3(div_up(rows, warps * SMR_ROWS)), dim3(32 * warps), bytes, s, r);
            return check_launch("softmax_rows_kernel");
        };
        // 66 KiB of exponentials per block at most: three blocks per SM
        if (words) {
            if (p->axis_size <= 128)  return go(KernelTag<softmax_rows_kernel<1, true, 8>>(), 8);
            // (rows of 512: 96.9 us for an attention layer with two warps per block, 96.5 with four, 99.1 with eight, 100.5 with one)
            if (p->axis_size <= 512)  return go(KernelTag<softmax_rows_kernel<4, true, 4>>(), 4);
            if (p->axis_size <= 1024) return go(KernelTag<softmax_rows_kernel<8, true, 4>>(), 4);
            return go(KernelTag<softmax_rows_kernel<16, true, 2>>(), 2);
        }
        if (p->axis_size <= 128)  return go(KernelTag<softmax_rows_kernel<1, false, 8>>(), 8);
        if (p->axis_size <= 512)  return go(KernelTag<softmax_rows_kernel<4, false, 8>>(), 8);
        if (p->axis_size <= 1024) return go(KernelTag<softmax_rows_kernel<8, false, 4>>(), 4);
        return go(KernelTag<softmax_rows_kernel<16, false, 2>>(), 2);
    }
    auto go = [&](auto tag) -> int {
        if (const int rc = allow_shared<decltype(tag)::kernel>(smem)) return rc;
        launch_pdl(tag.kernel, dim3((unsigned)rows), dim3(SM_THREADS), smem, s, a);
        return check_launch("softmax_kernel");
    };
    if (mode == ROW_SOFTMAX)     return go(KernelTag<softmax_kernel<ROW_SOFTMAX>>());
    if (mode == ROW_LOG_SOFTMAX) return go(KernelTag<softmax_kernel<ROW_LOG_SOFTMAX>>());
    return go(KernelTag<softmax_kernel<ROW_L2_NORM>>());
}

extern "C" int b200k_softmax_q8(const b200k_softmax_params* p, void* stream)
{
    return launch_rows(p, stream, ROW_SOFTMAX, "softmax_q8");
}

extern "C" int b200k_log_softmax_q(const b200k_softmax_params* p, void* stream)
{
    return launch_rows(p, stream, ROW_LOG_SOFTMAX, "log_softmax_q");
}

extern "C" int b200k_l2_normalization_q(const b200k_softmax_params* p, void* stream)
{
    return launch_rows(p, stream, ROW_L2_NORM, "l2_normalization_q");
}

extern "C" int b200k_arg_min_max_q(const b200k_arg_min_max_params* p, void* stream)
{
    B200K_REQUIRE(p, B200K_E_INVALID, "arg_min_max_q: null params");
    B200K_REQUIRE(p->x.data && p->y, B200K_E_INVALID, "arg_min_max_q: null tensor pointer");
    B200K_REQUIRE(p->outer > 0 && p->axis_size > 0 && p->inner > 0, B200K_E_INVALID, "arg_min_max_q: bad shape");
    B200K_REQUIRE(p->x.dtype == B200K_U8 || p->x.dtype == B200K_S8 || p->x.dtype == B200K_S16 || p->x.dtype == B200K_F32,
                  B200K_E_UNSUPPORTED, "arg_min_max_q: unsupported element type %d", p->x.dtype);
    B200K_REQUIRE(p->function == 0 || p->function == 1, B200K_E_INVALID, "arg_min_max_q: function %d is neither Min (0) nor Max (1)", p->function);
    ArgArgs a;
    a.x = make_view(p->x); a.y = p->y;
    a.outer = p->outer; a.axis = p->axis_size; a.inner = p->inner; a.want_max = p->function; a.out64 = p->out_int64 ? 1 : 0;
    a.rows = (long long)p->outer * p->inner;
    cudaStream_t s = (cudaStream_t)stream;
    if (p->inner == 1 && p->axis_size < 64 && is_q8(p->x.dtype) && p->x.scale > 0.f && ordinary_quant(p->x) && ((uintptr_t)p->x.data & 15) == 0 &&
        a.rows < (1ll << 38)) {
        launch_pdl(arg_min_max_bytes_kernel, dim3(div_up(a.rows, ARG_ROWS)), dim3(ARG_ROWS), (size_t)ARG_ROWS * p->axis_size, s, a);
        return check_launch("arg_min_max_bytes_kernel");
    }
    if (p->inner == 1 && p->axis_size >= 64) {
        B200K_REQUIRE(a.rows < (1ll << 34), B200K_E_TOOBIG, "arg_min_max_q: too many rows");
        launch_pdl(arg_min_max_kernel<true>, dim3((unsigned)div_up(a.rows * 32, 256)), dim3(256), 0, s, a);
    } else {
        B200K_REQUIRE(a.rows < (1ll << 38), B200K_E_TOOBIG, "arg_min_max_q: too many rows");
        launch_pdl(arg_min_max_kernel<false>, dim3((unsigned)div_up(a.rows, 256)), dim3(256), 0, s, a);
    }
    return check_launch("arg_min_max_kernel");
}
