// FullyConnected with [N, K] weights on mma.sync for the shapes that the tcgen05 and the weight-streaming kernels cannot take:
// N not a multiple of 16 (classifier heads), K or the rows' addresses not multiples of 16 bytes, any number of rows.
//
// A CTA computes 32 rows x 32 columns.  Tiles this small give a classifier head one CTA per SM, and their eight warps split K
// instead: the whole K extent (up to FM_KT at a time) of the 64 operand rows is copied to shared memory at once - one
// round trip to memory instead of one per K step - every warp multiplies each eighth 32-byte slice, and the partial sums meet
// in shared memory.  The weights do not depend on the kernel before this one, so their copies start before the wait for it.
// Up to a few hundred rows bound by that round trip and the reduction: 200 x 1280 x 1001 takes 6.4 us against 25.3 us with a
// warp per output column and dp4a, whose 32 CTA rows read every activation byte through the L1 once per eight columns.  Many
// rows are bound by the operands' traffic from L2 (each is read again for every 32 rows or columns of the other) and, above
// 1700 bytes of K per pass, by one CTA per SM whose copies and MMAs take turns: 4096 x 1280 x 1001 74 us, 4096 x 4096 x 1001
// 231 us (146 TOP/s), 4096 x 4099 x 4099 1351 us; the dp4a kernels take 446, 1102 and 6767 us.  No size measured from
// 5 to 4096 rows is slower than with them.
//
// Zero points as in the other kernels: sum (x - zx)(w - zw) = sum x w - zw sum x - zx sum w + K zx zw, the row and column
// sums from MMAs against ones.
#include "common.cuh"

namespace b200k {

constexpr int FM_T = 32;                         // tile edge
constexpr int FM_WARPS = 8, FM_THREADS = 32 * FM_WARPS;
constexpr int FM_KT = 2048;                      // bytes of K in shared memory at most
constexpr int FM_RED_PITCH = FM_T * FM_T + 4;    // partial sums of a warp, in words

struct FcMmaArgs {
    const uint8_t* x; const uint8_t* w; const int32_t* bias; uint8_t* y; int32_t* acc_out;
    const float* w_scales; const float* b_scales;
    float w_scale, b_scale;
    int zx, zw, M, K, N, kt;                     // kt: bytes of K per pass, a multiple of 32
    Requant rq;
    float inv_sy, lo, hi;
};

// bytes [k0, k0 + kt) of 32 rows of a [rows, K] matrix from row r0 on, zeros beyond it; VEC: whole aligned 16-byte pieces
template <bool VEC>
__device__ __forceinline__ void fm_copy(uint8_t* s, int pitch, const uint8_t* base, int r0, int rows, int k0, int kt, int K)
{
    const int pieces = kt >> 4;
    // eight lanes walk along a row, so that a warp's copies are four runs of 128 bytes
    for (int r = threadIdx.x >> 3; r < FM_T; r += FM_THREADS / 8) {
        const uint8_t* p = base + (long long)(r0 + r) * K + k0;
        uint8_t* d = s + r * pitch;
        for (int c = threadIdx.x & 7; c < pieces; c += 8) {
            const int n = r0 + r < rows ? K - k0 - c * 16 : 0;           // bytes of the row from here on
            if (VEC) {
                // (K is a multiple of 16: a piece is whole or empty)
                if (n > 0) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(d + c * 16)), "l"(p + c * 16) : "memory");
                else       *(uint4*)(d + c * 16) = make_uint4(0, 0, 0, 0);
            } else {
                *(uint4*)(d + c * 16) = load16_any(p + c * 16, n);
            }
        }
    }
}

template <bool XU, bool WU, bool VEC>
__global__ void __launch_bounds__(FM_THREADS) fc_mma_kernel(const FcMmaArgs a)
{
    extern __shared__ uint4 fm_smem[];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int pitch = ((a.kt + 127) & ~127) + 16;            // 16 mod 128: a fragment's eight rows fall on different banks
    uint8_t* s_w = (uint8_t*)fm_smem;
    uint8_t* s_x = s_w + FM_T * pitch;
    int* s_red = (int*)fm_smem;                              // [warps][FM_RED_PITCH], after the operands
    const int n0 = blockIdx.x * FM_T, m0 = blockIdx.y * FM_T;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    int acc[2][4][4], rsum[2][4], csum[4][4];
    #pragma unroll
    for (int i = 0; i < 2; ++i)
        #pragma unroll
        for (int j = 0; j < 4; ++j) {
            rsum[i][j] = 0; csum[j][i] = 0; csum[j][i + 2] = 0;
            #pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0;
        }
    for (int k0 = 0; k0 < a.K; k0 += a.kt) {
        if (k0 > 0) __syncthreads();
        fm_copy<VEC>(s_w, pitch, a.w, n0, a.N, k0, a.kt, a.K);
        if (k0 == 0) asm volatile("griddepcontrol.wait;" ::: "memory");      // the activations come from the kernel before this one
        fm_copy<VEC>(s_x, pitch, a.x, m0, a.M, k0, a.kt, a.K);
        if (VEC) asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        const int kend = min(a.kt, a.K - k0);
        for (int k = warp * 32; k < kend; k += 32 * FM_WARPS) {
            constexpr uint32_t ones = 0x01010101u;
            uint32_t fa[2][4], fb[4][2];
            #pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint8_t* p = s_x + (i * 16 + g) * pitch + k + 4 * t;
                fa[i][0] = *(const uint32_t*)p;        fa[i][1] = *(const uint32_t*)(p + 8 * pitch);
                fa[i][2] = *(const uint32_t*)(p + 16); fa[i][3] = *(const uint32_t*)(p + 8 * pitch + 16);
            }
            #pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint8_t* p = s_w + (j * 8 + g) * pitch + k + 4 * t;
                fb[j][0] = *(const uint32_t*)p; fb[j][1] = *(const uint32_t*)(p + 16);
            }
            #pragma unroll
            for (int i = 0; i < 2; ++i)
                #pragma unroll
                for (int j = 0; j < 4; ++j) mma_8bit<XU, WU>(acc[i][j], fa[i][0], fa[i][1], fa[i][2], fa[i][3], fb[j][0], fb[j][1]);
            if (a.zw != 0) {
                #pragma unroll
                for (int i = 0; i < 2; ++i) mma_8bit<XU, WU>(rsum[i], fa[i][0], fa[i][1], fa[i][2], fa[i][3], ones, ones);
            }
            if (a.zx != 0) {
                #pragma unroll
                for (int j = 0; j < 4; ++j) mma_8bit<XU, WU>(csum[j], ones, ones, ones, ones, fb[j][0], fb[j][1]);
            }
        }
    }
    __syncthreads();                                         // the operands have been read
    #pragma unroll
    for (int i = 0; i < 2; ++i)
        #pragma unroll
        for (int j = 0; j < 4; ++j)
            #pragma unroll
            for (int e = 0; e < 4; e += 2) {
                const int row = i * 16 + g + (e >> 1) * 8, col = j * 8 + 2 * t;
                const int s = a.zw * rsum[i][e];             // (c0 / c2 of a ones-MMA: the sum of fragment row g / g + 8)
                *(int2*)(s_red + warp * FM_RED_PITCH + row * FM_T + col) =
                    make_int2(acc[i][j][e] - s - a.zx * csum[j][0], acc[i][j][e + 1] - s - a.zx * csum[j][1]);
            }
    __syncthreads();
    // four neighbouring outputs per thread
    const int row = threadIdx.x >> 3, col = (threadIdx.x & 7) * 4, m = m0 + row;
    if (m >= a.M) return;
    int4 v = make_int4(0, 0, 0, 0);
    #pragma unroll
    for (int w = 0; w < FM_WARPS; ++w) {
        const int4 q = *(const int4*)(s_red + w * FM_RED_PITCH + row * FM_T + col);
        v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
    }
    const int kzz = a.K * a.zx * a.zw, total[4] = {v.x + kzz, v.y + kzz, v.z + kzz, v.w + kzz};
    #pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int n = n0 + col + e;
        if (n >= a.N) break;
        const float s = __fmul_rn(a.rq.sx, a.w_scales ? a.w_scales[n] : a.w_scale);
        const float b = a.bias ? __fmul_rn(__int2float_rn(a.bias[n]), a.b_scales ? a.b_scales[n] : a.b_scale) : 0.f;
        const long long o = (long long)m * a.N + n;
        if (a.acc_out) a.acc_out[o] = total[e];
        a.y[o] = (uint8_t)requant_fast(total[e], s, b, a.bias != nullptr, a.rq.sy, a.inv_sy, (float)a.rq.zy, a.lo, a.hi);
    }
}

bool fc_mma_eligible(const b200k_fc_params* p)
{
    if (!p->transpose_w || !p->x.data || !p->w.data || !p->y.data) return false;
    if (!is_q8(p->x.dtype) || !is_q8(p->w.dtype) || !is_q8(p->y.dtype)) return false;
    if (p->bias.data && p->bias.dtype != B200K_S32) return false;
    if (p->w.scales && p->w.zero_point != 0) return false;
    if (!ordinary_quant(p->y)) return false;
    return (p->m + FM_T - 1) / FM_T <= 65535;
}

int launch_fc_mma(const b200k_fc_params* p, cudaStream_t stream)
{
    FcMmaArgs a;
    a.x = (const uint8_t*)p->x.data; a.w = (const uint8_t*)p->w.data; a.bias = (const int32_t*)p->bias.data;
    a.y = (uint8_t*)p->y.data; a.acc_out = p->acc_out;
    a.w_scales = p->w.scales; a.b_scales = p->bias.scales; a.w_scale = p->w.scale; a.b_scale = p->bias.scale;
    a.zx = p->x.zero_point; a.zw = p->w.scales ? 0 : p->w.zero_point;
    a.M = p->m; a.K = p->k; a.N = p->n;
    a.rq = make_requant(p->x.scale, p->y, p->clamp_lo, p->clamp_hi);
    a.inv_sy = rn_reciprocal(p->y.scale);
    a.lo = fmaxf(a.rq.tlo, (float)a.rq.clo);
    a.hi = fminf(a.rq.thi, (float)a.rq.chi);
    // equal passes over K, each a multiple of 32 bytes
    const int passes = (p->k + FM_KT - 1) / FM_KT;
    a.kt = ((p->k + passes - 1) / passes + 31) & ~31;
    const size_t operands = 2 * FM_T * (size_t)(((a.kt + 127) & ~127) + 16), sums = FM_WARPS * FM_RED_PITCH * sizeof(int);
    const size_t smem = operands > sums ? operands : sums;
    const bool vec = p->k % 16 == 0 && (((uintptr_t)p->x.data | (uintptr_t)p->w.data) & 15) == 0;
    const dim3 grid(div_up(p->n, FM_T), div_up(p->m, FM_T), 1);
    auto go = [&](auto tag) -> int {
        if (const int rc = allow_shared<decltype(tag)::kernel>(smem)) return rc;
        launch_pdl(tag.kernel, grid, dim3(FM_THREADS), smem, stream, a);
        return check_launch("fc_mma_kernel");
    };
    const bool xu = p->x.dtype == B200K_U8, wu = p->w.dtype == B200K_U8;
    #define B200K_FC_MMA(XU, WU) (vec ? go(KernelTag<fc_mma_kernel<XU, WU, true>>()) : go(KernelTag<fc_mma_kernel<XU, WU, false>>()))
    if (xu) return wu ? B200K_FC_MMA(true, true) : B200K_FC_MMA(true, false);
    return wu ? B200K_FC_MMA(false, true) : B200K_FC_MMA(false, false);
    #undef B200K_FC_MMA
}

}  // namespace b200k
