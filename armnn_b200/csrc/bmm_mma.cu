// BatchMatMul on the tensor cores: out[b] = X[b] (M x K) * Y[b] (K x N), 8-bit operands, int32 accumulation, the fp32
// requantisation of the reference (src/backends/reference/workloads/BatchMatMulImpl.cpp:15-139 of the Arm NN tree).
//
// Both operands of a BatchMatMul are activations that arrive in whatever layout the graph has: [M, K] or (transpose_x)
// [K, M], [K, N] or (transpose_y) [N, K], with no load-time pass in which to re-pack them and no scratch memory in the
// entry point's contract.  The tensor-memory pipeline of the convolution kernel wants both operands K-contiguous; this
// kernel takes either layout as it is: a 128 x 128 tile per CTA, K in steps of 64 bytes, mma.sync m16n8k32 on int8.
//
// An operand that is K-contiguous in memory is staged as [row][k] (pitch 80 bytes) and a lane reads its fragment words
// directly.  An operand that is contiguous along M (or N) is staged as it lies, [k][m] (pitch 136 bytes): a lane reads
// the words that hold four consecutive m at four consecutive k and transposes the 4 x 4 bytes in registers, which gives
// it one fragment register for each of four m-tiles, provided the tiles' rows are assigned as row = 4 g + tile instead of
// 16 tile + g.  A matrix product does not care which rows an MMA tile holds as long as the epilogue writes each
// accumulator where its row belongs, so the assignment is simply different for that layout.  Both pitches make the
// fragment loads conflict-free.
//
// Three stages: the copies of the step after next are in flight during a step's MMAs (cp.async; operands at odd addresses
// go through registers instead).  Outputs are re-quantised two per instruction, gathered in shared memory and leave in
// 16-byte pieces of rows.  Attention scores and context (64 x 512 x 64 x 512 and 64 x 512 x 512 x 64) took 56.0 and 29.2 us
// with one stage, a byte store and a scalar requantisation per output; 17.7 and 14.6 us now.
//
// Zero points: sum (x - zx)(y - zy) = sum x y - zy sum_k x - zx sum_k y + K zx zy.  The row sums of X and column sums of
// Y come from dp4a on the fragments a lane holds anyway (a third of the registers of MMAs against ones, so that two CTAs
// share an SM), only for a non-zero zero point.
#include "common.cuh"

namespace b200k {

constexpr int BM_T = 128, BM_K = 64;                 // tile rows, K step in bytes; 128 or 64 columns
constexpr int BM_STAGES = 3;
constexpr int BM_PITCH_K = 80;                       // [row][k] staging: 20 words, rows g = 0..7 land on distinct banks

struct BmmTcArgs {
    const uint8_t* x; const uint8_t* y; uint8_t* out; int32_t* acc_out;
    int zx, zy, B, M, K, N;
    long long bsx, bsy;
    float m;                                         // sx * sy
    Quant4 quant;                                    // output quantisation
    int s8;                                          // output type
};

// w[j] = four consecutive rows' bytes at k + j  ->  o[i] = row i's bytes at k .. k + 3
__device__ __forceinline__ void bm_transpose4(const uint32_t* w, uint32_t* o)
{
    const uint32_t t0 = __byte_perm(w[0], w[1], 0x5140), t1 = __byte_perm(w[2], w[3], 0x5140);
    const uint32_t t2 = __byte_perm(w[0], w[1], 0x7362), t3 = __byte_perm(w[2], w[3], 0x7362);
    o[0] = __byte_perm(t0, t1, 0x5410); o[1] = __byte_perm(t0, t1, 0x7632);
    o[2] = __byte_perm(t2, t3, 0x5410); o[3] = __byte_perm(t2, t3, 0x7632);
}

// One operand's ROWS x 64 tile: KC: the operand is K-contiguous (element (r, k) at r * ld + k, ld = K); otherwise (k, r) at
// k * ld + r.  Pieces of 16 bytes along the contiguous index, NP per thread; zeros beyond the matrix.
template <bool KC, int ROWS, int THREADS>
struct BmOperand {
    static constexpr int PIECES = ROWS * BM_K / 16, NP = PIECES / THREADS;
    static constexpr int PER = KC ? BM_K / 16 : ROWS / 16;                     // pieces per row (per k)
    static constexpr int PITCH = KC ? BM_PITCH_K : ROWS + 8;                   // 136 (72): k rows 4 apart land 8 banks apart
    static constexpr int BYTES = (KC ? ROWS : BM_K) * PITCH;
    const uint8_t* base; int ld, r0, rows, K; bool vec;
    // the piece's address and how many of its bytes exist
    __device__ __forceinline__ const uint8_t* piece(int i, int k0, int& n) const
    {
        const int idx = threadIdx.x + i * THREADS, q = idx / PER, c = (idx % PER) * 16;
        const int slow = KC ? r0 + q : k0 + q, fast = KC ? k0 + c : r0 + c;
        n = slow < (KC ? rows : K) ? (KC ? K : rows) - fast : 0;
        return base + (long long)slow * ld + fast;
    }
    __device__ __forceinline__ uint8_t* place(uint8_t* s, int i) const
    {
        const int idx = threadIdx.x + i * THREADS;
        return s + (idx / PER) * PITCH + (idx % PER) * 16;                     // KC: 16-byte aligned, else 8
    }
    // copies in the background; operands at odd addresses and ragged ends through registers
    __device__ __forceinline__ void fetch(uint8_t* s, int k0) const
    {
        if (vec) {
            #pragma unroll
            for (int i = 0; i < NP; ++i) {
                int n;
                const uint8_t* p = piece(i, k0, n);
                const uint32_t d = (uint32_t)__cvta_generic_to_shared(place(s, i));
                // (16-byte aligned with a row length of whole pieces: a piece is whole or empty)
                const int whole = n > 0 ? 16 : 0;
                if (n <= 0) p = base;
                if (KC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(p), "r"(whole) : "memory");
                else {
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(p), "r"(whole >> 1) : "memory");
                    asm volatile("cp.async.ca.shared.global [%0 + 8], [%1 + 8], 8, %2;" ::"r"(d), "l"(p), "r"(whole >> 1) : "memory");
                }
            }
            return;
        }
        uint4 v[NP];
        #pragma unroll
        for (int i = 0; i < NP; ++i) {
            int n;
            const uint8_t* p = piece(i, k0, n);
            v[i] = load16_any(p, n);
        }
        #pragma unroll
        for (int i = 0; i < NP; ++i) {
            uint8_t* d = place(s, i);
            *(uint2*)d = make_uint2(v[i].x, v[i].y);
            *(uint2*)(d + 8) = make_uint2(v[i].z, v[i].w);
        }
    }
};

// TX / TY: the operand is stored transposed with respect to the K-contiguous form the MMA wants, i.e. X as [K, M]
// (transpose_x) and Y as [K, N] (no transpose_y).  WN: warps along N, 32 columns each (two along M, 64 rows each).
template <bool TX, bool TY, bool XU, bool YU, int WN>
__global__ void __launch_bounds__(64 * WN, WN == 4 ? 2 : 4) bmm_mma_kernel(const BmmTcArgs a)
{
    constexpr int THREADS = 64 * WN, BN = 32 * WN, OPITCH = BN + 16;
    typedef BmOperand<!TX, BM_T, THREADS> XOp;
    typedef BmOperand<!TY, BN, THREADS> YOp;
    constexpr int STAGE = (XOp::BYTES + YOp::BYTES + 15) & ~15;
    extern __shared__ uint4 bm_smem[];
    uint8_t* smem = (uint8_t*)bm_smem;
    pdl_enter();
    const int b = blockIdx.z, m0 = blockIdx.y * BM_T, n0 = blockIdx.x * BN;
    XOp xo; YOp yo;
    xo.base = a.x + (long long)b * a.bsx; xo.ld = TX ? a.M : a.K; xo.r0 = m0; xo.rows = a.M; xo.K = a.K;
    yo.base = a.y + (long long)b * a.bsy; yo.ld = TY ? a.N : a.K; yo.r0 = n0; yo.rows = a.N; yo.K = a.K;
    xo.vec = (((uintptr_t)xo.base | (uintptr_t)xo.ld) & 15) == 0;
    yo.vec = (((uintptr_t)yo.base | (uintptr_t)yo.ld) & 15) == 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int wm = warp / WN, wn = warp % WN;                // warp tile: rows wm * 64 .. + 64, columns wn * 32 .. + 32

    int acc[4][4][4];
    int rsum[4][2], csum[4];                                 // this lane's share of the sums of rows g, g + 8 and column g of a tile
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        rsum[i][0] = rsum[i][1] = csum[i] = 0;
        #pragma unroll
        for (int j = 0; j < 4; ++j)
            #pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0;
    }

    const int steps = (a.K + BM_K - 1) / BM_K;
    auto fetch = [&](int step) {
        uint8_t* s = smem + (step % BM_STAGES) * STAGE;
        if (step < steps) { xo.fetch(s, step * BM_K); yo.fetch(s + XOp::BYTES, step * BM_K); }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    #pragma unroll
    for (int i = 0; i < BM_STAGES - 1; ++i) fetch(i);
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(BM_STAGES - 2) : "memory");
        __syncthreads();                                     // this step's tile is there, and everyone has left the one before it
        fetch(step + BM_STAGES - 1);
        const uint8_t* s_a = smem + (step % BM_STAGES) * STAGE;
        const uint8_t* s_b = s_a + XOp::BYTES;
        #pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            uint32_t fa[4][4], fb[4][2];                     // [tile][register]
            if (!TX) {
                #pragma unroll
                for (int mi = 0; mi < 4; ++mi) {
                    const uint8_t* p = s_a + (wm * 64 + mi * 16 + g) * XOp::PITCH + ks * 32 + 4 * t;
                    fa[mi][0] = *(const uint32_t*)p;                       fa[mi][1] = *(const uint32_t*)(p + 8 * XOp::PITCH);
                    fa[mi][2] = *(const uint32_t*)(p + 16);                fa[mi][3] = *(const uint32_t*)(p + 8 * XOp::PITCH + 16);
                }
            } else {
                // rows of tile mi: 4 g + mi (fragment rows g) and 32 + 4 g + mi (fragment rows g + 8)
                #pragma unroll
                for (int half = 0; half < 2; ++half)
                    #pragma unroll
                    for (int kh = 0; kh < 2; ++kh) {
                        uint32_t w[4], o[4];
                        #pragma unroll
                        for (int j = 0; j < 4; ++j)
                            w[j] = *(const uint32_t*)(s_a + (ks * 32 + kh * 16 + 4 * t + j) * XOp::PITCH + wm * 64 + half * 32 + 4 * g);
                        bm_transpose4(w, o);
                        #pragma unroll
                        for (int mi = 0; mi < 4; ++mi) fa[mi][kh * 2 + half] = o[mi];
                    }
            }
            if (!TY) {
                #pragma unroll
                for (int ni = 0; ni < 4; ++ni) {
                    const uint8_t* p = s_b + (wn * 32 + ni * 8 + g) * YOp::PITCH + ks * 32 + 4 * t;
                    fb[ni][0] = *(const uint32_t*)p; fb[ni][1] = *(const uint32_t*)(p + 16);
                }
            } else {
                // columns of tile ni: 4 g + ni
                #pragma unroll
                for (int kh = 0; kh < 2; ++kh) {
                    uint32_t w[4], o[4];
                    #pragma unroll
                    for (int j = 0; j < 4; ++j)
                        w[j] = *(const uint32_t*)(s_b + (ks * 32 + kh * 16 + 4 * t + j) * YOp::PITCH + wn * 32 + 4 * g);
                    bm_transpose4(w, o);
                    #pragma unroll
                    for (int ni = 0; ni < 4; ++ni) fb[ni][kh] = o[ni];
                }
            }
            #pragma unroll
            for (int mi = 0; mi < 4; ++mi)
                #pragma unroll
                for (int ni = 0; ni < 4; ++ni)
                    mma_8bit<XU, YU>(acc[mi][ni], fa[mi][0], fa[mi][1], fa[mi][2], fa[mi][3], fb[ni][0], fb[ni][1]);
            if (a.zy != 0) {
                #pragma unroll
                for (int mi = 0; mi < 4; ++mi)
                    #pragma unroll
                    for (int q = 0; q < 4; ++q) rsum[mi][q & 1] = dp4a_mixed<XU, true>(fa[mi][q], 0x01010101u, rsum[mi][q & 1]);
            }
            if (a.zx != 0) {
                #pragma unroll
                for (int ni = 0; ni < 4; ++ni)
                    #pragma unroll
                    for (int q = 0; q < 2; ++q) csum[ni] = dp4a_mixed<YU, true>(fb[ni][q], 0x01010101u, csum[ni]);
            }
        }
    }
    // the four lanes of a quad hold parts of the same row (column)
    int cs[4][2];                                            // [n-tile][fragment column 2t, 2t + 1]
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        #pragma unroll
        for (int s = 1; s <= 2; s <<= 1) {
            rsum[i][0] += __shfl_xor_sync(0xffffffffu, rsum[i][0], s);
            rsum[i][1] += __shfl_xor_sync(0xffffffffu, rsum[i][1], s);
            csum[i] += __shfl_xor_sync(0xffffffffu, csum[i], s);
        }
        cs[i][0] = a.zx * __shfl_sync(0xffffffffu, csum[i], 8 * t);
        cs[i][1] = a.zx * __shfl_sync(0xffffffffu, csum[i], 8 * t + 4);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();                                         // the stages become the output tile, [128][BN] bytes

    const int kzz = a.K * a.zx * a.zy;
    const f32x2 m2 = pack2(a.m, a.m), zero2 = pack2(0.f, 0.f);
    #pragma unroll
    for (int mi = 0; mi < 4; ++mi)
        #pragma unroll
        for (int half = 0; half < 2; ++half) {               // fragment rows g and g + 8
            const int row = wm * 64 + (TX ? half * 32 + 4 * g + mi : mi * 16 + half * 8 + g);
            const int rs = kzz - a.zy * rsum[mi][half];
            int tot[4][2];                                   // [n-tile][fragment column 2t, 2t + 1]
            #pragma unroll
            for (int ni = 0; ni < 4; ++ni)
                #pragma unroll
                for (int e = 0; e < 2; ++e) tot[ni][e] = acc[mi][ni][half * 2 + e] + rs - cs[ni][e];
            if (a.acc_out && m0 + row < a.M) {
                #pragma unroll
                for (int ni = 0; ni < 4; ++ni)
                    #pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int n = n0 + wn * 32 + (TY ? 4 * (2 * t + e) + ni : ni * 8 + 2 * t + e);
                        if (n < a.N) a.acc_out[((long long)b * a.M + m0 + row) * a.N + n] = tot[ni][e];
                    }
            }
            auto requant = [&](int v0, int v1, int v2, int v3) -> uint32_t {
                float z[4];
                a.quant(fma2(pack2(__int2float_rn(v0), __int2float_rn(v1)), m2, zero2), fma2(pack2(__int2float_rn(v2), __int2float_rn(v3)), m2, zero2), z);
                return sat_pack4(z, a.s8 != 0);
            };
            uint8_t* o = smem + row * OPITCH + wn * 32;
            if (TY) {
                // fragment column c of the four tiles: output columns 4 c .. 4 c + 3
                *(uint2*)(o + 8 * t) = make_uint2(requant(tot[0][0], tot[1][0], tot[2][0], tot[3][0]), requant(tot[0][1], tot[1][1], tot[2][1], tot[3][1]));
            } else {
                #pragma unroll
                for (int ni = 0; ni < 4; ni += 2) {
                    const uint32_t w = requant(tot[ni][0], tot[ni][1], tot[ni + 1][0], tot[ni + 1][1]);
                    *(uint16_t*)(o + ni * 8 + 2 * t) = (uint16_t)w;
                    *(uint16_t*)(o + ni * 8 + 8 + 2 * t) = (uint16_t)(w >> 16);
                }
            }
        }
    __syncthreads();
    uint8_t* out = a.out + ((long long)b * a.M + m0) * a.N + n0;
    const int rows = min(BM_T, a.M - m0), cols = min(BN, a.N - n0);
    if ((a.N & 15) == 0 && ((uintptr_t)a.out & 15) == 0) {
        for (int i = threadIdx.x; i < BM_T * (BN / 16); i += THREADS) {
            const int r = i / (BN / 16), c = (i % (BN / 16)) * 16;
            if (r < rows && c < cols) *(uint4*)(out + (long long)r * a.N + c) = *(const uint4*)(smem + r * OPITCH + c);
        }
    } else if ((a.N & 3) == 0 && ((uintptr_t)a.out & 3) == 0) {
        for (int i = threadIdx.x; i < BM_T * (BN / 4); i += THREADS) {
            const int r = i / (BN / 4), c = (i % (BN / 4)) * 4;
            if (r < rows && c < cols) *(uint32_t*)(out + (long long)r * a.N + c) = *(const uint32_t*)(smem + r * OPITCH + c);
        }
    } else {
        for (int i = threadIdx.x; i < BM_T * BN; i += THREADS) {
            const int r = i / BN, c = i % BN;
            if (r < rows && c < cols) out[(long long)r * a.N + c] = smem[r * OPITCH + c];
        }
    }
}

bool bmm_mma_eligible(const b200k_bmm_params* p)
{
    if (!p->x.data || !p->y.data || !p->out.data) return false;
    if (!is_q8(p->x.dtype) || !is_q8(p->y.dtype) || !is_q8(p->out.dtype)) return false;
    if (p->batch < 1 || p->batch > 65535 || p->m < 1 || p->k < 1 || p->n < 1) return false;
    if ((p->m + BM_T - 1) / BM_T > 65535) return false;
    // (the accumulator is below 2^31 in magnitude)
    if (!quotient_holds(2147483648.0 * fabs((double)p->x.scale * (double)p->y.scale), p->out)) return false;
    // (the int32 accumulator of the reference and of the generic kernel has the same range)
    return true;
}

int launch_bmm_mma(const b200k_bmm_params* p, cudaStream_t stream)
{
    BmmTcArgs a;
    a.x = (const uint8_t*)p->x.data; a.y = (const uint8_t*)p->y.data; a.out = (uint8_t*)p->out.data; a.acc_out = p->acc_out;
    a.zx = p->x.zero_point; a.zy = p->y.zero_point;
    a.B = p->batch; a.M = p->m; a.K = p->k; a.N = p->n;
    a.bsx = p->batch_stride_x; a.bsy = p->batch_stride_y;
    // v = float(acc) * fl(sx * sy): the multiplier is formed once here with the same single rounding as on the device
    a.m = p->x.scale * p->y.scale;
    a.quant.sy = p->out.scale; a.quant.inv_sy = rn_reciprocal(p->out.scale); a.quant.zy = (float)p->out.zero_point;
    a.s8 = p->out.dtype == B200K_S8;
    const bool tx = p->transpose_x != 0, ty = p->transpose_y == 0;       // "transposed" = not K-contiguous
    const bool xu = p->x.dtype == B200K_U8, yu = p->y.dtype == B200K_U8;
    // 64 columns per tile where the matrix has no more
    const bool narrow = p->n <= 64;
    const int bn = narrow ? 64 : 128;
    const dim3 grid(div_up(p->n, bn), div_up(p->m, BM_T), (unsigned)p->batch);
    auto operand = [](bool kc, int rows) { return kc ? rows * BM_PITCH_K : BM_K * (rows + 8); };
    const size_t stages = (size_t)BM_STAGES * ((operand(!tx, BM_T) + operand(!ty, bn) + 15) & ~15), tile = (size_t)BM_T * (bn + 16);
    const size_t smem = stages > tile ? stages : tile;
    auto go = [&](auto tag) -> int {
        if (const int rc = allow_shared<decltype(tag)::kernel>(smem)) return rc;
        launch_pdl(tag.kernel, grid, dim3(narrow ? 128 : 256), smem, stream, a);
        return check_launch("bmm_mma_kernel");
    };
    #define B200K_BMM_WIDTH(TX, TY, XU, YU) (narrow ? go(KernelTag<bmm_mma_kernel<TX, TY, XU, YU, 2>>()) : go(KernelTag<bmm_mma_kernel<TX, TY, XU, YU, 4>>()))
    #define B200K_BMM_TYPES(TX, TY)                                                                                    \
        (xu ? (yu ? B200K_BMM_WIDTH(TX, TY, true, true) : B200K_BMM_WIDTH(TX, TY, true, false))                        \
            : (yu ? B200K_BMM_WIDTH(TX, TY, false, true) : B200K_BMM_WIDTH(TX, TY, false, false)))
    if (tx) return ty ? B200K_BMM_TYPES(true, true) : B200K_BMM_TYPES(true, false);
    return ty ? B200K_BMM_TYPES(false, true) : B200K_BMM_TYPES(false, false);
    #undef B200K_BMM_TYPES
    #undef B200K_BMM_WIDTH
}

}  // namespace b200k
