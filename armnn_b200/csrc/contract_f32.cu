// Float32 Convolution2d, DepthwiseConvolution2d, FullyConnected and BatchMatMul: the reference's loops with the
// reference's rounding (src/backends/reference/workloads/ConvImpl.cpp:118-232, FullyConnected.cpp:32-62,
// BatchMatMulImpl.cpp:15-139) - a rounded product and a rounded sum per term, terms in the reference's order (input
// channel outermost, then filter row and column) - so that the results are CpuRef's bit for bit.
//
// The order only binds the terms of ONE output, so the contractions are register-tiled like any matrix product: a CTA
// computes BM output pixels (rows) x BN output channels (columns), and every accumulator walks the terms alone and in
// order.  No split over the terms and no tensor cores: either would round differently.
#include "common.cuh"

namespace b200k {

// ---- tiled contraction -------------------------------------------------------------------------------------------
//
// 128 threads, TM rows x TN columns of outputs each.  Terms arrive in chunks of CC channels x all T taps (T = 1 for the
// matrix products): both operands are gathered by 4-byte cp.async into [term][row] / [term][column] tiles, double-buffered.
// (REGS) where both operands are contiguous along the channel and 16-byte aligned, a thread loads four channels at a time
// of ITS row into registers while the chunk before is computed, and scatters them afterwards: 3 instructions per word
// against about 15 for a 4-byte copy.  The cp.async form serves odd channel counts, large filters and the other layouts: an
// operand that is contiguous along the channel has up to 8 lanes side by side on the channel axis (one 32-byte sector per
// row); with the pitches at 4 mod 32 words and an odd T the lanes of a copy fall on different banks.
//
// Two operations per term and no FMA, two terms per packed instruction: (a0, a1) x (b0, b1) and (a0, a1) x (b1, b0), so
// that only the swapped pairs have to be assembled.  A product that must be rounded before it is added is formed as
// fma2(a, b, 0) (see pack2 in common.cuh); the sign of a zero product, which that form loses, cannot change a sum that
// starts at +0.  The next term's operands are read while this one's are used.
//
// The floor is the fp32 pipes: two rounded operations per term are 64 terms per clock and SM, 26 us for the 462 M terms of
// 8 x 56 x 56 x 32 -> 64, 3 x 3 (1722 us with one output per thread).  The 4 x 8 outputs of a thread keep the shared-memory
// pipe at 12 of 16 cycles: 53 us (8 x 4 outputs and every B value stored twice filled both pipes: 75 us).
constexpr int F32_THREADS = 128;
constexpr int F32_MAX_TAPS = 64;                 // a row's in-image taps are a 64-bit mask
constexpr int F32_QUADS = 10;                    // REGS: (tap, channel quad) pairs of a chunk at most

struct F32Args {
    const float* x; const float* w; const float* bias; float* y;
    long long M; int N, C;                       // rows, columns, channels (terms = C * T)
    int T, KW, CC;                               // taps, filter width, channels per chunk (a power of two)
    int H, W, OH, OW, sh, sw, pt, pl, dh, dw;    // convolution geometry
    long long a_row, a_c;                        // matrix operand A: element (m, c) at m * a_row + c * a_c
    long long b_col, b_c, b_tap;                 // operand B: element (c, tap, n) at n * b_col + c * b_c + tap * b_tap
    long long bsa, bsb, bso;                     // batch strides (gridDim.z)
    int n_off;                                   // first column (more columns than one grid can hold: several launches)
};

// One word from global to shared memory in the background, or a zero at once (nothing is read then)
__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src, bool ok)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %2, 0;\n\t"
                 "@p cp.async.ca.shared.global [%0], [%1], 4;\n\t"
                 "@!p st.shared.b32 [%0], 0;\n\t}" ::"r"(dst), "l"(src), "r"((int)ok) : "memory");
}
__device__ __forceinline__ void lds_pairs(uint32_t addr, f32x2& a, f32x2& b)
{
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}

// CONV: A rows are output pixels of an NHWC tensor.  AKC / BKC: the operand is contiguous along the channel axis.  ONE: one tap
// (32 channels per chunk, four per copying lane).  REGS: the operands go through registers, 16 bytes at a time.
template <int TM, int TN, bool CONV, bool AKC, bool BKC, bool ONE, bool REGS>
__global__ void __launch_bounds__(F32_THREADS) contract_f32_kernel(const F32Args a)
{
    constexpr int BM = TN == 8 ? 64 : 32, BN = BM, RG = BM / TM, PA = BM + 4, PB = BN + 4;
    static_assert(RG * (BN / TN) == F32_THREADS, "one thread per TM x TN outputs");
    constexpr int NRA = BM * 8 / F32_THREADS, NRB = BN * 8 / F32_THREADS;       // rows of a thread with 8 channel lanes
    extern __shared__ float4 f32_smem[];
    __shared__ int s_toff[CONV ? F32_MAX_TAPS : 1];          // tap offsets in A, elements
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int t = threadIdx.x;
    const long long m0 = (long long)blockIdx.x * BM;
    const int n0 = a.n_off + blockIdx.y * BN;
    const float* x = a.x + blockIdx.z * a.bsa;
    const float* w = a.w + blockIdx.z * a.bsb;
    const int chunk_rows = a.CC * (ONE ? 1 : a.T);
    float* const sA = (float*)f32_smem;          // two buffers of A, then two of B
    float* const sB = sA + 2 * chunk_rows * PA;

    // A thread's share of the K-contiguous copies: channel lane cl, rows r0, r0 + step, ..., taps ph, ph + phs, ... (more
    // than one tap phase only where there are fewer rows than threads)
    constexpr int NB = ONE ? 4 : 1;
    const int T = ONE ? 1 : a.T, lanes_c = ONE ? 8 : a.CC;
    const int cl = t & (lanes_c - 1), rest = t / lanes_c, step = F32_THREADS / lanes_c;
    const int ra0 = rest % BM, pha = rest / BM, phsa = step > BM ? step / BM : 1;
    const int rb0 = rest % BN, phb = rest / BN, phsb = step > BN ? step / BN : 1;
    // where a row of A starts (its tap 0) and which of its taps lie inside the image
    auto locate = [&](int r, const float*& p, unsigned long long& mk) {
        const long long m = m0 + r;
        p = x;
        mk = 0;
        if (r >= BM || m >= a.M) return;
        if (!CONV) { p = x + m * a.a_row; mk = 1; return; }
        const long long q = m / a.OW;
        const int ox = (int)(m - q * a.OW);
        const int n = (int)(q / a.OH), oy = (int)(q - (long long)n * a.OH);
        const int iy = oy * a.sh - a.pt, ix = ox * a.sw - a.pl;
        p = x + (((long long)n * a.H + iy) * a.W + ix) * a.C;
        int ky = 0, kx = 0;
        for (int i = 0; i < a.T; ++i) {
            if ((unsigned)(iy + ky * a.dh) < (unsigned)a.H && (unsigned)(ix + kx * a.dw) < (unsigned)a.W) mk |= 1ull << i;
            if (++kx == a.KW) { kx = 0; ++ky; }
        }
    };
    const float* pA[AKC && !REGS ? NRA : 1];
    unsigned long long mask[AKC && !REGS ? NRA : 1], vmask = 0;
    const float* va = x;
    if (CONV) {
        for (int i = t; i < a.T; i += F32_THREADS) {
            const int ky = i / a.KW, kx = i - ky * a.KW;
            s_toff[i] = (ky * a.dh * a.W + kx * a.dw) * a.C;
        }
        __syncthreads();
    }
    if (REGS) locate(t % BM, va, vmask);
    else if (AKC) {
        #pragma unroll
        for (int j = 0; j < NRA; ++j) { locate(ra0 + j * step, pA[j], mask[j]); pA[j] += cl; }
    }
    // REGS: thread t serves row t mod BM (of A and of B) and every PHS-th of the chunk's (tap, channel quad) pairs
    constexpr int PHS = F32_THREADS / BM, SLOTS = REGS ? (F32_QUADS + PHS - 1) / PHS : 1;
    const int vr = t % BM, vph = t / BM, quads = REGS ? a.CC / 4 : 1, pairs = REGS ? T * quads : 0;
    float4 ra[SLOTS], rb[SLOTS];
    const float* vb = REGS ? w + (long long)min(n0 + vr, a.N - 1) * a.b_col : w;
    auto load_regs = [&](int c0) {
        #pragma unroll
        for (int i = 0; i < SLOTS; ++i) {
            const int q = vph + i * PHS;
            const int tap = ONE ? 0 : q / quads, c = (ONE ? q : q - tap * quads) * 4;
            const bool in = q < pairs && c0 + c < a.C;
            const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
            ra[i] = in && ((vmask >> tap) & 1) ? *(const float4*)(va + (CONV && !ONE ? s_toff[tap] : 0) + c0 + c) : none;
            rb[i] = in ? *(const float4*)(vb + (ONE ? 0 : tap * (int)a.b_tap) + c0 + c) : none;
        }
    };
    auto store_regs = [&](int buf) {
        #pragma unroll
        for (int i = 0; i < SLOTS; ++i) {
            const int q = vph + i * PHS;
            if (q >= pairs) break;
            const int tap = ONE ? 0 : q / quads, c = (ONE ? q : q - tap * quads) * 4;
            float* da = sA + buf * chunk_rows * PA + (c * T + tap) * PA + vr;
            float* db = sB + buf * chunk_rows * PB + (c * T + tap) * PB + vr;
            da[0] = ra[i].x; da[T * PA] = ra[i].y; da[2 * T * PA] = ra[i].z; da[3 * T * PA] = ra[i].w;
            db[0] = rb[i].x; db[T * PB] = rb[i].y; db[2 * T * PB] = rb[i].z; db[3 * T * PB] = rb[i].w;
        }
    };
    auto fetch = [&](int c0, int buf) {
        const uint32_t da = (uint32_t)__cvta_generic_to_shared(sA + buf * chunk_rows * PA), db = (uint32_t)__cvta_generic_to_shared(sB + buf * chunk_rows * PB);
        const bool c_in = c0 + cl < a.C;
        if (AKC) {
            #pragma unroll
            for (int j = 0; j < NRA; ++j) {
                const int r = ra0 + j * step;
                if (r >= BM) break;
                const float* p = pA[j] + c0;
                uint32_t d = da + (uint32_t)((cl * T + pha) * PA + r) * 4u;
                if (ONE) {
                    const bool in = (mask[j] & 1) != 0;
                    #pragma unroll
                    for (int b = 0; b < NB; ++b) cp_async4(d + (uint32_t)(8 * b * PA) * 4u, p + 8 * b, in && c0 + cl + 8 * b < a.C);
                } else {
                    const unsigned long long mk = c_in ? mask[j] : 0;
                    #pragma unroll 3
                    for (int tap = pha; tap < T; tap += phsa, d += (uint32_t)(phsa * PA) * 4u) cp_async4(d, p + s_toff[tap], (mk >> tap) & 1);
                }
            }
        } else {
            for (int i = t; i < a.CC * BM; i += F32_THREADS) {
                const int c = i / BM, r = i - c * BM;
                cp_async4(da + (uint32_t)(c * PA + r) * 4u, x + (m0 + r) * a.a_row + (c0 + c) * a.a_c, m0 + r < a.M && c0 + c < a.C);
            }
        }
        if (BKC) {
            #pragma unroll
            for (int j = 0; j < NRB; ++j) {
                const int r = rb0 + j * step;
                if (r >= BN) break;
                const bool in = n0 + r < a.N;
                const float* p = w + (long long)(n0 + r) * a.b_col + phb * a.b_tap + c0 + cl;
                uint32_t d = db + (uint32_t)((cl * T + phb) * PB + r) * 4u;
                if (ONE) {
                    #pragma unroll
                    for (int b = 0; b < NB; ++b) cp_async4(d + (uint32_t)(8 * b * PB) * 4u, p + 8 * b, in && c0 + cl + 8 * b < a.C);
                } else {
                    const bool ok = in && c_in;
                    #pragma unroll 3
                    for (int tap = phb; tap < T; tap += phsb, p += phsb * a.b_tap, d += (uint32_t)(phsb * PB) * 4u) cp_async4(d, p, ok);
                }
            }
        } else {
            for (int i = t; i < a.CC * BN; i += F32_THREADS) {
                const int c = i / BN, r = i - c * BN;
                cp_async4(db + (uint32_t)(c * PB + r) * 4u, w + (long long)(n0 + r) * a.b_col + (c0 + c) * a.b_c, n0 + r < a.N && c0 + c < a.C);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const int rg = t % RG, cg = t / RG;
    f32x2 acc[TM / 2][TN / 2][2];                // [row pair][column pair][straight, swapped]
    const f32x2 zero2 = pack2(0.f, 0.f);
    #pragma unroll
    for (int i = 0; i < TM / 2; ++i)
        #pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j][0] = acc[i][j][1] = zero2;
    auto operands = [&](uint32_t pa, uint32_t pb, f32x2* av, f32x2* bv) {
        lds_pairs(pa, av[0], av[1]);
        if (TN == 2) asm volatile("ld.shared.b64 %0, [%1];" : "=l"(bv[0]) : "r"(pb));
        #pragma unroll
        for (int h = 0; h < TN / 4; ++h) lds_pairs(pb + h * 16, bv[h * 2], bv[h * 2 + 1]);
    };

    if (REGS) load_regs(0);
    else fetch(0, 0);
    int buf = 0;
    for (int c0 = 0; c0 < a.C; c0 += a.CC, buf ^= 1) {
        const bool more = c0 + a.CC < a.C;
        if (REGS) {
            store_regs(buf);                     // (one barrier per chunk: everyone has left the chunk before last)
            __syncthreads();
            if (more) load_regs(c0 + a.CC);
        } else {
            if (more) {
                fetch(c0 + a.CC, buf ^ 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
        }
        uint32_t pa = (uint32_t)__cvta_generic_to_shared(sA + buf * chunk_rows * PA + rg * TM);
        uint32_t pb = (uint32_t)__cvta_generic_to_shared(sB + buf * chunk_rows * PB + cg * TN);
        const int rows = min(a.CC, a.C - c0) * T;
        f32x2 av[2][TM / 2], bv[2][TN / 2];
        operands(pa, pb, av[0], bv[0]);
        auto term = [&](int cur) {
            pa += PA * 4; pb += PB * 4;
            operands(pa, pb, av[cur ^ 1], bv[cur ^ 1]);      // (past the last term: into the slack row, never used)
            #pragma unroll
            for (int i = 0; i < TM / 2; ++i) {
                float lo, hi;
                unpack2(av[cur][i], lo, hi);
                const f32x2 sw = pack2(hi, lo);
                #pragma unroll
                for (int j = 0; j < TN / 2; ++j) {
                    acc[i][j][0] = add2(acc[i][j][0], fma2(av[cur][i], bv[cur][j], zero2));
                    acc[i][j][1] = add2(acc[i][j][1], fma2(sw, bv[cur][j], zero2));
                }
            }
        };
        int k = 0;
        for (; k + 4 <= rows; k += 4) { term(0); term(1); term(0); term(1); }
        for (; k < rows; k += 2) { term(0); if (k + 1 < rows) term(1); }
        if (!REGS) __syncthreads();
    }
    // Only now may the next kernel's blocks be placed: with all of this grid resident from the start, early ones would
    // take the free slots unevenly, and where the next kernel is another contraction its CTAs would pile up on a few SMs.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    float* y = a.y + blockIdx.z * a.bso;
    const int col = n0 + cg * TN;
    const bool vec = TN >= 4 && (a.N & 3) == 0 && (((uintptr_t)y) & 15) == 0 && col + TN <= a.N;
    #pragma unroll
    for (int i = 0; i < TM; ++i) {
        const long long m = m0 + rg * TM + i;
        if (m >= a.M) continue;
        float o[TN];
        #pragma unroll
        for (int j = 0; j < TN; ++j) {
            // row i of a pair: columns j and j ^ 1 lie straight and swapped, by turns
            float lo, hi;
            unpack2(acc[i >> 1][j >> 1][(i ^ j) & 1], lo, hi);
            o[j] = (j & 1) ? hi : lo;
            if (a.bias && col + j < a.N) o[j] = __fadd_rn(o[j], a.bias[col + j]);
        }
        float* p = y + m * a.N + col;
        if (vec) {
            #pragma unroll
            for (int j = 0; j < TN; j += 4) *(float4*)(p + j) = make_float4(o[j], o[(j + 1) % TN], o[(j + 2) % TN], o[(j + 3) % TN]);
            continue;
        }
        #pragma unroll
        for (int j = 0; j < TN; ++j)
            if (col + j < a.N) p[j] = o[j];
    }
}

static int launch_contract_f32(F32Args& a, int batch, bool conv, bool akc, bool bkc, cudaStream_t s)
{
    // chunk: about 32 terms, so that three CTAs of the large tile fit an SM
    const bool one = a.T == 1;
    a.CC = one ? 32 : 8;
    while (!one && a.CC > 1 && a.CC * a.T > 40) a.CC >>= 1;
    // through registers: 16-byte pieces of both operands, taps few enough for the registers of a thread
    const bool regs = akc && bkc && a.T <= F32_QUADS && (a.C & 3) == 0 && (((uintptr_t)a.x | (uintptr_t)a.w) & 15) == 0 &&
                      (a.a_row & 3) == 0 && (a.b_col & 3) == 0 && (a.bsa & 3) == 0 && (a.bsb & 3) == 0 && a.b_tap < (1 << 20);
    if (regs && !one) a.CC = a.T <= F32_QUADS / 2 ? (F32_QUADS / a.T >= 4 ? 16 : 8) : 4;
    // The 64 x 64 tile (4 x 8 outputs per thread) where it gives every SM a CTA, else 32 x 32.  Measured on both sides (us, 64
    // against 32): matrices of K = 512 with 64 tiles of the large kind 30.9 / 29.4, 135 tiles 31.1 / 47.9, 160 tiles 54.5 / 59.3,
    // 512 tiles 103 / 160; 3 x 3 convolutions with 49 tiles 26.7 / 19.3, 98 - 100 tiles 27.0 / 25.7 and 60.9 / 45.0, 147 tiles
    // 31.9 / 31.8, 196 tiles 38.1 / 40.2: convolutions change sides at one CTA per SM, matrices already at about half of that.
    const long long big = ((a.M + 63) / 64) * ((a.N + 63) / 64) * batch;
    const int bm = big >= sm_count() ? 64 : 32, bn = bm;
    const size_t smem = ((size_t)a.CC * a.T * 2 * (bm + 4 + bn + 4) + 2 * (bm + 4)) * sizeof(float);   // and a slack row of each
    auto go = [&](auto tag) -> int {
        if (const int rc = allow_shared<decltype(tag)::kernel>(smem)) return rc;
        // (more than 65535 batches or column tiles: several launches)
        F32Args q = a;
        for (int b0 = 0; b0 < batch; b0 += 65535)
            for (long long j0 = 0; j0 < a.N; j0 += 65535ll * bn) {
                q.x = a.x + b0 * a.bsa; q.w = a.w + b0 * a.bsb; q.y = a.y + b0 * a.bso;
                q.n_off = (int)j0;
                const long long cols = a.N - j0 < 65535ll * bn ? a.N - j0 : 65535ll * bn;
                launch_pdl(tag.kernel, dim3(div_up(a.M, bm), div_up(cols, bn), (unsigned)(batch - b0 < 65535 ? batch - b0 : 65535)),
                           dim3(F32_THREADS), smem, s, q);
                const int rc = check_launch("contract_f32_kernel");
                if (rc) return rc;
            }
        return B200K_OK;
    };
    #define B200K_F32_KERNELS(TM, TN)                                                                                  \
        do {                                                                                                           \
            if (regs && conv && one) return go(KernelTag<contract_f32_kernel<TM, TN, true, true, true, true, true>>()); \
            if (regs && conv)        return go(KernelTag<contract_f32_kernel<TM, TN, true, true, true, false, true>>()); \
            if (regs)                return go(KernelTag<contract_f32_kernel<TM, TN, false, true, true, true, true>>()); \
            if (conv && one)         return go(KernelTag<contract_f32_kernel<TM, TN, true, true, true, true, false>>()); \
            if (conv)                return go(KernelTag<contract_f32_kernel<TM, TN, true, true, true, false, false>>()); \
            if (akc && bkc)          return go(KernelTag<contract_f32_kernel<TM, TN, false, true, true, true, false>>()); \
            if (akc)                 return go(KernelTag<contract_f32_kernel<TM, TN, false, true, false, true, false>>()); \
            if (bkc)                 return go(KernelTag<contract_f32_kernel<TM, TN, false, false, true, true, false>>()); \
            return go(KernelTag<contract_f32_kernel<TM, TN, false, false, false, true, false>>());                     \
        } while (0)
    if (bm == 64) B200K_F32_KERNELS(4, 8);
    B200K_F32_KERNELS(4, 2);
    #undef B200K_F32_KERNELS
}

// ---- one output per thread: depthwise convolutions, and filters with more taps than a chunk holds ---------------------

struct ConvF32Args {
    const float* x; const float* w; const float* bias; float* y;
    int N, H, W, C, OH, OW, OC, KH, KW, sh, sw, pt, pl, dh, dw, dm;
    long long total;
};

template <bool DEPTHWISE>
__global__ void __launch_bounds__(256) conv_f32_kernel(const ConvF32Args a)
{
    pdl_enter();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.total) return;
    const int co = (int)(i % a.OC);
    long long t = i / a.OC;
    const int ox = (int)(t % a.OW); t /= a.OW;
    const int oy = (int)(t % a.OH);
    const int n = (int)(t / a.OH);
    float sum = 0.0f;
    const int c_end = DEPTHWISE ? 1 : a.C;
    for (int c = 0; c < c_end; ++c) {
        const int ci = DEPTHWISE ? co / a.dm : c;
        for (int ky = 0; ky < a.KH; ++ky) {
            const int iy = oy * a.sh + ky * a.dh - a.pt;
            for (int kx = 0; kx < a.KW; ++kx) {
                const int ix = ox * a.sw + kx * a.dw - a.pl;
                const float wv = DEPTHWISE ? a.w[((long long)ky * a.KW + kx) * a.OC + co]
                                           : a.w[(((long long)co * a.KH + ky) * a.KW + kx) * a.C + ci];
                const bool inside = iy >= 0 && iy < a.H && ix >= 0 && ix < a.W;
                const float xv = inside ? a.x[(((long long)n * a.H + iy) * a.W + ix) * a.C + ci] : 0.0f;
                sum = __fadd_rn(sum, __fmul_rn(wv, xv));
            }
        }
    }
    if (a.bias) sum = __fadd_rn(sum, a.bias[co]);
    a.y[i] = sum;
}

// Depthwise with one output channel per input channel, C a multiple of 4: four channels per thread with 128-bit loads,
// neighbouring threads on neighbouring channels.  Bound by its launch and the loads' latency at the usual sizes.
__global__ void __launch_bounds__(256) dwconv_f32_vec4_kernel(const ConvF32Args a, int total4)
{
    pdl_enter();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total4) return;
    const int c4n = a.C >> 2;
    int t = i / c4n;
    const int c = (i - t * c4n) * 4;
    const int q = t / a.OW, ox = t - q * a.OW;
    const int n = q / a.OH, oy = q - n * a.OH;
    const int iy0 = oy * a.sh - a.pt, ix0 = ox * a.sw - a.pl;
    const float* xp = a.x + (((long long)n * a.H + iy0) * a.W + ix0) * a.C + c;
    const float* wp = a.w + c;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int ky = 0; ky < a.KH; ++ky) {
        const bool iny = (unsigned)(iy0 + ky * a.dh) < (unsigned)a.H;
        const float* xr = xp + (long long)ky * a.dh * a.W * a.C;
        #pragma unroll 3
        for (int kx = 0; kx < a.KW; ++kx, wp += a.OC) {
            const bool in = iny && (unsigned)(ix0 + kx * a.dw) < (unsigned)a.W;
            const float4 xv = in ? *(const float4*)(xr + (long long)kx * a.dw * a.C) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 wv = *(const float4*)wp;
            sum.x = __fadd_rn(sum.x, __fmul_rn(wv.x, xv.x)); sum.y = __fadd_rn(sum.y, __fmul_rn(wv.y, xv.y));
            sum.z = __fadd_rn(sum.z, __fmul_rn(wv.z, xv.z)); sum.w = __fadd_rn(sum.w, __fmul_rn(wv.w, xv.w));
        }
    }
    if (a.bias) {
        sum.x = __fadd_rn(sum.x, a.bias[c]);     sum.y = __fadd_rn(sum.y, a.bias[c + 1]);
        sum.z = __fadd_rn(sum.z, a.bias[c + 2]); sum.w = __fadd_rn(sum.w, a.bias[c + 3]);
    }
    *(float4*)(a.y + (long long)i * 4) = sum;
}

static int launch_conv_f32(const b200k_conv2d_params* p, cudaStream_t s, bool depthwise, const char* who)
{
    B200K_REQUIRE(p, B200K_E_INVALID, "%s: null params", who);
    B200K_REQUIRE(p->x.data && p->w.data && p->y.data, B200K_E_INVALID, "%s: null tensor pointer", who);
    B200K_REQUIRE(p->x.dtype == B200K_F32 && p->w.dtype == B200K_F32 && p->y.dtype == B200K_F32 &&
                  (!p->bias.data || p->bias.dtype == B200K_F32), B200K_E_UNSUPPORTED, "%s: every tensor must be Float32", who);
    B200K_REQUIRE(!p->add_operand.data, B200K_E_UNSUPPORTED, "%s: a fused Add is only available on quantised Convolution2d", who);
    B200K_REQUIRE(p->n > 0 && p->h > 0 && p->wd > 0 && p->c > 0 && p->oh > 0 && p->ow > 0 && p->oc > 0 && p->kh > 0 && p->kw > 0 &&
                  p->stride_h > 0 && p->stride_w > 0 && p->dil_h > 0 && p->dil_w > 0, B200K_E_INVALID, "%s: bad geometry", who);
    B200K_REQUIRE(!depthwise || p->oc % p->c == 0, B200K_E_INVALID, "%s: output channels %d not a multiple of input channels %d", who, p->oc, p->c);
    ConvF32Args a;
    a.x = (const float*)p->x.data; a.w = (const float*)p->w.data; a.bias = (const float*)p->bias.data; a.y = (float*)p->y.data;
    a.N = p->n; a.H = p->h; a.W = p->wd; a.C = p->c; a.OH = p->oh; a.OW = p->ow; a.OC = p->oc; a.KH = p->kh; a.KW = p->kw;
    a.sh = p->stride_h; a.sw = p->stride_w; a.pt = p->pad_top; a.pl = p->pad_left; a.dh = p->dil_h; a.dw = p->dil_w;
    a.dm = depthwise ? p->oc / p->c : 1;
    a.total = (long long)p->n * p->oh * p->ow * p->oc;
    if (!depthwise && (long long)p->kh * p->kw <= F32_MAX_TAPS &&
        ((long long)p->kh * p->dil_h * p->wd + (long long)p->kw * p->dil_w) * p->c < (1ll << 31)) {
        F32Args f;
        memset(&f, 0, sizeof(f));
        f.x = a.x; f.w = a.w; f.bias = a.bias; f.y = a.y;
        f.M = (long long)a.N * a.OH * a.OW; f.N = a.OC; f.C = a.C;
        f.T = a.KH * a.KW; f.KW = a.KW;
        f.H = a.H; f.W = a.W; f.OH = a.OH; f.OW = a.OW; f.sh = a.sh; f.sw = a.sw; f.pt = a.pt; f.pl = a.pl; f.dh = a.dh; f.dw = a.dw;
        f.b_col = (long long)f.T * a.C; f.b_c = 1; f.b_tap = a.C;
        return launch_contract_f32(f, 1, true, true, true, s);
    }
    if (depthwise && a.dm == 1 && (a.C & 3) == 0 && a.total / 4 < (1ll << 31) - 256 && (((uintptr_t)a.x | (uintptr_t)a.w | (uintptr_t)a.y) & 15) == 0) {
        launch_pdl(dwconv_f32_vec4_kernel, dim3(div_up(a.total / 4, 256)), dim3(256), 0, s, a, (int)(a.total / 4));
        return check_launch("dwconv_f32_vec4_kernel");
    }
    if (depthwise) launch_pdl(conv_f32_kernel<true>, dim3(div_up(a.total, 256)), dim3(256), 0, s, a);
    else           launch_pdl(conv_f32_kernel<false>, dim3(div_up(a.total, 256)), dim3(256), 0, s, a);
    return check_launch("conv_f32_kernel");
}

}  // namespace b200k

using namespace b200k;

extern "C" int b200k_conv2d_f32(const b200k_conv2d_params* p, void* stream)
{
    return launch_conv_f32(p, (cudaStream_t)stream, false, "conv2d_f32");
}

extern "C" int b200k_dwconv2d_f32(const b200k_conv2d_params* p, void* stream)
{
    return launch_conv_f32(p, (cudaStream_t)stream, true, "dwconv2d_f32");
}

extern "C" int b200k_fully_connected_f32(const b200k_fc_params* p, void* stream)
{
    B200K_REQUIRE(p, B200K_E_INVALID, "fully_connected_f32: null params");
    B200K_REQUIRE(p->x.data && p->w.data && p->y.data, B200K_E_INVALID, "fully_connected_f32: null tensor pointer");
    B200K_REQUIRE(p->x.dtype == B200K_F32 && p->w.dtype == B200K_F32 && p->y.dtype == B200K_F32 &&
                  (!p->bias.data || p->bias.dtype == B200K_F32), B200K_E_UNSUPPORTED, "fully_connected_f32: every tensor must be Float32");
    B200K_REQUIRE(p->m > 0 && p->k > 0 && p->n > 0, B200K_E_INVALID, "fully_connected_f32: bad shape");
    F32Args a;
    memset(&a, 0, sizeof(a));
    a.x = (const float*)p->x.data; a.w = (const float*)p->w.data; a.bias = (const float*)p->bias.data; a.y = (float*)p->y.data;
    a.M = p->m; a.C = p->k; a.N = p->n; a.T = a.KW = 1;
    a.a_row = p->k; a.a_c = 1;
    a.b_col = p->transpose_w ? p->k : 1; a.b_c = p->transpose_w ? 1 : p->n;
    return launch_contract_f32(a, 1, false, true, p->transpose_w != 0, (cudaStream_t)stream);
}

extern "C" int b200k_batch_matmul_f32(const b200k_bmm_params* p, void* stream)
{
    B200K_REQUIRE(p, B200K_E_INVALID, "batch_matmul_f32: null params");
    B200K_REQUIRE(p->x.data && p->y.data && p->out.data, B200K_E_INVALID, "batch_matmul_f32: null tensor pointer");
    B200K_REQUIRE(p->x.dtype == B200K_F32 && p->y.dtype == B200K_F32 && p->out.dtype == B200K_F32, B200K_E_UNSUPPORTED,
                  "batch_matmul_f32: every tensor must be Float32");
    B200K_REQUIRE(p->batch > 0 && p->m > 0 && p->k > 0 && p->n > 0 && p->batch_stride_x >= 0 && p->batch_stride_y >= 0,
                  B200K_E_INVALID, "batch_matmul_f32: bad shape");
    F32Args a;
    memset(&a, 0, sizeof(a));
    a.x = (const float*)p->x.data; a.w = (const float*)p->y.data; a.y = (float*)p->out.data;
    a.M = p->m; a.C = p->k; a.N = p->n; a.T = a.KW = 1;
    a.a_row = p->transpose_x ? 1 : p->k; a.a_c = p->transpose_x ? p->m : 1;
    a.b_col = p->transpose_y ? p->k : 1; a.b_c = p->transpose_y ? 1 : p->n;
    a.bsa = p->batch_stride_x; a.bsb = p->batch_stride_y; a.bso = (long long)p->m * p->n;
    return launch_contract_f32(a, p->batch, false, !p->transpose_x, p->transpose_y != 0, (cudaStream_t)stream);
}
