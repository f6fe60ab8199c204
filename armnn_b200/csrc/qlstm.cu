// One QLstm step, reproducing RefQLstmWorkload::Execute operation by operation
// (src/backends/reference/workloads/RefQLstmWorkload.cpp:46-541, LstmUtils.cpp:16-256 of the Arm NN tree).
//
// CpuRef keeps the gate pre-activations in int16 buffers and re-quantises them after EVERY multiply-accumulate of the
// mat-vec products (LstmUtils.cpp:87-111), so a gate value is the end of a K-long chain
//     acc <- clamp16(round_half_away(fl(fl(fl(acc * sG) + fl(fl(w * sw) * x)) / sG)))
// whose result depends on every intermediate rounding and saturation; an int32 dot product followed by one requantisation
// is a different function.  But acc is an integer and acc * sG / sG is acc up to a few roundings, so the step adds
// round(r), r = w x sw / sG, whatever acc is, unless r lies within
//     E = 2^-24 (3 |acc| + 8 |r| + 8)
// of a half or the sum reaches the clamp.  One fused multiply-add does that step:
//     T' = RN(T + w xc),  xc = x sw / sG,  T = 1.5 * 2^23 + acc.
// r depends on the product of two bytes only.  The host lists, per pair of gates, the input magnitudes for which SOME weight
// byte comes that close to a half (with |acc| <= QL_LEVEL; with the scales of the reference's own test a third of the inputs
// for two gates, one in a hundred for the others).  A block of 16 steps without such an input is 16 FMAs.  In any other
// block d = w xc - (T' - T), exact, is formed as well, and its largest magnitude tells whether every rounding was the
// reference's.  Half blocks that cannot vouch for themselves (two per thread and row on average) are noted down with the
// accumulators they began with, and their doubtful steps are evaluated with the reference's own arithmetic at the end of the
// chain: as a step's increment does not depend on acc, a rounding that went the other way shifts everything after it by the
// same integer.  A warp with an accumulator that might reach the clamp evaluates the block by the reference's arithmetic.
//
// A cluster of CTAs works on R (1 or 2) batch rows: every CTA runs the chains of its share of the units (a thread has two
// gates of one unit, a packed pair, and converts each weight once for all R rows; weights come through shared memory, a
// tile ahead) and writes the results into the shared memory of the row's owner; CTA r of the cluster then takes row r
// through (peephole) -> layer norm -> activations -> cell update -> output gate -> hidden state -> projection (chains of the
// same kind) -> outputs.  Layer-norm sums are sequential in the reference: one thread per gate, its operands read ahead.
//
// Bound by the fp32 and integer pipes in the chains (about 60 % of the time at 512 units) and by the latency of the sequential
// sums and of the projection's chains.  Three layers (40 or 256 -> 512 units -> 256) at batch 128: 475 us with one CTA per row and
// the reference's arithmetic in every step, 310 us with blocks of eight steps, 283 us with 16 and both rows interleaved, 255 us
// since notes keep their weights.
#include <mutex>
#include <type_traits>
#include "common.cuh"

namespace b200k {

constexpr int QL_UNITS = 256;                    // units a CTA works on at a time: one thread per unit and pair of gates
constexpr int QL_THREADS = 2 * QL_UNITS;
constexpr int QL_SEG = 1024;                     // steps whose factors are staged at once, at most
constexpr int QL_TILE = 64, QL_PITCH = QL_TILE + 16;     // weight bytes per row and tile; conflict-free 128-bit reads
constexpr int QL_TILE_BYTES = 4 * QL_UNITS * QL_PITCH;
constexpr int QL_NOTES = 8;                      // doubtful half blocks a thread can note down per row
constexpr int QL_BLOCK = 16;                     // steps of a block
constexpr float QL_LEVEL = 2048.0f;              // |acc| up to which the host's list of inputs holds
constexpr float QL_NEAR_CLAMP = 32000.0f;        // |acc| from which on saturation is possible (zero points included)
constexpr float QL_ULP = 6.0e-8f;                // a little more than 2^-24
constexpr int QL_GATE_SLACK = 64;                // floats behind the gate buffers (the projection factors are padded)
constexpr float QL_MAGIC = 12582912.0f;          // 1.5 * 2^23

// round_half_away(fl(v / scale)) without the division unit (inv = rn_reciprocal(scale), NaN where the quotient does not hold):
// Markstein's correctly rounded quotient and the 1.5 * 2^23 constant; exact halves, and whatever is not finite, go through the
// division.
__device__ __forceinline__ float ql_round_div(float v, float scale, float inv)
{
    const float p = __fmul_rn(v, inv);
    const float q = __fmaf_rn(__fmaf_rn(-p, scale, v), inv, p);
    float n = __fsub_rn(__fadd_rn(q, QL_MAGIC), QL_MAGIC);
    if (!(fabsf(__fsub_rn(q, n)) < 0.5f)) n = roundf(__fdiv_rn(v, scale));
    return n;
}
__device__ __forceinline__ float q16f(float v, float scale, float inv)          // Quantize<int16_t>, offset 0, as float
{
    return fminf(fmaxf(ql_round_div(v, scale, inv), -32768.f), 32767.f);
}
__device__ __forceinline__ float q16zf(float v, float scale, float zp)
{
    return fminf(fmaxf(__fadd_rn(zp, roundf(__fdiv_rn(v, scale))), -32768.f), 32767.f);
}

// Input magnitudes 0 .. 255 (|q - zero point|), one bit each, that can bring a product close to a half.
struct QlDanger { uint32_t bits[8]; };

struct QlArgs {
    b200k_qlstm_params p;
    int cifg, peephole, ln, proj;
    int seg, both;                               // staged steps: a multiple of 16; both sources fit at once
    int exact_only;                              // scales outside the range the error bound holds for: every step by the reference's arithmetic
    int vec_i, vec_o, vec_p;                     // weight rows are whole aligned 16-byte pieces
    int nbuf;                                    // weight tiles in shared memory: 1 or 2
    int proj_staged;                             // the projection weights fit the tiles' space
    unsigned tile_off;                           // where the weight tiles begin in shared memory
    float inv_gate[4], inv_ln[4], inv_cell, inv_out;     // reciprocals of the scales that are divided by, gates i, f, c, o
    QlDanger danger[3][2];                       // [input, recurrent, projection][pair of gates: (i, c), (f, o)]
};

__device__ __forceinline__ uint32_t ql_cluster_size() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t ql_cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void ql_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void ql_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// a float into the shared memory of CTA `rank` of the cluster, at the address `mine` has in this CTA
__device__ __forceinline__ void ql_store_remote(float* mine, uint32_t rank, float v)
{
    const uint32_t local = (uint32_t)__cvta_generic_to_shared(mine);
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}
__device__ __forceinline__ void ql_copy16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void ql_copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void ql_copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// four weights of a row from k on, zeros beyond K
__device__ __forceinline__ uint32_t ql_weights4(const int8_t* w, int k, int K)
{
    uint32_t v = 0;
    #pragma unroll
    for (int i = 0; i < 4; ++i)
        if (k + i < K) v |= (uint32_t)(uint8_t)w[k + i] << (8 * i);
    return v;
}

// One step of a pair of chains with the reference's arithmetic.  acc2: integers; products that the reference rounds
// before adding are fma2(a, b, 0) (a packed multiply feeding a packed add would be contracted); the quotient is
// Markstein's correctly rounded one.
struct QlExact {
    f32x2 sG2, nsG2, iG2, sw2;
    float lo, hi;                                // clamp
    __device__ __forceinline__ void set(float sGa, float sGb, float iGa, float iGb, float swa, float swb, float l, float h)
    {
        sG2 = pack2(sGa, sGb); nsG2 = pack2(-sGa, -sGb); iG2 = pack2(iGa, iGb); sw2 = pack2(swa, swb);
        lo = l; hi = h;
    }
    // fl(acc * sG) + t, to be divided by sG
    __device__ __forceinline__ f32x2 dividend(f32x2 T, f32x2 w2, float x) const
    {
        const f32x2 zero2 = pack2(0.f, 0.f), magic2 = pack2(QL_MAGIC, QL_MAGIC);
        const f32x2 t2 = fma2(fma2(w2, sw2, zero2), pack2(x, x), zero2);                      // fl(fl(w * sw) * x)
        return add2(fma2(sub2(T, magic2), sG2, zero2), t2);
    }
    __device__ __forceinline__ f32x2 quotient(f32x2 a2) const
    {
        const f32x2 p2 = mul2(a2, iG2);
        return fma2(fma2(p2, nsG2, a2), iG2, p2);                                             // RN(a / sG)
    }
};

// a byte of each of two words as a pair of floats, signed
__device__ __forceinline__ f32x2 ql_weight_pair(uint32_t a, uint32_t b, int j, f32x2 off2)
{
    return sub2(pack2(__uint_as_float(__byte_perm(a, 0x4b000000u, 0x7440 + j)), __uint_as_float(__byte_perm(b, 0x4b000000u, 0x7440 + j))), off2);
}

// A block of steps by the reference's arithmetic, halves and clamp included.  x: the steps' dequantised values.
__device__ __noinline__ f32x2 ql_slow_block(f32x2 T, uint4 wa, uint4 wb, const float* x, const QlExact* e)
{
    const f32x2 magic2 = pack2(QL_MAGIC, QL_MAGIC), woff2 = pack2(8388608.0f + 128.0f, 8388608.0f + 128.0f);
    const QlExact ex = *e;
    uint32_t ma[4] = {wa.x ^ 0x80808080u, wa.y ^ 0x80808080u, wa.z ^ 0x80808080u, wa.w ^ 0x80808080u};
    uint32_t mb[4] = {wb.x ^ 0x80808080u, wb.y ^ 0x80808080u, wb.z ^ 0x80808080u, wb.w ^ 0x80808080u};
    #pragma unroll 1
    for (int j = 0; j < QL_BLOCK; j += 4) {
        #pragma unroll
        for (int i = 0; i < 4; ++i) {
            const f32x2 a2 = ex.dividend(T, ql_weight_pair(ma[0], mb[0], i, woff2), x[j + i]), q2 = ex.quotient(a2);
            float qa, qb, na, nb;
            unpack2(q2, qa, qb);
            unpack2(sub2(add2(q2, magic2), magic2), na, nb);
            const bool ha = !(fabsf(__fsub_rn(qa, na)) < 0.5f), hb = !(fabsf(__fsub_rn(qb, nb)) < 0.5f);
            if (ha || hb) {                                  // (halves, and quotients that overflow on the way)
                float aa, ab, sa, sb;
                unpack2(a2, aa, ab); unpack2(ex.sG2, sa, sb);
                if (ha) na = roundf(__fdiv_rn(aa, sa));
                if (hb) nb = roundf(__fdiv_rn(ab, sb));
            }
            T = add2(pack2(fminf(fmaxf(na, ex.lo), ex.hi), fminf(fmaxf(nb, ex.lo), ex.hi)), magic2);
        }
        ma[0] = ma[1]; ma[1] = ma[2]; ma[2] = ma[3];
        mb[0] = mb[1]; mb[1] = mb[2]; mb[2] = mb[3];
    }
    return T;
}

// Bounds of a block: x = how far an accumulator can move in it (|w| <= 128, half a unit of rounding per step),
// corrections that notes may bring included; y = the part of E that does not depend on the accumulators it begins with.
__device__ __forceinline__ float2 ql_bounds(float sum_abs, float max_abs)
{
    const float s = __fmaf_rn(128.5f, sum_abs, 0.5f * QL_BLOCK + 0.5f) + 8.0f * QL_NOTES;
    return make_float2(s, QL_ULP * (3.0f * s + 8.0f * 128.0f * max_abs + 8.0f));
}

// The bounds of a block whose largest factors (of the two chains) the lanes of half a warp have, a step each; listed: one of the
// inputs is on the host's list.  Called by whole warps.
struct QlBlockInfo { float2 bounds; uint8_t listed; };
__device__ __forceinline__ QlBlockInfo ql_block_info(float factor, const QlDanger& danger, int mag, int exact_only)
{
    float sum = factor, mx = factor;
    const uint32_t on_list = (danger.bits[(mag >> 5) & 7] >> (mag & 31)) & 1u;
    #pragma unroll
    for (int d = 1; d < QL_BLOCK; d *= 2) {
        sum += __shfl_xor_sync(0xffffffffu, sum, d);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
    }
    const uint32_t votes = __ballot_sync(0xffffffffu, on_list != 0);
    QlBlockInfo info;
    info.bounds = ql_bounds(exact_only ? 1e30f : sum, mx);
    info.listed = (votes >> (threadIdx.x & 16) & 0xffffu) != 0;
    return info;
}

// A doubtful half block: the two accumulators before it (whose 16 bits are the low halves of T's words), its weight bytes as
// ql_block has them (fetching them again at the end of the chain cost more than the evaluation), and its first step.
struct QlNote {
    uint4 w;
    uint32_t acc, pos;
};
// A packed pair of chains and its doubtful half blocks.  Only the notes have an address, so that the rest stays in registers.
struct QlChains {
    f32x2 T;
    int notes;
    QlNote* note;
};

// What noted half blocks are corrected from, and the weight rows of the pair.
struct QlSource {
    const float2* xc;                            // factors of the pair, by position
    const float* xf;                             // dequantised values
    const float2* bounds;                        // by block
    const uint8_t* listed;                       // by block: one of the inputs is on the host's list
    const QlExact* e;
    const int8_t* wa; const int8_t* wb;          // weight rows: position 0 is step `first` of `K`
    int first, K, aligned;                       // aligned: weights come in whole aligned words
    __device__ __forceinline__ uint4 weights16(const int8_t* w, int pos) const
    {
        if (aligned) return *(const uint4*)(w + first + pos);
        return make_uint4(ql_weights4(w, first + pos, K), ql_weights4(w, first + pos + 4, K), ql_weights4(w, first + pos + 8, K), ql_weights4(w, first + pos + 12, K));
    }
};

// Evaluates the doubtful steps of the noted half blocks with the reference's arithmetic and corrects the accumulators.
__device__ __noinline__ f32x2 ql_resolve(f32x2 end, int notes, const QlNote* list, const float2* xc, const float* xf, const float2* bounds, const QlExact* exact)
{
    const f32x2 magic2 = pack2(QL_MAGIC, QL_MAGIC), woff2 = pack2(8388608.0f + 128.0f, 8388608.0f + 128.0f);
    const QlExact e = *exact;
    f32x2 corr2 = pack2(0.f, 0.f);               // what the reference's accumulators are ahead by
    QlNote next = list[0];
    #pragma unroll 1
    for (int i = 0; i < notes; ++i) {
        const QlNote note = next;
        if (i + 1 < notes) next = list[i + 1];
        const int pos = (int)note.pos;
        const float a0 = (float)(short)(note.acc & 0xffffu), a1 = (float)((int)note.acc >> 16);
        const float thr = 0.5f - __fmaf_rn(3.0f * QL_ULP, fmaxf(fabsf(a0), fabsf(a1)), bounds[pos / QL_BLOCK].y);
        const uint32_t ma[2] = {note.w.x, note.w.y}, mb[2] = {note.w.z, note.w.w};
        f32x2 T[9], w2[8];
        T[0] = pack2(a0 + QL_MAGIC, a1 + QL_MAGIC);
        uint32_t doubtful = 0;
        #pragma unroll
        for (int j = 0; j < 8; ++j) {
            w2[j] = ql_weight_pair(ma[j >> 2], mb[j >> 2], j & 3, woff2);
            const float2 c = xc[pos + j];
            const f32x2 c2 = pack2(c.x, c.y);
            T[j + 1] = fma2(w2[j], c2, T[j]);
            float d0, d1;
            unpack2(fma2(w2[j], c2, sub2(T[j], T[j + 1])), d0, d1);
            if (!(fmaxf(fabsf(d0), fabsf(d1)) < thr)) doubtful |= 1u << j;
        }
        #pragma unroll 1
        while (doubtful) {
            const int k = __ffs((int)doubtful) - 1;
            doubtful &= doubtful - 1;
            f32x2 t = T[0], next = T[1], w = w2[0];
            #pragma unroll
            for (int j = 1; j < 8; ++j)
                if (j == k) { t = T[j]; next = T[j + 1]; w = w2[j]; }
            const f32x2 q2 = e.quotient(e.dividend(add2(t, corr2), w, xf[pos + k]));
            float qa, qb, na, nb;
            unpack2(q2, qa, qb);
            unpack2(sub2(add2(q2, magic2), magic2), na, nb);
            if (!(fabsf(__fsub_rn(qa, na)) < 0.5f)) na = roundf(qa);
            if (!(fabsf(__fsub_rn(qb, nb)) < 0.5f)) nb = roundf(qb);
            corr2 = sub2(pack2(na, nb), sub2(next, magic2));
        }
    }
    return add2(end, corr2);
}

// A block of steps, from position `pos` on, of the pairs of chains of R rows; ma, mb: the weight bytes with their sign flipped.
template <int R>
__device__ __forceinline__ void ql_block(QlChains (&ch)[R], const uint32_t (&ma)[4], const uint32_t (&mb)[4], int pos, const QlSource (&src)[R])
{
    const f32x2 magic2 = pack2(QL_MAGIC, QL_MAGIC), woff2 = pack2(8388608.0f + 128.0f, 8388608.0f + 128.0f);
    float2 bd[R];
    float amax[R];
    bool checked = false, beyond = false, done[R];
    #pragma unroll
    for (int r = 0; r < R; ++r) {
        bd[r] = src[r].bounds[pos / QL_BLOCK];
        checked |= src[r].listed[pos / QL_BLOCK] != 0;
        float f0, f1;
        unpack2(sub2(ch[r].T, magic2), f0, f1);
        amax[r] = fmaxf(fabsf(f0), fabsf(f1));
        beyond |= !(amax[r] + bd[r].x <= QL_LEVEL) || ch[r].notes > QL_NOTES - 2;
        done[r] = false;
    }
    if (__any_sync(0xffffffffu, beyond)) {
        checked = true;
        #pragma unroll
        for (int r = 0; r < R; ++r) {
            const bool far = __any_sync(0xffffffffu, !(amax[r] + bd[r].x <= QL_NEAR_CLAMP));
            if (far || __any_sync(0xffffffffu, ch[r].notes > QL_NOTES - 2)) {
                ch[r].T = ql_resolve(ch[r].T, ch[r].notes, ch[r].note, src[r].xc, src[r].xf, src[r].bounds, src[r].e);
                ch[r].notes = 0;
                if (far) {
                    ch[r].T = ql_slow_block(ch[r].T, src[r].weights16(src[r].wa, pos), src[r].weights16(src[r].wb, pos), src[r].xf + pos, src[r].e);
                    done[r] = true;
                }
            }
        }
    }
    f32x2 t[R];
    #pragma unroll
    for (int r = 0; r < R; ++r) t[r] = ch[r].T;
    auto factors = [&](int r, int j, f32x2& c0, f32x2& c1) {
        const float4 x = *(const float4*)(src[r].xc + pos + j);
        c0 = pack2(x.x, x.y); c1 = pack2(x.z, x.w);
    };
    if (!checked) {
        #pragma unroll
        for (int j = 0; j < QL_BLOCK; j += 2) {
            const f32x2 w0 = ql_weight_pair(ma[j >> 2], mb[j >> 2], j & 3, woff2), w1 = ql_weight_pair(ma[j >> 2], mb[j >> 2], (j + 1) & 3, woff2);
            #pragma unroll
            for (int r = 0; r < R; ++r) {
                f32x2 c0, c1;
                factors(r, j, c0, c1);
                t[r] = fma2(w1, c1, fma2(w0, c0, t[r]));
            }
        }
        #pragma unroll
        for (int r = 0; r < R; ++r)
            if (!done[r]) ch[r].T = t[r];
        return;
    }
    float dmax[R][2];
    f32x2 half[R];
    #pragma unroll
    for (int r = 0; r < R; ++r) dmax[r][0] = dmax[r][1] = 0.f;
    #pragma unroll
    for (int j = 0; j < QL_BLOCK; j += 2) {
        const f32x2 w0 = ql_weight_pair(ma[j >> 2], mb[j >> 2], j & 3, woff2), w1 = ql_weight_pair(ma[j >> 2], mb[j >> 2], (j + 1) & 3, woff2);
        #pragma unroll
        for (int r = 0; r < R; ++r) {
            if (j == QL_BLOCK / 2) half[r] = t[r];
            f32x2 c0, c1;
            factors(r, j, c0, c1);
            const f32x2 t0 = t[r], t1 = fma2(w0, c0, t0), t2 = fma2(w1, c1, t1);
            float d0, d1, d2, d3;
            unpack2(fma2(w0, c0, sub2(t0, t1)), d0, d1);
            unpack2(fma2(w1, c1, sub2(t1, t2)), d2, d3);
            float& m = dmax[r][j >= QL_BLOCK / 2];
            m = fmaxf(fmaxf(m, fabsf(d0)), fabsf(d1));
            m = fmaxf(fmaxf(m, fabsf(d2)), fabsf(d3));
            t[r] = t2;
        }
    }
    #pragma unroll
    for (int r = 0; r < R; ++r) {
        if (done[r]) continue;
        const float e = __fmaf_rn(3.0f * QL_ULP, amax[r], bd[r].y);
        const bool n0 = !(__fadd_rn(dmax[r][0], e) < 0.5f), n1 = !(__fadd_rn(dmax[r][1], e) < 0.5f);
        if (n0 || n1) {
            auto note = [&](f32x2 begin, int h) {
                float t0, t1;
                unpack2(begin, t0, t1);
                QlNote& to = ch[r].note[ch[r].notes++];
                to.w = make_uint4(ma[2 * h], ma[2 * h + 1], mb[2 * h], mb[2 * h + 1]);
                to.acc = __byte_perm(__float_as_uint(t0), __float_as_uint(t1), 0x5410);
                to.pos = (uint32_t)(pos + h * (QL_BLOCK / 2));
            };
            if (n0) note(ch[r].T, 0);
            if (n1) note(half[r], 1);
        }
        ch[r].T = t[r];
    }
}

template <int R>
__global__ void __launch_bounds__(QL_THREADS, 1) qlstm_step_kernel(const __grid_constant__ QlArgs a)
{
    pdl_enter();
    const b200k_qlstm_params& p = a.p;
    const int I = p.input_size, U = p.num_units, O = p.output_size;
    const int tid = threadIdx.x;
    const int nct = (int)ql_cluster_size(), rank = (int)ql_cluster_rank();
    const int b0 = (int)(blockIdx.x / (unsigned)nct) * R;    // first of the cluster's rows
    if (nct > 1) ql_cluster_arrive();                        // (every CTA of the cluster runs before anyone writes to it)

    extern __shared__ float4 ql_smem[];
    __shared__ QlDanger s_danger[3][2];
    __shared__ QlExact s_exact[2][2];
    float* gates = (float*)ql_smem;                          // [4][U] int16 gate buffers as integer-valued floats (o, i, f, c)
    auto gate = [&](int g) { return gates + ((g + 1) & 3) * U; };
    float* work = gates + ((4 * U + QL_GATE_SLACK + 3) & ~3);
    // chains of the gates, by row and pair (i and c, f and o): factors of every step; by block of steps: its bounds, and
    // whether one of its inputs is on the host's list
    const int nblk = a.seg / QL_BLOCK;
    float2* xc = (float2*)work;                              // [R][2][seg]
    float2* bounds = xc + R * 2 * a.seg;                     // [R][2][nblk]
    float* xf = (float*)(bounds + R * 2 * nblk);             // [R][seg] dequantised values
    uint8_t* listed = (uint8_t*)(xf + R * a.seg);            // [R][2][nblk]
    // afterwards, in the same place:
    float* cell = work;                                      // [U] new cell state (integer-valued)
    float* stat = cell + U;                                  // [4][2] mean, 1 / stddev per gate
    float* hid = stat + 8;                                   // [U rounded up to 16] dequantised hidden state
    // and, where the i, f and c gates were:
    float2* hc = (float2*)(gates + ((U + 3) & ~3));          // [U rounded up to 16] projection factor of a unit, twice
    float2* hbounds = hc + ((U + 15) & ~15);                 // [U rounded up to 16, / 16]
    uint8_t* hlisted = (uint8_t*)(hbounds + ((U + 15) & ~15) / QL_BLOCK);    // the same
    // weights: nbuf tiles of 4 x QL_UNITS rows (gate-major), then the whole projection matrix
    uint8_t* tiles = (uint8_t*)ql_smem + a.tile_off;

    const int8_t* wi[4] = {a.cifg ? p.w_i2f : p.w_i2i, p.w_i2f, p.w_i2c, p.w_i2o};       // (CIFG: a chain that nobody reads)
    const int8_t* wr[4] = {a.cifg ? p.w_r2f : p.w_r2i, p.w_r2f, p.w_r2c, p.w_r2o};
    const float si[4] = {a.cifg ? p.s_i2f : p.s_i2i, p.s_i2f, p.s_i2c, p.s_i2o};
    const float sr[4] = {a.cifg ? p.s_r2f : p.s_r2i, p.s_r2f, p.s_r2c, p.s_r2o};
    const float sint[4] = {a.cifg ? p.forget_intermediate_scale : p.input_intermediate_scale, p.forget_intermediate_scale,
                           p.cell_intermediate_scale, p.output_intermediate_scale};

    for (int i = tid; i < (int)(sizeof(s_danger) / 4); i += QL_THREADS) ((uint32_t*)s_danger)[i] = ((const uint32_t*)a.danger)[i];
    if (tid < 4) {
        const int src = tid >> 1, pr = tid & 1;
        s_exact[src][pr].set(pr ? sint[1] : sint[0], pr ? sint[3] : sint[2], a.inv_gate[pr], a.inv_gate[pr + 2], src ? (pr ? sr[1] : sr[0]) : (pr ? si[1] : si[0]),
                             src ? (pr ? sr[3] : sr[2]) : (pr ? si[3] : si[2]), -32768.f, 32767.f);
    }

    auto row_of = [&](int r) { return min(b0 + r, p.batch - 1); };          // a cluster's missing last row repeats its first
    // n steps from k0 on of source `src` (0 input, 1 previous output), at position `at` of the staged arrays
    auto stage = [&](int src, int k0, int n, int at) {
        const int n16 = (n + 15) & ~15;
        float c[4];
        #pragma unroll
        for (int g = 0; g < 4; ++g) c[g] = __fdiv_rn(src == 0 ? si[g] : sr[g], sint[g]);
        const int K = src == 0 ? I : O, zp = src == 0 ? p.input_zp : p.output_state_zp;
        const float scale = src == 0 ? p.input_scale : p.output_state_scale;
        const int8_t* base = src == 0 ? p.input : p.output_state_in;
        __syncthreads();
        // a step per thread; 16 neighbouring lanes have a block (whole warps take part in its reduction)
        for (int i = tid; (i & ~31) < R * n16; i += QL_THREADS) {
            const bool in = i < R * n16;
            const int r = in ? i / n16 : 0, k = in ? i - r * n16 : 0;
            const int q = in && k < n ? (int)base[(long long)row_of(r) * K + k0 + k] - zp : 0, mag = abs(q);
            const float v = __fmul_rn(__int2float_rn(q), scale);
            if (in) xf[r * a.seg + at + k] = v;
            #pragma unroll
            for (int pr = 0; pr < 2; ++pr) {
                const float2 f = make_float2(__fmul_rn(v, pr ? c[1] : c[0]), __fmul_rn(v, pr ? c[3] : c[2]));
                if (in) xc[(r * 2 + pr) * a.seg + at + k] = f;
                const QlBlockInfo info = ql_block_info(fmaxf(fabsf(f.x), fabsf(f.y)), s_danger[src][pr], mag, a.exact_only);
                if (in && (tid & 15) == 0) {
                    bounds[(r * 2 + pr) * nblk + (at + k) / QL_BLOCK] = info.bounds;
                    listed[(r * 2 + pr) * nblk + (at + k) / QL_BLOCK] = info.listed;
                }
            }
        }
        __syncthreads();
    };

    // ---- the gates' chains: input weights first, then recurrent weights, continuing the same accumulators.  Usually both
    // sources are staged side by side once; a long layer's are staged piece by piece.
    const int Us = (U + nct - 1) / nct, u_lo = rank * Us, u_hi = min(U, u_lo + Us);
    const int I16 = (I + 15) & ~15;
    __syncthreads();
    if (a.both) { stage(0, 0, I, 0); stage(1, 0, O, I16); }
    if (nct > 1) ql_cluster_wait();
    const int pr = tid / QL_UNITS, ul = tid % QL_UNITS;      // this thread's gates: pr and pr + 2; its unit within the pass
    for (int ub = u_lo; ub < u_hi; ub += QL_UNITS) {
        const int units = min(QL_UNITS, u_hi - ub);
        const bool busy = (ul & ~31) < units;                // (warp-uniform; lanes beyond the last unit repeat it)
        QlChains ch[R];
        QlNote notes[R][QL_NOTES];
        #pragma unroll
        for (int r = 0; r < R; ++r) { ch[r].T = pack2(QL_MAGIC, QL_MAGIC); ch[r].notes = 0; ch[r].note = notes[r]; }
        // by source, and by the pieces of it that are staged at once
        #pragma unroll 1
        for (int piece = 0, src = 0; src < 2; ) {
            const int K = src == 0 ? I : O, step = a.both ? K : a.seg;
            const int k0 = piece * step, n = min(step, K - k0), at = a.both && src ? I16 : 0;
            const bool vec = src == 0 ? a.vec_i : a.vec_o;
            if (!a.both) stage(src, k0, n, 0);
            auto fetch = [&](int t, int buf) {               // the tile of steps [t, t + QL_TILE)
                #pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const int8_t* w = (src ? wr[g] : wi[g]) + (long long)ub * K + k0 + t;
                    uint8_t* d = tiles + buf * QL_TILE_BYTES + g * QL_UNITS * QL_PITCH;
                    if (vec) {
                        const int c = (tid & 3) * 16;
                        #pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int row = h * (QL_THREADS / 4) + (tid >> 2);
                            if (row < units && t + c < n) ql_copy16(d + row * QL_PITCH + c, w + (long long)row * K + c);
                        }
                    } else {
                        const int c = (tid & 15) * 4;
                        #pragma unroll 4
                        for (int row = tid >> 4; row < units; row += QL_THREADS / 16)
                            if (t + c < n) *(uint32_t*)(d + row * QL_PITCH + c) = ql_weights4(w + (long long)row * K, c, n - t);
                    }
                }
                ql_copy_commit();
            };
            QlSource from[R];
            #pragma unroll
            for (int r = 0; r < R; ++r) {
                from[r].xc = xc + (r * 2 + pr) * a.seg + at; from[r].xf = xf + r * a.seg + at;
                from[r].bounds = bounds + (r * 2 + pr) * nblk + at / QL_BLOCK;
                from[r].listed = listed + (r * 2 + pr) * nblk + at / QL_BLOCK;
                from[r].e = &s_exact[src][pr];
                const long long row = (long long)(ub + min(ul, units - 1)) * K;
                from[r].wa = (src ? (pr ? wr[1] : wr[0]) : (pr ? wi[1] : wi[0])) + row;
                from[r].wb = (src ? (pr ? wr[3] : wr[2]) : (pr ? wi[3] : wi[2])) + row;
                from[r].first = k0; from[r].K = K; from[r].aligned = vec;
            }
            const uint8_t* ta = tiles + (pr * QL_UNITS + min(ul, units - 1)) * QL_PITCH;
            fetch(0, 0);
            int buf = 0;
            #pragma unroll 1
            for (int t = 0; t < n; t += QL_TILE) {
                const bool ahead = a.nbuf == 2 && t + QL_TILE < n;
                if (ahead) { fetch(t + QL_TILE, buf ^ 1); ql_copy_wait<1>(); }
                else ql_copy_wait<0>();
                __syncthreads();
                if (busy) {
                    const uint8_t* tb = ta + buf * QL_TILE_BYTES;
                    #pragma unroll 1
                    for (int k = t; k < min(n, t + QL_TILE); k += QL_BLOCK) {
                        const uint4 na = *(const uint4*)(tb + k - t), nb = *(const uint4*)(tb + 2 * QL_UNITS * QL_PITCH + k - t);
                        const uint32_t ma[4] = {na.x ^ 0x80808080u, na.y ^ 0x80808080u, na.z ^ 0x80808080u, na.w ^ 0x80808080u};
                        const uint32_t mb[4] = {nb.x ^ 0x80808080u, nb.y ^ 0x80808080u, nb.z ^ 0x80808080u, nb.w ^ 0x80808080u};
                        ql_block<R>(ch, ma, mb, k, from);
                    }
                }
                __syncthreads();                             // (everyone has left the tile before it is overwritten)
                if (a.nbuf == 2) buf ^= 1;
                else if (t + QL_TILE < n) fetch(t + QL_TILE, 0);
            }
            #pragma unroll
            for (int r = 0; r < R; ++r) {
                ch[r].T = ql_resolve(ch[r].T, ch[r].notes, ch[r].note, from[r].xc, from[r].xf, from[r].bounds, from[r].e);
                ch[r].notes = 0;
            }
            ++piece;
            if (piece * step >= K) { piece = 0; ++src; }
        }
        if (ul < units) {
            #pragma unroll
            for (int r = 0; r < R; ++r) {
                float f[2];
                unpack2(sub2(ch[r].T, pack2(QL_MAGIC, QL_MAGIC)), f[0], f[1]);
                #pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float* to = gate(pr + 2 * h) + ub + ul;
                    if (nct > 1) ql_store_remote(to, (uint32_t)r, f[h]);
                    else *to = f[h];
                }
            }
        }
    }
    if (nct > 1) { ql_cluster_arrive(); ql_cluster_wait(); }
    else __syncthreads();
    // from here on CTA r works alone on row r
    const int b = b0 + rank;
    if (rank >= R || b >= p.batch) return;

    const float sc = p.cell_state_scale, isc = a.inv_cell;
    const int g0 = a.cifg ? 1 : 0;
    const int16_t* peep[4] = {p.w_c2i, p.w_c2f, nullptr, p.w_c2o};
    const float speep[4] = {p.s_c2i, p.s_c2f, 0.f, p.s_c2o};
    const int16_t* lnw[4] = {p.ln_i, p.ln_f, p.ln_c, p.ln_o};
    const float slnw[4] = {p.s_lni, p.s_lnf, p.s_lnc, p.s_lno};
    const int32_t* gbias[4] = {p.b_i, p.b_f, p.b_c, p.b_o};
    const float sgb[4] = {p.s_bi, p.s_bf, p.s_bc, p.s_bo};

    // The projection weights, [O][U16 + 16] bytes, into the space of the weight tiles by threads [first, QL_THREADS): done
    // by the warps that have nothing to do while the layer-norm sums run.
    const int U16 = (U + 15) & ~15, ppitch = U16 + 16;
    bool proj_pending = a.proj && a.proj_staged;
    auto stage_projection = [&](int first) {
        const int piece = a.vec_p ? 16 : 4, per_row = U16 / piece, step = QL_THREADS - first;
        int j = (tid - first) / per_row, c = (tid - first) - j * per_row;
        const int dj = step / per_row, dc = step - dj * per_row;
        while (j < O) {
            if (a.vec_p) ql_copy16(tiles + j * ppitch + c * 16, p.w_proj + (long long)j * U + c * 16);
            else         *(uint32_t*)(tiles + j * ppitch + c * 4) = ql_weights4(p.w_proj + (long long)j * U, c * 4, U);
            j += dj; c += dc;
            if (c >= per_row) { c -= per_row; ++j; }
        }
        if (a.vec_p) ql_copy_commit();
    };

    // Post-processing of gates [gfirst, glast]: peephole, layer norm, activation.  `cellsrc` is the cell
    // state the peephole reads (old state for i and f, new state for o), as integer-valued floats.
    auto gate_post = [&](int gfirst, int glast, const int16_t* cell_in_global, const float* cell_smem) {
        // layer-norm weights and biases of this thread's first unit, on their way during the sums
        int16_t lw[4];
        int32_t gb[4];
        #pragma unroll
        for (int g = 0; g < 4; ++g) {
            const bool need = a.ln && g >= gfirst && g <= glast && tid < U;
            lw[g] = need ? lnw[g][tid] : (int16_t)0; gb[g] = need ? gbias[g][tid] : 0;
        }
        if (a.peephole) {
            for (int g = gfirst; g <= glast; ++g) {
                if (!peep[g]) continue;
                for (int u = tid; u < U; u += QL_THREADS) {
                    const float cv = cell_smem ? cell_smem[u] : (float)cell_in_global[(long long)b * U + u];
                    const float pv = __fmul_rn(__fmul_rn((float)peep[g][u], speep[g]), __fmul_rn(cv, sc));
                    gate(g)[u] = q16f(__fadd_rn(__fmul_rn(gate(g)[u], sint[g]), pv), sint[g], a.inv_gate[g]);
                }
            }
            __syncthreads();
        }
        if (a.ln) {
            // sequential sums, one thread (in its own warp) per gate: LstmUtils.cpp:46-53
            const int w = tid >> 5;
            if ((tid & 31) == 0 && w <= glast - gfirst) {
                const int g = gfirst + w;
                const float* v = gate(g);
                const float s = sint[g];
                float sum = 0.f, sum_sq = 0.f;
                auto add = [&](float q) {
                    const float x = __fmul_rn(q, s);
                    sum = __fadd_rn(sum, x);
                    sum_sq = __fadd_rn(sum_sq, __fmul_rn(x, x));
                };
                int i = 0;
                if ((U & 3) == 0 && U >= 8) {                // 128-bit reads, eight values ahead
                    const float4* q = (const float4*)v;
                    float4 c0 = q[0], c1 = q[1];
                    #pragma unroll 1
                    for (; i + 8 <= U; i += 8) {
                        const int next = min((i >> 2) + 2, (U >> 2) - 2);
                        const float4 n0 = q[next], n1 = q[next + 1];
                        add(c0.x); add(c0.y); add(c0.z); add(c0.w);
                        add(c1.x); add(c1.y); add(c1.z); add(c1.w);
                        c0 = n0; c1 = n1;
                    }
                }
                #pragma unroll 4
                for (; i < U; ++i) add(v[i]);
                const float fu = (float)U;
                const float mean = __fdiv_rn(sum, fu);
                const float variance = __fsub_rn(__fdiv_rn(sum_sq, fu), __fmul_rn(mean, mean));
                const float sd = variance == 0.f ? __fsqrt_rn(1e-8f) : __fsqrt_rn(variance);
                stat[g * 2] = mean;
                stat[g * 2 + 1] = __fdiv_rn(1.0f, sd);
            }
            if (w >= 4 && proj_pending) stage_projection(128);
            proj_pending = false;
            __syncthreads();
        }
        for (int u = tid; u < U; u += QL_THREADS) {
            #pragma unroll
            for (int g = 0; g < 4; ++g) {
                if (g < gfirst || g > glast) continue;
                float q = gate(g)[u];
                float s = sint[g];
                if (a.ln) {
                    if (u != tid) { lw[g] = lnw[g][u]; gb[g] = gbias[g][u]; }
                    const float sln = __fmul_rn(__fmul_rn(p.input_scale, slnw[g]), 1024.f), isln = a.inv_ln[g];
                    q = q16f(__fmul_rn(__fsub_rn(__fmul_rn(q, s), stat[g * 2]), stat[g * 2 + 1]), sln, isln);      // normalise
                    q = q16f(__fmul_rn(__fmul_rn((float)lw[g], slnw[g]), __fmul_rn(q, sln)), sln, isln);           // * weight
                    q = q16f(__fadd_rn(__fmul_rn(q, sln), __fmul_rn(__int2float_rn(gb[g]), sgb[g])), 1.f / 4096, 4096.f);        // + bias
                    s = 1.f / 4096;
                }
                const float v = __fmul_rn(q, s);
                const float r = g == 2 ? tanhf(v) : __fdiv_rn(1.f, __fadd_rn(1.f, expf(-v)));
                gate(g)[u] = q16f(r, sc, isc);
            }
        }
        __syncthreads();
    };

    // (without peephole the output gate does not see the new cell state: all gates at once)
    gate_post(g0, a.peephole ? 2 : 3, p.cell_state_in, nullptr);

    // ---- cell state: c = Q(f * c_in); c = Q(c + g * i)  (or g * Q(1 - f) with CIFG); clip
    for (int u = tid; u < U; u += QL_THREADS) {
        const float cin = __fmul_rn((float)p.cell_state_in[(long long)b * U + u], sc);
        const float f = gate(1)[u];
        float c = q16f(__fmul_rn(__fmul_rn(f, sc), cin), sc, isc);
        const float ig = a.cifg ? q16f(__fsub_rn(1.0f, __fmul_rn(f, sc)), sc, isc) : gate(0)[u];
        c = q16f(__fadd_rn(__fmul_rn(c, sc), __fmul_rn(__fmul_rn(gate(2)[u], sc), __fmul_rn(ig, sc))), sc, isc);
        if (p.cell_clip > 0.0f) {
            const float fv = __fmul_rn(c, sc);
            float r = (p.cell_clip < fv) ? p.cell_clip : fv;
            r = (-p.cell_clip > r) ? -p.cell_clip : r;
            c = q16f(r, sc, isc);
        }
        cell[u] = c;
        p.cell_state_out[(long long)b * U + u] = (int16_t)c;
    }
    __syncthreads();

    if (a.peephole) gate_post(3, 3, nullptr, cell);

    // ---- hidden = Q8(o * Q16(tanh(c))), its projection factors and magnitudes
    const float hzp = (float)p.hidden_state_zp, cp = a.proj ? __fdiv_rn(p.s_proj, p.output_scale) : 0.f;
    for (int u = tid; (u & ~31) < U16; u += QL_THREADS) {
        float h = 0.f;
        int mag = 0;
        if (u < U) {
            const float t = q16f(tanhf(__fmul_rn(cell[u], sc)), sc, isc);
            const float hv = __fmul_rn(__fmul_rn(gate(3)[u], sc), __fmul_rn(t, sc));
            const float hq = fminf(fmaxf(__fadd_rn(hzp, roundf(__fdiv_rn(hv, p.hidden_state_scale))), -128.f), 127.f);
            const float d = __fsub_rn(hq, hzp);
            h = __fmul_rn(d, p.hidden_state_scale);          // dequantised hidden state
            mag = (int)fabsf(d);
        }
        const float f = __fmul_rn(h, cp);
        const QlBlockInfo info = ql_block_info(fabsf(f), s_danger[2][0], mag, a.exact_only);
        if (u < U16) {
            hid[u] = h;
            hc[u] = make_float2(f, f);
            if ((u & 15) == 0) { hbounds[u / QL_BLOCK] = info.bounds; hlisted[u / QL_BLOCK] = info.listed; }
        }
    }

    // ---- projection (int16 accumulator at the OUTPUT's scale and offset) and outputs
    if (proj_pending) stage_projection(0);
    const float so = p.output_scale, zo = (float)p.output_zp;
    auto finish = [&](int j, float acc) {                    // acc: int16 accumulator of output j (projection), or unused
        float out8;
        if (a.proj) {
            out8 = fminf(fmaxf(__fadd_rn(zo, roundf(__fdiv_rn(__fmul_rn(__fsub_rn(acc, zo), so), so))), -128.f), 127.f);
            if (p.projection_clip > 0.0f) {
                const float fv = __fmul_rn(__fsub_rn(out8, zo), so);
                float r = (p.projection_clip < fv) ? p.projection_clip : fv;
                r = (-p.projection_clip > r) ? -p.projection_clip : r;
                out8 = fminf(fmaxf(__fadd_rn(zo, roundf(__fdiv_rn(r, so))), -128.f), 127.f);
            }
        } else {
            out8 = fminf(fmaxf(__fadd_rn(zo, roundf(__fdiv_rn(hid[j], so))), -128.f), 127.f);
        }
        p.output[(long long)b * O + j] = (int8_t)out8;
        const float ov = __fmul_rn(__fsub_rn(out8, zo), so);
        const float hs = fminf(fmaxf(__fadd_rn((float)p.output_state_zp, roundf(__fdiv_rn(ov, p.output_state_scale))), -128.f), 127.f);
        p.output_state_out[(long long)b * O + j] = (int8_t)hs;
    };
    if (!a.proj) {
        __syncthreads();
        for (int j = tid; j < O; j += QL_THREADS) finish(j, 0.f);
        return;
    }
    if (tid == 0) s_exact[0][0].set(so, so, a.inv_out, a.inv_out, p.s_proj, p.s_proj, -32768.f - zo, 32767.f - zo);
    if (a.proj_staged && a.vec_p) ql_copy_wait<0>();
    __syncthreads();
    // two outputs, half of them apart, per thread; the chains run on acc - zo, an integer like the gates' accumulators
    const int O2 = (O + 1) / 2;
    for (int j0 = tid; (j0 & ~31) < O2; j0 += QL_THREADS) {
        const int j = min(j0, O2 - 1), j1 = min(j + O2, O - 1);      // (idle lanes repeat the last pair)
        const int8_t* w[2] = {p.w_proj + (long long)j * U, p.w_proj + (long long)j1 * U};
        float first[2] = {0.f, 0.f};                         // the int16 buffer starts as raw zeros
        if (p.b_proj) {
            first[0] = q16zf(__fmul_rn(__int2float_rn(p.b_proj[j]), p.s_bproj), so, zo);
            first[1] = q16zf(__fmul_rn(__int2float_rn(p.b_proj[j1]), p.s_bproj), so, zo);
        }
        QlChains ch[1];
        QlNote notes[QL_NOTES];
        ch[0].T = pack2(QL_MAGIC + (first[0] - zo), QL_MAGIC + (first[1] - zo));
        ch[0].notes = 0; ch[0].note = notes;
        QlSource from[1];
        from[0].xc = hc; from[0].xf = hid; from[0].bounds = hbounds; from[0].listed = hlisted; from[0].e = &s_exact[0][0];
        from[0].wa = a.proj_staged ? (const int8_t*)tiles + j * ppitch : w[0];
        from[0].wb = a.proj_staged ? (const int8_t*)tiles + j1 * ppitch : w[1];
        from[0].first = 0; from[0].K = U; from[0].aligned = a.proj_staged;
        uint4 na = from[0].weights16(from[0].wa, 0), nb = from[0].weights16(from[0].wb, 0);
        #pragma unroll 1
        for (int k = 0; k < U16; k += QL_BLOCK) {
            const uint32_t ma[4] = {na.x ^ 0x80808080u, na.y ^ 0x80808080u, na.z ^ 0x80808080u, na.w ^ 0x80808080u};
            const uint32_t mb[4] = {nb.x ^ 0x80808080u, nb.y ^ 0x80808080u, nb.z ^ 0x80808080u, nb.w ^ 0x80808080u};
            if (k + QL_BLOCK < U16) { na = from[0].weights16(from[0].wa, k + QL_BLOCK); nb = from[0].weights16(from[0].wb, k + QL_BLOCK); }
            ql_block<1>(ch, ma, mb, k, from);
        }
        float f0, f1;
        unpack2(sub2(ql_resolve(ch[0].T, ch[0].notes, ch[0].note, from[0].xc, from[0].xf, from[0].bounds, from[0].e), pack2(QL_MAGIC, QL_MAGIC)), f0, f1);
        if (j0 < O2) {
            finish(j, f0 + zo);
            if (j + O2 < O) finish(j + O2, f1 + zo);
        }
    }
}

// ---- host: which input magnitudes need the reference's arithmetic ----------------------------------------------------------

// For one gate: r = |w| mag c over all weight magnitudes.  r less its nearest integer through 1.5 * 2^52 (where that stops
// being exact, from 2^51 on, the bound has long exceeded a half): 33 000 steps that vectorise, 45 us on a host core against
// 130 with a conversion to an integer.
static void ql_list_magnitudes(float sx, float sw, float sG, uint32_t* bits)
{
    const double c = (double)sx * (double)sw / (double)sG, unit = 1.0 / 16777216.0, magic = 6755399441055744.0;
    for (int mag = 1; mag < 256; ++mag) {
        int near = 0;
        for (int w = 0; w <= 128; ++w) {
            const double r = (double)(w * mag) * c, t = r - ((r + magic) - magic);
            near |= 0.5 - fabs(t) <= (8.0 * r + 8.0 + 3.0 * QL_LEVEL) * unit;
        }
        if (near) bits[mag >> 5] |= 1u << (mag & 31);
    }
}

// The scales of a layer that its plan depends on, gates i, f, c, o in turn (CIFG: the input gate's chains are repeats of the
// forget gate's).
static void ql_plan_scales(const b200k_qlstm_params* p, float* s)
{
    const bool cifg = p->w_i2i == nullptr;
    const float all[17] = {p->input_scale, p->output_state_scale, p->hidden_state_scale, p->output_scale, p->w_proj ? p->s_proj : 1.f,
                           cifg ? p->s_i2f : p->s_i2i, p->s_i2f, p->s_i2c, p->s_i2o, cifg ? p->s_r2f : p->s_r2i, p->s_r2f, p->s_r2c, p->s_r2o,
                           cifg ? p->forget_intermediate_scale : p->input_intermediate_scale, p->forget_intermediate_scale,
                           p->cell_intermediate_scale, p->output_intermediate_scale};
    memcpy(s, all, sizeof(all));
}
// scales that the error bound holds for
static bool ql_plan_ordinary(const b200k_qlstm_plan& plan)
{
    for (float s : plan.scales)
        if (!(s >= 1e-8f && s <= 1e8f)) return false;
    return true;
}
static void ql_make_plan(b200k_qlstm_plan& plan)             // from its scales
{
    memset(plan.magnitudes, 0, sizeof(plan.magnitudes));
    if (!ql_plan_ordinary(plan)) return;
    const float *s = plan.scales, *si = s + 5, *sr = s + 9, *sint = s + 13;
    for (int g = 0; g < 4; ++g) {
        ql_list_magnitudes(s[0], si[g], sint[g], plan.magnitudes[0][g & 1]);
        ql_list_magnitudes(s[1], sr[g], sint[g], plan.magnitudes[1][g & 1]);
    }
    ql_list_magnitudes(s[2], s[4], s[3], plan.magnitudes[2][0]);
}

// The plans made last (a bounded table: the oldest makes room): a network that is loaded again, or several times, does not make
// them again, and layers that are stepped without a plan of their own have theirs here.
static b200k_qlstm_plan ql_plan_for(const float* scales)
{
    static b200k_qlstm_plan table[256];
    static int used = 0, next = 0;
    static std::mutex guard;
    {
        std::lock_guard<std::mutex> lock(guard);
        for (int i = 0; i < used; ++i)
            if (memcmp(table[i].scales, scales, sizeof(table[i].scales)) == 0) return table[i];
    }
    b200k_qlstm_plan plan;
    memcpy(plan.scales, scales, sizeof(plan.scales));
    ql_make_plan(plan);
    std::lock_guard<std::mutex> lock(guard);
    table[next] = plan;
    next = (next + 1) & 255;
    if (used < 256) ++used;
    return plan;
}

}  // namespace b200k

using namespace b200k;

extern "C" int b200k_qlstm_prepare(const b200k_qlstm_params* p, b200k_qlstm_plan* plan)
{
    B200K_REQUIRE(p && plan, B200K_E_INVALID, "qlstm_prepare: null params or plan");
    float scales[17];
    ql_plan_scales(p, scales);
    *plan = ql_plan_for(scales);
    return B200K_OK;
}

extern "C" int b200k_qlstm_step(const b200k_qlstm_params* p, void* stream)
{
    B200K_REQUIRE(p, B200K_E_INVALID, "qlstm_step: null params");
    B200K_REQUIRE(p->batch > 0 && p->input_size > 0 && p->num_units > 0 && p->output_size > 0, B200K_E_INVALID,
                  "qlstm_step: bad shape");
    B200K_REQUIRE(p->input && p->output_state_in && p->cell_state_in && p->output_state_out && p->cell_state_out &&
                  p->output, B200K_E_INVALID, "qlstm_step: null state/input/output pointer");
    B200K_REQUIRE(p->w_i2f && p->w_i2c && p->w_i2o && p->w_r2f && p->w_r2c && p->w_r2o, B200K_E_INVALID,
                  "qlstm_step: missing mandatory weights");
    QlArgs a;
    a.p = *p;
    a.cifg = p->w_i2i == nullptr;
    a.peephole = p->w_c2f != nullptr;
    a.ln = p->ln_f != nullptr;
    a.proj = p->w_proj != nullptr;
    B200K_REQUIRE(a.cifg || p->w_r2i, B200K_E_INVALID, "qlstm_step: input-to-input weights without recurrent-to-input weights");
    B200K_REQUIRE(!a.peephole || (p->w_c2o && (a.cifg || p->w_c2i)), B200K_E_INVALID, "qlstm_step: incomplete peephole weights");
    B200K_REQUIRE(!a.ln || (p->ln_c && p->ln_o && (a.cifg || p->ln_i) && p->b_f && p->b_c && p->b_o && (a.cifg || p->b_i)),
                  B200K_E_INVALID, "qlstm_step: layer norm needs all layer-norm weights and gate biases");
    B200K_REQUIRE(a.proj || p->num_units == p->output_size, B200K_E_INVALID,
                  "qlstm_step: without projection the output size must equal the number of units");
    float scales[17];
    ql_plan_scales(p, scales);
    const bool own = p->plan && memcmp(p->plan->scales, scales, sizeof(scales)) == 0;
    const b200k_qlstm_plan plan = own ? *p->plan : ql_plan_for(scales);
    auto byte = [](int z) { return z >= -128 && z <= 127; };
    a.exact_only = !byte(p->input_zp) || !byte(p->output_state_zp) || !byte(p->output_zp) || !byte(p->hidden_state_zp) || !ql_plan_ordinary(plan);
    static_assert(sizeof(a.danger) == sizeof(plan.magnitudes), "a plan holds what the kernel reads");
    memcpy(a.danger, plan.magnitudes, sizeof(a.danger));
    const float ln[4] = {p->s_lni, p->s_lnf, p->s_lnc, p->s_lno};
    for (int g = 0; g < 4; ++g) {
        a.inv_gate[g] = rn_reciprocal(scales[13 + g]);
        a.inv_ln[g] = rn_reciprocal(p->input_scale * ln[g] * 1024.f);
    }
    a.inv_cell = rn_reciprocal(p->cell_state_scale);
    a.inv_out = rn_reciprocal(p->output_scale);
    auto aligned = [](const void* q) { return ((uintptr_t)q & 15) == 0; };
    a.vec_i = p->input_size % 16 == 0 && aligned(p->w_i2i) && aligned(p->w_i2f) && aligned(p->w_i2c) && aligned(p->w_i2o);
    a.vec_o = p->output_size % 16 == 0 && aligned(p->w_r2i) && aligned(p->w_r2f) && aligned(p->w_r2c) && aligned(p->w_r2o);
    a.vec_p = p->num_units % 16 == 0 && aligned(p->w_proj);
    cudaStream_t s = (cudaStream_t)stream;
    const int sms = sm_count();
    // Two rows per pair of CTAs (each weight converted once for both) as soon as that fills most SMs; below, the units of one
    // row are spread over up to eight CTAs, so that a small batch still uses the machine.
    int rows = 1, cs = 1;
    if (p->batch >= 2 && p->batch * 5ll >= sms * 3ll) { rows = 2; cs = 2; }
    else while (cs < 8 && p->batch * cs * 2 <= sms + sms / 4 && p->num_units >= 32 * cs) cs *= 2;
    // Shared memory: the gates; the staged factors, or what comes after the chains; the weight tiles, or the projection
    // matrix.  Very large layers make do with fewer staged steps and one tile.
    auto up16 = [](int v) { return (v + 15) & ~15; };
    const size_t limit = 226 * 1024, U = (size_t)p->num_units;
    const size_t gates = 4 * ((4 * U + QL_GATE_SLACK + 3) & ~(size_t)3), after = 8 * U + 32 + 64;      // (64: padding)
    const int wanted = up16(p->input_size) + up16(p->output_size);
    a.seg = wanted < QL_SEG ? wanted : QL_SEG;
    a.nbuf = 2;
    size_t smem;
    for (;;) {
        const size_t staged = (size_t)rows * a.seg * (2 * 8 + 4) + (size_t)rows * 2 * (a.seg / QL_BLOCK) * (8 + 1);
        a.tile_off = (unsigned)((gates + staged + 15) & ~(size_t)15);
        smem = a.tile_off + (size_t)a.nbuf * QL_TILE_BYTES;
        if (smem < gates + after) smem = gates + after;
        if (smem <= limit) break;
        if (a.nbuf == 2) a.nbuf = 1;
        else if (a.seg > 128) a.seg = a.seg / 2 > 128 ? up16(a.seg / 2) : 128;
        else if (rows == 2) rows = cs = 1;
        else break;
    }
    B200K_REQUIRE(smem <= limit, B200K_E_TOOBIG, "qlstm_step: layer too large for the shared-memory resident kernel");
    a.both = a.seg >= wanted;
    // The projection matrix takes the tiles' place if the steps before it, whose data begin where the staged factors were,
    // end before the tiles do (moved back if they need to be).
    const size_t behind = (gates + after + 15) & ~(size_t)15;
    if (a.proj && behind > a.tile_off && behind + (size_t)a.nbuf * QL_TILE_BYTES <= limit) {
        a.tile_off = (unsigned)behind;
        smem = a.tile_off + (size_t)a.nbuf * QL_TILE_BYTES;
    }
    const size_t whole = a.tile_off + (size_t)p->output_size * (up16(p->num_units) + 16);
    a.proj_staged = a.proj && a.tile_off >= behind && whole <= limit;
    if (a.proj_staged && whole > smem) smem = whole;
    auto launch = [&](auto tag) -> int {
        if (const int rc = allow_shared<decltype(tag)::kernel>(smem)) return rc;
        launch_pdl_cluster(tag.kernel, dim3((unsigned)((p->batch + rows - 1) / rows * cs)), dim3(QL_THREADS), smem, s, (unsigned)cs, a);
        return check_launch("qlstm_step_kernel");
    };
    return rows == 2 ? launch(KernelTag<qlstm_step_kernel<2>>()) : launch(KernelTag<qlstm_step_kernel<1>>());
}
