// The "prepare" stage for a warp that shares its SM with the walk of the chunks: one warp turns one (chunk, head) of q, k, g,
// beta into the chunk operands kd, qd, kr, E_tot, INV, Mqk, built in place in ONE record-shaped block of shared memory (layout
// of fkda_common.cuh).  Numerics: tests/torch_ref.py:153-229 of the reference.
//
// Lane c + 16 hh owns columns 8c .. 8c+7 of rows 8 hh .. 8 hh + 7:
//   * a lane's piece of a row is one 16-byte load (a warp instruction covers two whole 256-byte rows), and it is one row of an
//     8 x 8 core matrix of the record; with the padded strides all accesses are free of bank conflicts.  Rows are loaded two
//     ahead of their use.  (Copying the pieces straight to their places with cp.async took 40 % longer: such scattered
//     16-byte writes pass at one per cycle.)
//   * a row norm is a chain of eight FMAs in the lane and four butterfly steps over the 16 lanes of a row, the contract's
//     summation order; the first step also splits the work, eight lanes going on with q and eight with k;
//   * the gate's running sum over the rows is sequential: rows 8-15 start from the sum of rows 0-7, which every warp forms
//     first, four columns per lane.  Those gates are formed a second time with their rows: keeping them takes 64
//     registers and unrolled loops, and the code of unrolled loops did not stay in the instruction cache beside the
//     walking warps' (every second instruction waited for its fetch: 1.42 ms against 0.58 for 96 chains of 512 chunks);
//   * two columns share an instruction where the arithmetic is fp32 (packed f32x2, each half rounded as the scalar
//     instruction).
// The 16x16x128 products and the fp16 inverse run on mma.sync fragments.
#pragma once

#include "fkda_common.cuh"
#include "fkda_internal.h"
#include "fkda_sm100.cuh"

namespace fkda {

// Packed pairs of fp32 values.
typedef unsigned long long f2_t;
__device__ __forceinline__ f2_t f2_pack(float lo, float hi) {
    f2_t r;
    asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2_t x, float& lo, float& hi) { asm("mov.b64 {%0,%1}, %2;" : "=f"(lo), "=f"(hi) : "l"(x)); }
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) {
    f2_t r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2_t f2_mul(f2_t a, f2_t b) {
    f2_t r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2_t f2_add(f2_t a, f2_t b) {
    f2_t r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2_t f2_of_bf2(uint32_t x) { return f2_pack(bf_lo(x), bf_hi(x)); }
__device__ __forceinline__ uint32_t bf2_of_f2(f2_t x) {
    float lo, hi;
    f2_unpack(x, lo, hi);
    return pack_bf2(lo, hi);
}

constexpr int kPrepKiLbo = 272;   // ki tile: K-major core matrices, 16-byte K chunks 272 bytes apart (256 + 16 padding)
static_assert(16 * kPrepKiLbo <= kTcKrBytes, "the ki tile fits the KR part of the record");
static_assert(kChunk * sizeof(float) <= 512, "sigmoid(beta) in fp32 fits the INV part until the inverse is written");

// What a warp asks for before it starts on a unit: the gates of rows 0-7 (4 columns per lane, for the sum that rows 8-15 start
// from), the first two rows of my half, and the unit's scalars.
struct PrepRow {
    uint4 q, k, g;        // columns 8c .. 8c+7
};
struct PrepHead {
    uint2 g7[8];          // g of rows 0 .. 7, columns 4 lane .. 4 lane + 3
    PrepRow row[2];
    float4 dt0, dt1;      // dt_bias of my 8 columns
    float4 dt7;           // dt_bias of columns 4 lane ..
    float a_log;
    __nv_bfloat16 beta;   // logit of row `lane` (lanes below 16; 0 past the end, as zero padding does)
};
// Where a unit's rows are: the lane's columns of its first row in each tensor.
struct PrepSrc {
    const uint4 *q, *k, *g;
    uint32_t step;        // 16-byte pieces between rows
    int row0, last;       // my first row, the unit's last row
};
__device__ __forceinline__ PrepSrc prep_src(const TwoPassArgs& a, int64_t t0, int len, int h, int lane) {
    const int64_t off = t0 * a.token_stride + (int64_t)h * kD + 8 * (lane & 15);
    return PrepSrc{reinterpret_cast<const uint4*>(a.q + off), reinterpret_cast<const uint4*>(a.k + off),
                   reinterpret_cast<const uint4*>(a.g + off), (uint32_t)(a.token_stride >> 3), 8 * (lane >> 4), len - 1};
}
// Row i of my half; a row past the end reads the last valid row (its factors are zero).
__device__ __forceinline__ void prep_load_row(const PrepSrc& s, int i, PrepRow& x) {
    const uint64_t off = (uint64_t)(uint32_t)min(s.row0 + i, s.last) * s.step;
    x.k = s.k[off];
    x.q = s.q[off];
    x.g = s.g[off];
}
__device__ __forceinline__ void prep_load(const TwoPassArgs& a, const PrepSrc& s, int64_t t0, int len, int h, int lane, PrepHead& x) {
    const uint2* g = reinterpret_cast<const uint2*>(a.g + t0 * a.token_stride + (int64_t)h * kD + 4 * lane);
#pragma unroll
    for (int i = 0; i < 8; ++i) x.g7[i] = g[(uint64_t)(uint32_t)min(i, s.last) * (2 * s.step)];
#pragma unroll
    for (int i = 0; i < 2; ++i) prep_load_row(s, i, x.row[i]);
    const float4* dt = reinterpret_cast<const float4*>(a.dt_bias + (int64_t)h * kD);
    x.dt0 = dt[2 * (lane & 15)];
    x.dt1 = dt[2 * (lane & 15) + 1];
    x.dt7 = dt[lane];
    x.a_log = a.A_log[h];
    x.beta = __float2bfloat16_rn(0.0f);
    if (lane < len) x.beta = a.beta[(t0 + lane) * a.beta_token_stride + h];   // len <= 16
}

__device__ __forceinline__ uint4 prep_lds(uint32_t addr) {
    uint4 x;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(addr) : "memory");
    return x;
}
__device__ __forceinline__ void prep_sts(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// 1 / norm of one row of q and of k from my partial sums of squares, over the 16 lanes of the row.
__device__ __forceinline__ void prep_row_norms(float q, float k, int lane, float* qi, float* ki) {
    const bool up = (lane & 8) != 0;
    float v = __fadd_rn(up ? k : q, __shfl_xor_sync(0xffffffffu, up ? q : k, 8));
#pragma unroll
    for (int off = 4; off >= 1; off >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, off));
    v = rsqrt_approx(__fadd_rn(v, 1e-6f));
    const float o = __shfl_xor_sync(0xffffffffu, v, 8);
    *qi = up ? o : v;
    *ki = up ? v : o;
}

// 1 / norm of two rows of q and of k from my partial sums of squares, over the 16 lanes of a row.  The first two butterfly steps
// also split the four sums among the lanes of a row (the sums are those of a plain butterfly: every step adds the same two
// numbers, whichever lane keeps the result).
__device__ __forceinline__ void prep_two_norms(const float (&q)[2], const float (&k)[2], int lane, float (&qi)[2], float (&ki)[2]) {
    const bool up = (lane & 8) != 0, second = (lane & 4) != 0;
    const float r0 = __shfl_xor_sync(0xffffffffu, up ? q[0] : k[0], 8), r1 = __shfl_xor_sync(0xffffffffu, up ? q[1] : k[1], 8);
    const float v0 = __fadd_rn(up ? k[0] : q[0], r0), v1 = __fadd_rn(up ? k[1] : q[1], r1);
    float v = __fadd_rn(second ? v1 : v0, __shfl_xor_sync(0xffffffffu, second ? v0 : v1, 4));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
    v = rsqrt_approx(__fadd_rn(v, 1e-6f));
    const float w = __shfl_xor_sync(0xffffffffu, v, 4);   // my tensor's other row
    const float m0 = second ? w : v, m1 = second ? v : w;
    const float o0 = __shfl_xor_sync(0xffffffffu, m0, 8), o1 = __shfl_xor_sync(0xffffffffu, m1, 8);
    qi[0] = up ? o0 : m0;
    qi[1] = up ? o1 : m1;
    ki[0] = up ? m0 : o0;
    ki[1] = up ? m1 : o1;
}

// gate_scale * sigmoid(exp(A_log) * (g + dt_bias)) of two columns, added to their running sum.  sigmoid(x) = tanh(x/2)/2 + 1/2;
// the halving of x is exact and folded into the factor `ae`.  (The last product is scalar: a packed one followed by the packed
// sum is contracted into one FMA and loses a rounding.)
__device__ __forceinline__ f2_t prep_add_gate(f2_t run, uint32_t g, f2_t dt, f2_t ae, float gs) {
    const f2_t half2 = f2_pack(0.5f, 0.5f);
    float x0, x1, y0, y1;
    f2_unpack(f2_mul(ae, f2_add(f2_of_bf2(g), dt)), x0, x1);
    f2_unpack(f2_fma(f2_pack(tanh_approx(x0), tanh_approx(x1)), half2, half2), y0, y1);
    return f2_add(run, f2_pack(__fmul_rn(gs, y0), __fmul_rn(gs, y1)));
}

// One warp, one unit of `len` tokens (asked for with prep_load): fills the record block.  `acquire()` is called before the first
// write to the block, after work that needs none: it returns whether the block may be written.  `next()` is called when the
// unit's inputs are used up, before the products: it may load the next unit's head into `x`.
// kFewRows: units of 8 tokens or fewer are common, their missing rows are skipped (the code for it costs the others 2 %, and
// the walking warps beside them in fkda_fused.cuh 20 % in registers).
// kPaired: the norms of two rows are formed side by side.  A row's norm is a chain of latencies (eight products, five shuffles, the
// reciprocal root), and the shuffles of a row wait behind the stores of the row before it.  It pays in the kernel that only prepares
// (8 192 tokens, 32 heads, whole forward 275 -> 266 us; 1 000 tokens 47.3 -> 45.1); beside walking warps its registers cost more
// (fkda_short.cu: 512 x 16 tokens, 64 heads 489 -> 551 us; fkda_fused.cuh: 3 to 7 % slower).
template <bool kFewRows, bool kPaired, class Acquire, class Next>
__device__ __forceinline__ bool prep_compute(const TwoPassArgs& a, const PrepSrc& src, int len, uint8_t* rec_ptr, int lane, PrepHead& x,
                                             Acquire&& acquire, Next&& next) {
    const uint32_t rec = sm100::smem_u32(rec_ptr);
    const int c = lane & 15, hh = lane >> 4;
    const uint32_t b1 = rec + kTcB1 + c * kTcB1Lbo + hh * 128, kip = rec + kTcKr + c * kPrepKiLbo + hh * 128;
    float* beta_act = reinterpret_cast<float*>(rec_ptr + kTcInv);
    const float a_exp_half = __fmul_rn(ex2_approx(__fmul_rn(x.a_log, 1.4426950408889634f)), 0.5f);
    const f2_t ae = f2_pack(a_exp_half, a_exp_half);
    // ---- the gate sum over rows 0-7, from which the lanes of rows 8-15 go on: 4 columns per lane ----
    f2_t run[4];
    {
        f2_t r0 = f2_pack(0.0f, 0.0f), r1 = r0;
        const f2_t d0 = f2_pack(x.dt7.x, x.dt7.y), d1 = f2_pack(x.dt7.z, x.dt7.w);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float gs = i < len ? a.gate_scale : 0.0f;
            r0 = prep_add_gate(r0, x.g7[i].x, d0, ae, gs);
            r1 = prep_add_gate(r1, x.g7[i].y, d1, ae, gs);
        }
        float s[4];
        f2_unpack(r0, s[0], s[1]);
        f2_unpack(r1, s[2], s[3]);
#pragma unroll
        for (int p = 0; p < 4; ++p) {   // my columns 8c + 2p, + 1 are with lane 2c + p / 2
            const float y0 = __shfl_sync(0xffffffffu, s[2 * (p & 1)], 2 * c + (p >> 1)), y1 = __shfl_sync(0xffffffffu, s[2 * (p & 1) + 1], 2 * c + (p >> 1));
            run[p] = f2_pack(hh ? y0 : 0.0f, hh ? y1 : 0.0f);
        }
    }
    if (!acquire()) return false;
    if (lane < kChunk) {   // sigmoid(beta) of row `lane`
        const float sb = sigmoid_tanh(bf2f(x.beta));
        beta_act[lane] = sb;
        reinterpret_cast<__nv_bfloat16*>(rec_ptr + kTcBeta)[lane] = f2bf(sb);
    }
    // ---- rows: kd, qd, ki; one bf16 rounding per element and operation ----
    const f2_t dt[4] = {f2_pack(x.dt0.x, x.dt0.y), f2_pack(x.dt0.z, x.dt0.w), f2_pack(x.dt1.x, x.dt1.y), f2_pack(x.dt1.z, x.dt1.w)};
    const uint32_t sc2 = pack_bf2(a.scale, a.scale);
    const int rows = !kFewRows || len > 8 ? 8 : (len + 1) & ~1;   // rows of each half that are gone through
#pragma unroll 1
    for (int ib = 0; ib < rows; ib += 2) {
        float q_norm[2], k_norm[2];
        if constexpr (kPaired) {
            float qs[2] = {0.0f, 0.0f}, ks[2] = {0.0f, 0.0f};
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t k = (&x.row[u].k.x)[p], q = (&x.row[u].q.x)[p];
                    qs[u] = __fmaf_rn(bf_lo(q), bf_lo(q), qs[u]);
                    ks[u] = __fmaf_rn(bf_lo(k), bf_lo(k), ks[u]);
                    qs[u] = __fmaf_rn(bf_hi(q), bf_hi(q), qs[u]);
                    ks[u] = __fmaf_rn(bf_hi(k), bf_hi(k), ks[u]);
                }
            prep_two_norms(qs, ks, lane, q_norm, k_norm);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = ib + u;
            const bool valid = 8 * hh + i < len;
            const uint32_t kk[4] = {x.row[u].k.x, x.row[u].k.y, x.row[u].k.z, x.row[u].k.w};
            const uint32_t qq[4] = {x.row[u].q.x, x.row[u].q.y, x.row[u].q.z, x.row[u].q.w};
            const uint32_t gg[4] = {x.row[u].g.x, x.row[u].g.y, x.row[u].g.z, x.row[u].g.w};
            if (ib < 6) prep_load_row(src, i + 2, x.row[u]);   // two rows ahead of their use
            float qi, kj;
            if constexpr (kPaired) {
                qi = q_norm[u];
                kj = k_norm[u];
            } else {
                float qs = 0.0f, ks = 0.0f;
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    qs = __fmaf_rn(bf_lo(qq[p]), bf_lo(qq[p]), qs);
                    ks = __fmaf_rn(bf_lo(kk[p]), bf_lo(kk[p]), ks);
                    qs = __fmaf_rn(bf_hi(qq[p]), bf_hi(qq[p]), qs);
                    ks = __fmaf_rn(bf_hi(kk[p]), bf_hi(kk[p]), ks);
                }
                prep_row_norms(qs, ks, lane, &qi, &kj);
            }
            qi = valid ? qi : 0.0f;
            kj = valid ? kj : 0.0f;
            const float gs = valid ? a.gate_scale : 0.0f;
            const f2_t qi2 = f2_pack(qi, qi), ki2 = f2_pack(kj, kj);
            uint32_t kd[4], qd[4], ki[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                run[p] = prep_add_gate(run[p], gg[p], dt[p], ae, gs);
                float s0, s1;
                f2_unpack(run[p], s0, s1);
                const uint32_t ep = pack_bf2(ex2_approx(s0), ex2_approx(s1)), em = pack_bf2(ex2_approx(-s0), ex2_approx(-s1));
                const uint32_t kn = bf2_of_f2(f2_mul(f2_of_bf2(kk[p]), ki2)), qn = bf2_of_f2(f2_mul(f2_of_bf2(qq[p]), qi2));
                kd[p] = bf2_mul(kn, ep);
                qd[p] = bf2_mul(bf2_mul(qn, ep), sc2);
                ki[p] = bf2_mul(kn, em);
            }
            prep_sts(b1 + 16 * i, kd[0], kd[1], kd[2], kd[3]);
            prep_sts(b1 + 256 + 16 * i, qd[0], qd[1], qd[2], qd[3]);   // rows 16..31 = two row groups further
            prep_sts(kip + 16 * i, ki[0], ki[1], ki[2], ki[3]);
        }
    }
    if constexpr (kFewRows) {
#pragma unroll 1
        for (int i = rows; i < 8; ++i) {   // the other rows are zeros
            prep_sts(b1 + 16 * i, 0u, 0u, 0u, 0u);
            prep_sts(b1 + 256 + 16 * i, 0u, 0u, 0u, 0u);
            prep_sts(kip + 16 * i, 0u, 0u, 0u, 0u);
        }
    }
    // E_tot = 2^(sum over all rows): known to the lanes of rows 8-15; as bf16 also to the others, for kr
    uint32_t etb[4];
    {
        float et[8];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            float s0, s1;
            f2_unpack(run[p], s0, s1);
            et[2 * p] = ex2_approx(s0);
            et[2 * p + 1] = ex2_approx(s1);
            etb[p] = __shfl_sync(0xffffffffu, pack_bf2(et[2 * p], et[2 * p + 1]), c + 16);
        }
        if (hh) {
            float4* dst = reinterpret_cast<float4*>(rec_ptr + kTcEt) + 2 * c;
            dst[0] = make_float4(et[0], et[1], et[2], et[3]);
            dst[1] = make_float4(et[4], et[5], et[6], et[7]);
        }
    }
    __syncwarp();
    next();
    // ---- L = fp16(kd ki^T) masked * fp16(beta), Mqk = bf16(qd ki^T) masked ----
    Frag16 lfrag;  // L as the A / C fragment the inverse starts from
    {
        const int g = lane >> 2, t = lane & 3;
        float l0[4] = {0.f, 0.f, 0.f, 0.f}, l1[4] = {0.f, 0.f, 0.f, 0.f};
        float m0[4] = {0.f, 0.f, 0.f, 0.f}, m1[4] = {0.f, 0.f, 0.f, 0.f};
        // lane 8m + r addresses row r of the m-th 8x8 matrix of a fragment: matrix m of an A fragment is (row group
        // m & 1, K chunk m >> 1), matrix m of the B pair is (K chunk m & 1, row group m >> 1); rows are 16 bytes
        const int lr = lane & 7, lm = lane >> 3;
        const uint8_t* a_row = rec_ptr + kTcB1 + (lm >> 1) * kTcB1Lbo + (lm & 1) * 128 + lr * 16;
        const uint8_t* b_row = rec_ptr + kTcKr + (lm & 1) * kPrepKiLbo + (lm >> 1) * 128 + lr * 16;
#pragma unroll
        for (int j = 0; j < kD / 16; ++j) {
            uint32_t b00, b01, b10, b11, a0, a1, a2, a3, q0, q1, q2, q3;
            ldmatrix_x4(b00, b01, b10, b11, b_row + 2 * j * kPrepKiLbo);
            ldmatrix_x4(a0, a1, a2, a3, a_row + 2 * j * kTcB1Lbo);
            ldmatrix_x4(q0, q1, q2, q3, a_row + 2 * j * kTcB1Lbo + 256);  // qd = rows 16..31
            mma_bf16_f32acc(l0, a0, a1, a2, a3, b00, b01);  // columns 0-7
            mma_bf16_f32acc(l1, a0, a1, a2, a3, b10, b11);  // columns 8-15
            mma_bf16_f32acc(m0, q0, q1, q2, q3, b00, b01);
            mma_bf16_f32acc(m1, q0, q1, q2, q3, b10, b11);
        }
        __half bh[2];
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) bh[hr] = __float2half_rn(beta_act[g + 8 * hr]);
        // fragment element e of n-tile nt: row = g + 8*(e>>1), column = 8*nt + 2*t + (e&1)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                const int i = g + 8 * hr, j = 8 * nt + 2 * t;
                const float x0 = nt ? l1[2 * hr] : l0[2 * hr], x1 = nt ? l1[2 * hr + 1] : l0[2 * hr + 1];
                const float y0 = nt ? m1[2 * hr] : m0[2 * hr], y1 = nt ? m1[2 * hr + 1] : m0[2 * hr + 1];
                const __half h0 = (i > j) ? __hmul(__float2half_rn(x0), bh[hr]) : __float2half_rn(0.0f);
                const __half h1 = (i > j + 1) ? __hmul(__float2half_rn(x1), bh[hr]) : __float2half_rn(0.0f);
                const __half2 lh = __halves2half2(h0, h1);
                lfrag.r[hr + 2 * nt] = *reinterpret_cast<const uint32_t*>(&lh);
                *reinterpret_cast<uint32_t*>(rec_ptr + kTcMqk + tc_sq_off(i, j)) = pack_bf2((i >= j) ? y0 : 0.0f, (i >= j + 1) ? y1 : 0.0f);
            }
        }
    }
    // ---- kr = ki (*) bf(E_tot), over the ki tile ----
    {
        uint4 ki[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) ki[i] = prep_lds(kip + 16 * i);
        __syncwarp();   // every lane is done with ki and with beta_act
#pragma unroll
        for (int i = 0; i < 8; ++i)
            prep_sts(rec + kTcKr + tc_kr_off(8 * hh + i, c), bf2_mul(ki[i].x, etb[0]), bf2_mul(ki[i].y, etb[1]), bf2_mul(ki[i].z, etb[2]),
                     bf2_mul(ki[i].w, etb[3]));
    }
    neumann_inverse_warp(lfrag, rec_ptr + kTcInv, lane);
    __syncwarp();
    return true;
}

}  // namespace fkda
