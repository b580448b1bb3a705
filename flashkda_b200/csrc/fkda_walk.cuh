// One chunk step of a (sequence, head) chain on mma.sync, for ONE WARP that owns 16 * kMt rows of the chain's state and
// keeps them in registers as A fragments.  The recurrence S <- f(S, chunk) decouples completely over the state's V rows
// (each row sees the same chunk operands), so a chain can be cut into row slices that never talk to each other: no
// barrier and no hand-over between warps inside a chunk.
//
// Thread g = lane / 4, tq = lane % 4 holds, of row tile mt and K step j, the elements {(g | g+8) x columns 16j + {2tq, 2tq+1},
// (g | g+8) x 16j + 8 + {2tq, 2tq+1}}: an accumulator fragment of the update product has the same elements in the same
// threads, so the update S[v,k] = bf(fma(S[v,k], E_tot[k], DST[v,k])) runs fragment on fragment.
//
// The chain of one step is D1 = S . kd^T (eight dependent K steps) -> u' -> U = bf(u' INV^T) -> DST = U^T . kr -> S.  The
// steps of two chunks overlap: as soon as 16 columns of the state are refreshed, the K step of the NEXT chunk's D1 that
// reads them is issued, so the eight dependent products of D1 run inside the update instead of after it.
#pragma once

#include <cuda.h>

#include "fkda_common.cuh"
#include "fkda_internal.h"
#include "fkda_sm100.cuh"

namespace fkda {

// Four 8x8 b16 matrices, transposed on the way: thread (g, tq) receives elements (rows 2tq, 2tq+1; column g) of each.
__device__ __forceinline__ void ldmatrix_x4_t(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_a(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
// Four 8x8 b16 matrices out, transposed: lane 8m + r gives the address of row r (16 bytes) of the m-th transposed matrix.
__device__ __forceinline__ void stmatrix_x4_t(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3)
                 : "memory");
}
__device__ __forceinline__ void stmatrix_x4(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3)
                 : "memory");
}
__device__ __forceinline__ float2 lds_f2(uint32_t addr) {
    float2 x;
    asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(x.x), "=f"(x.y) : "r"(addr));
    return x;
}
__device__ __forceinline__ uint4 lds_u4(uint32_t addr) {
    uint4 x;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(addr) : "memory");
    return x;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
    uint32_t x;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(x) : "r"(addr));
    return x;
}

// (predicated: no branch in the middle of a chunk step)
__device__ __forceinline__ void store_if(bool yes, void* p, const uint4& x) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %0, 0;\n@p st.global.v4.b32 [%1], {%2,%3,%4,%5};\n}\n" ::"r"((int)yes), "l"(p), "r"(x.x),
                 "r"(x.y), "r"(x.z), "r"(x.w)
                 : "memory");
}

// bf(fma(s, e, d)) for a packed pair of state elements
__device__ __forceinline__ uint32_t update_pair(uint32_t s, const float2& e, float d0, float d1) {
    float y0, y1;
    fma2_rn(y0, y1, bf_lo(s), bf_hi(s), e.x, e.y, d0, d1);
    return pack_bf2(y0, y1);
}

// Tensor map over v (see encode_v_map).
struct alignas(64) VMap {
    CUtensorMap v;
};

// Per-lane byte offsets into a record (ldmatrix: lane 8m + r addresses row r of the m-th 8x8 matrix)
struct WalkLane {
    uint32_t b1;    // kd fragments of the token tiles 0, 1: (tile 0, K chunk 0), (0, 1), (1, 0), (1, 1); qd 256 bytes further
    uint32_t kr;    // kr: (tokens 0-7, column block 0), (8-15, 0), (0-7, 1), (8-15, 1)
    uint32_t sq;    // INV / Mqk: (row group 0, K chunk 0), (0, 1), (1, 0), (1, 1)
    uint32_t et;    // E_tot of columns 2tq, 2tq+1
    uint32_t beta;  // sigmoid(beta) of tokens 2tq, 2tq+1
};
__device__ __forceinline__ WalkLane walk_lane(int lane) {
    const int m = lane >> 3, r = lane & 7, tq = lane & 3;
    WalkLane w;
    w.b1 = (uint32_t)(kTcB1 + (m & 1) * kTcB1Lbo + (m >> 1) * 128 + r * 16);
    w.kr = (uint32_t)(kTcKr + (m & 1) * kTcKrLbo + (m >> 1) * kTcKrSbo + r * 16);
    w.sq = (uint32_t)((m & 1) * 256 + (m >> 1) * 128 + r * 16);
    w.et = (uint32_t)(kTcEt + tq * 8);
    w.beta = (uint32_t)(kTcBeta + tq * 4);
    return w;
}

// The products are issued in source order (volatile): a warp's tensor pipe takes one every 8 cycles and a dependent one
// after 20, so the order below is the schedule.
__device__ __forceinline__ void mma_ord(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    mma_bf16_f32acc(d, a[0], a[1], a[2], a[3], b0, b1);
}
__device__ __forceinline__ void mma_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}

// What a chunk needs before its update product; fetched while the previous chunk's update runs.
template <int kMt>
struct WalkHead {
    uint32_t inv[4], mqk[4], bp[2];
    uint32_t v[kMt][4];   // value fragments {row g: tokens 2tq,+1 | row g+8 | row g: tokens 2tq+8,+9 | row g+8}
    __device__ __forceinline__ void fetch(uint32_t rec, const WalkLane& wl) {
        ldmatrix_x4_a(inv[0], inv[1], inv[2], inv[3], rec + kTcInv + wl.sq);
        ldmatrix_x4_a(mqk[0], mqk[1], mqk[2], mqk[3], rec + kTcMqk + wl.sq);
        bp[0] = lds_u32(rec + wl.beta);
        bp[1] = lds_u32(rec + wl.beta + 16);
    }
    // rows past the sequence end (token >= len) count as zeros
    __device__ __forceinline__ void mask(int len, int tq) {
        const int left0 = len - 2 * tq, left1 = left0 - 8;
        const uint32_t m0 = left0 >= 2 ? 0xffffffffu : (left0 == 1 ? 0xffffu : 0u);
        const uint32_t m1 = left1 >= 2 ? 0xffffffffu : (left1 == 1 ? 0xffffu : 0u);
#pragma unroll
        for (int mt = 0; mt < kMt; ++mt) {
            v[mt][0] &= m0; v[mt][1] &= m0;
            v[mt][2] &= m1; v[mt][3] &= m1;
        }
    }
};

// kStrung: a product takes its pipe for 8.5 cycles and a warp issues in order, so the products of a block are strung together with
// the update of the block after it, pair by pair, and neither waits for the other.  That pays where a walking warp has its scheduler
// to itself (131 072 tokens, 32 heads 3.88 -> 3.75 ms); with the preparing warps beside it (fkda_fused.cuh) a block's update as one
// piece is as fast or faster (8 x 32 768 tokens, 64 heads: 8.47 ms against 8.74).
template <int kMt, bool kStrung = (kMt == 1)>
struct WalkState {
    uint32_t s[kMt][8][4];     // my state rows, A fragments
    float u0[kMt][2][4];       // S . kd^T of the current chunk, token tiles 0 and 1
    uint32_t qn[2][4];         // qd fragments of the current chunk's first two K steps

    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int mt = 0; mt < kMt; ++mt)
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[mt][j][e] = 0u;
    }
    // B fragments of K step j of D1: kd (the token tiles 0 and 1)
    __device__ __forceinline__ void fetch_kd(uint32_t (&b)[4], uint32_t rec, const WalkLane& wl, int j) {
        ldmatrix_x4_a(b[0], b[1], b[2], b[3], rec + wl.b1 + 2 * j * kTcB1Lbo);
    }
    __device__ __forceinline__ void fetch_qd(uint32_t (&b)[4], uint32_t rec, const WalkLane& wl, int j) {
        ldmatrix_x4_a(b[0], b[1], b[2], b[3], rec + wl.b1 + 2 * j * kTcB1Lbo + 256);
    }
    __device__ __forceinline__ void d1_step(float (&acc)[kMt][2][4], const uint32_t (&b)[4], int j) {
#pragma unroll
        for (int mt = 0; mt < kMt; ++mt) {
            if (j == 0) {
                mma_zero(acc[mt][0], s[mt][j], b[0], b[1]);
                mma_zero(acc[mt][1], s[mt][j], b[2], b[3]);
            } else {
                mma_ord(acc[mt][0], s[mt][j], b[0], b[1]);
                mma_ord(acc[mt][1], s[mt][j], b[2], b[3]);
            }
        }
    }
    // S . kd^T of the first chunk of a walk
    __device__ __forceinline__ void first(uint32_t rec, const WalkLane& wl) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            uint32_t b[4];
            fetch_kd(b, rec, wl, j);
            d1_step(u0, b, j);
        }
        fetch_qd(qn[0], rec, wl, 0);
        fetch_qd(qn[1], rec, wl, 1);
    }
    // One chunk, record at shared-memory address `rec`, operands of its head in `hd`; S . kd^T of the chunk at `next` is formed
    // on the way (`next` = `rec` when there is none: it is then not used).  `mid(j)` is called after block j of the update:
    // the caller fetches the next head and finishes the out rows there, in the shadow of the products.  kNext = false: this is
    // the only chunk.
    // The chain of a chunk is u' -> U -> DST -> update -> the next u0; at its start the tensor pipe would be idle, so that is
    // where most of the out term's S . qd^T goes, which only has to read each 16 columns of the state before they are updated
    // (all of D1 inside the update: 0.515 us per chunk step of recurrence_rows_kernel).
    // o[mt] = out of tokens 8 (i >> 1) + 2tq, +1 of row g + 8 (i & 1), i = 0 .. 3, complete after block 2.
    template <bool kNext = true, class Mid>
    __device__ __forceinline__ void chunk(uint32_t rec, uint32_t next, const WalkLane& wl, const WalkHead<kMt>& hd, uint32_t (&o)[kMt][4], Mid&& mid) {
        constexpr int kAhead = kStrung ? 3 : 2, kAheadB = kStrung ? 2 : 1;   // blocks whose operands (kr and E_tot, kd) are fetched ahead of their products
        uint32_t kr[8][4], b[8][4], q[8][4];
        float2 et[8][2];
        float o0[kMt][2][4];   // S . qd^T
        auto fetch_kr = [&](int j) {
            ldmatrix_x4_t(kr[j][0], kr[j][1], kr[j][2], kr[j][3], rec + wl.kr + 2 * j * kTcKrSbo);
            et[j][0] = lds_f2(rec + wl.et + 64 * j);
            et[j][1] = lds_f2(rec + wl.et + 64 * j + 32);
        };
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            q[0][e] = qn[0][e];
            q[1][e] = qn[1][e];
        }
        fetch_qd(q[2], rec, wl, 2);
        fetch_qd(q[3], rec, wl, 3);
        d1_step(o0, q[0], 0);
        d1_step(o0, q[1], 1);
#pragma unroll
        for (int j = 0; j < kAhead; ++j) fetch_kr(j);
        // ---- u' = (v (-) bf(u0)) (*) bf(beta);  U = bf(u' INV^T) as A fragments (tokens are the K dimension) ----
        uint32_t up[kMt][4], ufr[kMt][4];
#pragma unroll
        for (int mt = 0; mt < kMt; ++mt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const uint32_t x = pack_bf2(u0[mt][e >> 1][2 * (e & 1)], u0[mt][e >> 1][2 * (e & 1) + 1]);
                up[mt][e] = bf2_mul(bf2_sub(hd.v[mt][e], x), hd.bp[e >> 1]);
            }
        float c[kMt][2][4];
#pragma unroll
        for (int mt = 0; mt < kMt; ++mt) {
            mma_zero(c[mt][0], up[mt], hd.inv[0], hd.inv[1]);
            mma_zero(c[mt][1], up[mt], hd.inv[2], hd.inv[3]);
        }
        if constexpr (kNext) {
#pragma unroll
            for (int j = 0; j < kAheadB; ++j) fetch_kd(b[j], next, wl, j);
        }
        fetch_qd(q[4], rec, wl, 4);
        fetch_qd(q[5], rec, wl, 5);
        d1_step(o0, q[2], 2);
        d1_step(o0, q[3], 3);
#pragma unroll
        for (int mt = 0; mt < kMt; ++mt)
#pragma unroll
            for (int i = 0; i < 4; ++i) ufr[mt][i] = pack_bf2(c[mt][i >> 1][2 * (i & 1)], c[mt][i >> 1][2 * (i & 1) + 1]);
        // ---- blocks of 16 state columns: DST = U^T . kr two blocks ahead, the update, K step j of the next S . kd^T ----
        float d[8][kMt][2][4], m[kMt][2][4];
        auto dst = [&](int j) {
#pragma unroll
            for (int mt = 0; mt < kMt; ++mt) {
                mma_zero(d[j][mt][0], ufr[mt], kr[j][0], kr[j][1]);
                mma_zero(d[j][mt][1], ufr[mt], kr[j][2], kr[j][3]);
            }
        };
        dst(0);
        dst(1);
        fetch_qd(q[6], rec, wl, 6);
        fetch_qd(q[7], rec, wl, 7);
        d1_step(o0, q[4], 4);
        d1_step(o0, q[5], 5);
        auto update = [&](int j, int i) {   // pair i of the 4 kMt of block j
            const int mt = i >> 2, e = i & 3;
            s[mt][j][e] = update_pair(s[mt][j][e], et[j][e >> 1], d[j][mt][e >> 1][2 * (e & 1)], d[j][mt][e >> 1][2 * (e & 1) + 1]);
        };
        if constexpr (kStrung) {
#pragma unroll
            for (int i = 0; i < 4 * kMt; ++i) update(0, i);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j + kAhead < 8) fetch_kr(j + kAhead);
            if (kNext && j + kAheadB < 8) fetch_kd(b[j + kAheadB], next, wl, j + kAheadB);
            if constexpr (kStrung) {
#pragma unroll
                for (int i = 0; i < 2 * kMt; ++i) {
                    if constexpr (kNext) {
                        if (j == 0) mma_zero(u0[i >> 1][i & 1], s[i >> 1][0], b[0][2 * (i & 1)], b[0][2 * (i & 1) + 1]);
                        else mma_ord(u0[i >> 1][i & 1], s[i >> 1][j], b[j][2 * (i & 1)], b[j][2 * (i & 1) + 1]);
                    }
                    if (j < 7) update(j + 1, i);
                }
#pragma unroll
                for (int i = 0; i < 2 * kMt; ++i) {
                    if (j + 2 < 8) mma_zero(d[j + 2][i >> 1][i & 1], ufr[i >> 1], kr[j + 2][2 * (i & 1)], kr[j + 2][2 * (i & 1) + 1]);
                    if (j < 7) update(j + 1, 2 * kMt + i);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 4 * kMt; ++i) update(j, i);
                if constexpr (kNext) d1_step(u0, b[j], j);
                if (j + 2 < 8) dst(j + 2);
            }
            if (j == 0) {
                d1_step(o0, q[6], 6);
                d1_step(o0, q[7], 7);
            }
            if (j == 1) {   // the out term U Mqk^T
#pragma unroll
                for (int mt = 0; mt < kMt; ++mt) {
                    mma_zero(m[mt][0], ufr[mt], hd.mqk[0], hd.mqk[1]);
                    mma_zero(m[mt][1], ufr[mt], hd.mqk[2], hd.mqk[3]);
                }
            }
            if (j == 2) {   // out = bf(o0) (+) bf(U Mqk^T)
#pragma unroll
                for (int mt = 0; mt < kMt; ++mt)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        o[mt][i] = bf2_add(pack_bf2(o0[mt][i >> 1][2 * (i & 1)], o0[mt][i >> 1][2 * (i & 1) + 1]),
                                           pack_bf2(m[mt][i >> 1][2 * (i & 1)], m[mt][i >> 1][2 * (i & 1) + 1]));
            }
            mid(j);
            if (kNext && j == 5) {   // the next chunk's first products follow this one's last without a wait for their operands
                fetch_qd(qn[0], next, wl, 0);
                fetch_qd(qn[1], next, wl, 1);
            }
        }
    }
};

// ---- states between global memory and fragment registers, 16 rows (one row tile) at a time ----
// A staging tile per warp: 16 rows of 128 bf16 (256 bytes a row); the 16-byte piece c of row r sits at
// r * 256 + ((c ^ (r & 7)) * 16), so that neither ldmatrix / stmatrix (8 rows of one piece) nor whole-row accesses collide.
// Global memory sees whole rows (512 contiguous bytes per warp instruction).
constexpr int kWalkStageBytes = 16 * 256;
__device__ __forceinline__ uint32_t walk_stage_off(int r, int piece) { return (uint32_t)(r * 256 + ((piece ^ (r & 7)) << 4)); }

// kMt consecutive row tiles; `src` = element (first row, column 0); fp32 states are rounded to bf16.  The loads of all tiles
// are in flight before the first is staged.
template <int kMt, bool kFp32>
__device__ __forceinline__ void walk_load_tiles(uint32_t (&s)[kMt][8][4], uint8_t* stage, const void* src, int lane) {
    const uint32_t base = sm100::smem_u32(stage);
    const int r = (lane & 7) + 8 * ((lane >> 3) & 1), c = lane >> 4;
    const uint4* p = reinterpret_cast<const uint4*>(src) + lane;
    constexpr int kPer = kFp32 ? 16 : 8;   // 16-byte pieces per lane and tile
    uint4 x[kMt][kPer];
#pragma unroll
    for (int mt = 0; mt < kMt; ++mt)
#pragma unroll
        for (int i = 0; i < kPer; ++i) x[mt][i] = p[32 * (kPer * mt + i)];
#pragma unroll
    for (int mt = 0; mt < kMt; ++mt) {
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            if constexpr (kFp32)   // row i, columns 4 lane ..: half (lane & 1) of piece lane / 2
                *reinterpret_cast<uint2*>(stage + walk_stage_off(i, lane >> 1) + 8 * (lane & 1)) =
                    make_uint2(pack_bf2(__uint_as_float(x[mt][i].x), __uint_as_float(x[mt][i].y)),
                               pack_bf2(__uint_as_float(x[mt][i].z), __uint_as_float(x[mt][i].w)));
            else                   // row 2 i + lane / 16, piece lane % 16
                *reinterpret_cast<uint4*>(stage + walk_stage_off(2 * i + (lane >> 4), lane & 15)) = x[mt][i];
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) ldmatrix_x4_a(s[mt][j][0], s[mt][j][1], s[mt][j][2], s[mt][j][3], base + walk_stage_off(r, 2 * j + c));
        __syncwarp();
    }
}
__device__ __forceinline__ void walk_store_tile(const uint32_t (&s)[8][4], uint8_t* stage, void* dst, bool fp32, int lane) {
    const uint32_t base = sm100::smem_u32(stage);
    const int r = (lane & 7) + 8 * ((lane >> 3) & 1), c = lane >> 4;
#pragma unroll
    for (int j = 0; j < 8; ++j) stmatrix_x4(base + walk_stage_off(r, 2 * j + c), s[j][0], s[j][1], s[j][2], s[j][3]);
    __syncwarp();
    if (fp32) {
        float4* p = reinterpret_cast<float4*>(dst);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint2 y = *reinterpret_cast<const uint2*>(stage + walk_stage_off(i, lane >> 1) + 8 * (lane & 1));
            p[32 * i + lane] = make_float4(bf_lo(y.x), bf_hi(y.x), bf_lo(y.y), bf_hi(y.y));
        }
    } else {
        uint4* p = reinterpret_cast<uint4*>(dst);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            p[32 * i + lane] = *reinterpret_cast<const uint4*>(stage + walk_stage_off(2 * i + (lane >> 4), lane & 15));
    }
    __syncwarp();
}

}  // namespace fkda
