// Short sequences: a fixed batch whose sequences hold 1 .. 16 tokens each, or a ragged batch in which no sequence holds more
// than 16 (ONE chunk per sequence): a decode step of a large batch, the verification pass of speculative decoding.  Such a
// batch is bound by HBM traffic on the [128,128] states (read once, written once), so the whole forward of a (sequence, head)
// chain runs in ONE kernel with nothing staged in HBM and no workspace, and the kernel is built to keep state loads and
// stores in flight on every SM all the time:
//
// One persistent CTA per SM (12 warps), chains blockIdx.x, blockIdx.x + gridDim.x, ...
//   * two groups of four walking warps; each group owns two 32 KB stages of shared memory.  A stage takes the whole state of a
//     chain (bf16) or 64 of its rows (fp32: the groups share a chain).  A stage is filled by TMA, its rows go through the
//     registers of the walking warps (fkda_walk.cuh) and back into the stage in place, and leave by TMA; the group's other
//     stage is refilled meanwhile, so 64 KB of loads per SM are in flight beside the stores.  128-byte swizzle on both
//     ways: whole 128-byte lines for global memory, no bank conflicts for fragments;
//   * four preparing warps build the chunk operands of the coming chains in a ring of records (fkda_prep.cuh), the inputs of
//     their next chain in registers ahead of time.
// Everything is handed over through mbarriers with bounded waits.
// Bound by HBM: 32 768 chains of 2 tokens take 348 us with bf16 and 661 us with fp32 states, 1.01 and 1.05 of the copy bandwidth
// (554 and 833 us for the predecessor, whose four warps loaded, computed and stored one chain after the other); with 16
// tokens 476 and 795 us (776, 1 083), where the preparing warps take as long as the states.
// Numerics and results: those of the chunked kernels on the same inputs (tests/torch_ref.py:153-251 of the reference; the
// reference itself runs such batches through its two general kernels, csrc/smxx/fwd_kernel1.cuh / fwd_kernel2.cuh).
#include <cuda.h>
#include <string.h>

#include "fkda_common.cuh"
#include "fkda_internal.h"
#include "fkda_prep.cuh"
#include "fkda_walk.cuh"

namespace fkda {

using namespace sm100;

constexpr int kShortGroups = 2, kShortWalkers = 4 * kShortGroups, kShortPrep = 4;
constexpr int kShortThreads = (kShortWalkers + kShortPrep) * 32;
constexpr int kShortSlots = 4;                       // records (and value tiles) in the ring
constexpr int kShortStage = 32768;                   // state stage: 128 rows of bf16 or 64 rows of fp32
constexpr int kShortV = kShortGroups * 2 * kShortStage;                   // value tiles: two halves [16][64] bf16 each
constexpr int kShortVTile = kChunk * kD * 2;
constexpr int kShortOut = kShortV + kShortSlots * kShortVTile;            // per walking warp up to two out tiles [16][16]
constexpr int kShortRec = kShortOut + kShortWalkers * 2 * 512;
constexpr int kShortCtrl = kShortRec + kShortSlots * kTcRecord;
struct ShortCtrl {
    uint64_t full[kShortSlots];           // a record is complete and its value tile has landed
    uint64_t empty[kShortSlots];          // a slot has been read by all walking warps of its chain
    uint64_t sfull[kShortGroups][2];      // a state stage has landed
    uint64_t sdone[kShortGroups];         // the walking warps of a group have put their rows back
    int32_t len[kShortSlots];             // tokens of the slot's chain
    int32_t abort_flag;
};
constexpr int kShortSmemBytes = kShortCtrl + (int)sizeof(ShortCtrl) + 1024;
static_assert(kShortRec % 16 == 0 && kShortCtrl % 8 == 0 && kShortSmemBytes <= 232448, "shared-memory layout");
static_assert(kShortPrep <= kShortSlots, "no more preparing warps than slots (see fkda_fused.cuh)");

struct alignas(64) ShortMaps {
    CUtensorMap v, h0, hT;
};

// Where the fragments of row tile `row` (first row, inside the stage) and K step j live in a state stage.
// bf16: two boxes of 64 columns; lane's ldmatrix / stmatrix row.
__device__ __forceinline__ uint32_t short_bf16_off(int row, int j, int lane) {
    const int r = row + (lane & 7) + 8 * ((lane >> 3) & 1), piece = 2 * j + (lane >> 4);
    return (uint32_t)((piece >> 3) * 16384 + r * 128 + (((piece & 7) ^ (lane & 7)) << 4));
}
// fp32: four boxes of 32 columns; my element pair e of the fragment
__device__ __forceinline__ uint32_t short_fp32_off(int row, int j, int e, int lane) {
    const int g = lane >> 2, tq = lane & 3, piece = 4 * (j & 1) + 2 * (e >> 1) + (tq >> 1);
    return (uint32_t)((j >> 1) * 8192 + (row + g + 8 * (e & 1)) * 128 + ((piece ^ g) << 4) + 8 * (tq & 1));
}
template <int kMt, bool kFp32>
__device__ __forceinline__ void short_get(uint32_t (&s)[kMt][8][4], uint32_t stage, int row, int lane) {
#pragma unroll
    for (int mt = 0; mt < kMt; ++mt)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if constexpr (kFp32) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 x = lds_f2(stage + short_fp32_off(row + 16 * mt, j, e, lane));
                    s[mt][j][e] = pack_bf2(x.x, x.y);
                }
            } else {
                ldmatrix_x4_a(s[mt][j][0], s[mt][j][1], s[mt][j][2], s[mt][j][3], stage + short_bf16_off(row + 16 * mt, j, lane));
            }
        }
}
template <int kMt, bool kFp32>
__device__ __forceinline__ void short_put(const uint32_t (&s)[kMt][8][4], uint32_t stage, int row, int lane) {
#pragma unroll
    for (int mt = 0; mt < kMt; ++mt)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if constexpr (kFp32) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(stage + short_fp32_off(row + 16 * mt, j, e, lane)),
                                 "f"(bf_lo(s[mt][j][e])), "f"(bf_hi(s[mt][j][e]))
                                 : "memory");
            } else {
                stmatrix_x4(stage + short_bf16_off(row + 16 * mt, j, lane), s[mt][j][0], s[mt][j][1], s[mt][j][2], s[mt][j][3]);
            }
        }
}

// kRagged: a ragged batch behind the prefix kernel's decision; it may hold empty sequences (a check for them in the build for fixed
// batches as well: 357 -> 382 us for 32 768 decode steps)
template <bool kFp32, bool kRagged>
__global__ void __launch_bounds__(kShortThreads, 1)
short_kernel(const __grid_constant__ TwoPassArgs a, const __grid_constant__ ShortMaps maps) {
    grid_dep_wait();
    // a ragged batch that the prefix kernel has given to other kernels (a longer sequence: the general ones; one token
    // each: the decode kernel)
    if (kRagged && *a.short_flag != 1) return;
    extern __shared__ uint8_t smem_dyn[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    ShortCtrl& ctl = *reinterpret_cast<ShortCtrl*>(sm + kShortCtrl);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    volatile int* abort_flag = &ctl.abort_flag;
    if (!kRagged && a.status != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
        *a.status = 0;
        *a.records = 0;
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kShortSlots; ++s) {
            mbar_init(&ctl.full[s], 2);
            mbar_init(&ctl.empty[s], kFp32 ? kShortWalkers : 4);
        }
        for (int g = 0; g < kShortGroups; ++g) {
            mbar_init(&ctl.sfull[g][0], 1);
            mbar_init(&ctl.sfull[g][1], 1);
            mbar_init(&ctl.sdone[g], 4);
        }
        ctl.abort_flag = 0;
        mbar_fence_init();
    }
    __syncthreads();
    const int64_t n_chains = a.N * a.H;
    const int n_local = (int)((n_chains - blockIdx.x + gridDim.x - 1) / gridDim.x);   // (the grid is no larger than n_chains)
    bool failed = false;

    if (warp >= kShortWalkers) {
        // =========================== preparing warps ===========================
        const int p = warp - kShortWalkers;
        // first token, length (0 .. 16 tokens) and head of local chain i
        auto locate = [&](int i, int64_t* t0, int* len, int* h) {
            const int64_t chain = blockIdx.x + (int64_t)i * gridDim.x, n = chain / a.H;
            *h = (int)(chain - n * a.H);
            if (kRagged) {
                const int64_t b = a.cu_seqlens[n], e = a.cu_seqlens[n + 1];
                *len = e > b ? (int)(e - b) : 0;
                *t0 = *len > 0 ? b : 0;   // (an empty sequence: any address inside the tensors)
            } else {
                *t0 = n * a.T;
                *len = (int)a.T;
            }
        };
        PrepHead x;
        PrepSrc src;
        int64_t t0 = 0, t0n = 0;
        int len = 0, h = 0, lenn = 0, hn = 0;
        if (p < n_local) {
            locate(p, &t0, &len, &h);
            src = prep_src(a, t0, max(len, 1), h, lane);
            prep_load(a, src, t0, max(len, 1), h, lane, x);
        }
        for (int i = p; i < n_local; i += kShortPrep) {
            const int slot = i % kShortSlots;
            const uint32_t phase = 1u ^ ((i / kShortSlots) & 1);   // of empty[slot]: the first round finds the slots free
            const bool next_valid = i + kShortPrep < n_local;
            if (next_valid) locate(i + kShortPrep, &t0n, &lenn, &hn);
            uint8_t* rec = sm + kShortRec + slot * kTcRecord;
            auto acquire = [&]() {   // the slot is free: ask for the value tile
                if (__all_sync(0xffffffffu, mbar_wait_bounded(&ctl.empty[slot], phase, abort_flag, a.wait_ns)) == 0) return false;
                if (lane == 0) {
                    ctl.len[slot] = len;
                    // (tokens past the sequence end are masked by the walking warps)
                    mbar_arrive_expect_tx(&ctl.full[slot], kShortVTile);
                    tma_load_3d(sm + kShortV + slot * kShortVTile, &maps.v, 0, h, (int)t0, &ctl.full[slot]);
                    tma_load_3d(sm + kShortV + slot * kShortVTile + kShortVTile / 2, &maps.v, kD / 2, h, (int)t0, &ctl.full[slot]);
                }
                __syncwarp();
                return true;
            };
            auto next = [&]() {   // the inputs of my next chain travel while the products and the inverse run
                if (next_valid) {
                    src = prep_src(a, t0n, max(lenn, 1), hn, lane);
                    prep_load(a, src, t0n, max(lenn, 1), hn, lane, x);
                }
            };
            if (!prep_compute<true, false>(a, src, len, rec, lane, x, acquire, next)) {
                failed = true;
                *abort_flag = 1;
                // my value tile in flight lands before this CTA's shared memory goes
                if (i >= kShortPrep) mbar_wait_bounded(&ctl.full[slot], phase, nullptr, 100000000ull);
                break;
            }
            mbar_arrive_lane0(&ctl.full[slot], lane);
            t0 = t0n; len = lenn; h = hn;
        }
    } else {
        // =========================== walking warps ===========================
        constexpr int kMt = kFp32 ? 1 : 2;
        const int group = warp >> 2, wiw = warp & 3;
        const bool leader = wiw == 0 && lane == 0;
        const int row = wiw * 16 * kMt;                                // my first row in a stage
        const int vrow = (kFp32 ? 64 * group : 0) + row;               // my first state row = value column
        const int per = kFp32 ? 1 : kShortGroups;                      // my group takes local chains first, first + per, ...
        const int first = kFp32 ? 0 : group;
        const int n_items = n_local > first ? (n_local - first + per - 1) / per : 0;
        const bool has_in = a.initial_state != nullptr, has_out = a.final_state != nullptr;
        const WalkLane wl = walk_lane(lane);
        const uint32_t rec0 = smem_u32(sm + kShortRec);
        uint8_t* const stages = sm + group * 2 * kShortStage;
        uint32_t v_off[kMt];   // my value columns in a value tile (layout as in fused_kernel)
        const int v_tok = (lane & 7) + 8 * (lane >> 4);
#pragma unroll
        for (int mt = 0; mt < kMt; ++mt) {
            const int piece = (vrow + 16 * mt) / 8 + ((lane >> 3) & 1);   // 16-byte piece of a 256-byte value row
            v_off[mt] = smem_u32(sm + kShortV) + (uint32_t)((piece >> 3) * (kShortVTile / 2) + v_tok * 128 + (((piece & 7) ^ (lane & 7)) << 4));
        }
        const uint32_t o_tile = smem_u32(sm + kShortOut + warp * 2 * 512);
        const uint32_t o_frag = o_tile + (uint32_t)(v_tok * 32 + ((((lane >> 3) & 1) ^ ((v_tok >> 2) & 1)) << 4));
        const uint32_t o_row = o_tile + (uint32_t)((lane >> 1) * 32 + (((lane & 1) ^ ((lane >> 3) & 1)) << 4));
        auto chain_of = [&](int k) { return blockIdx.x + (int64_t)(first + k * per) * gridDim.x; };
        // (leader) item k's rows between global memory and stage k & 1
        auto state_load = [&](int k) {
            uint8_t* st = stages + (k & 1) * kShortStage;
            uint64_t* bar = &ctl.sfull[group][k & 1];
            const int y = (int)(chain_of(k) * kD) + (kFp32 ? 64 * group : 0);
            mbar_arrive_expect_tx(bar, kShortStage);
            if constexpr (kFp32) {
                for (int b = 0; b < 4; ++b) tma_load_2d(st + 8192 * b, &maps.h0, 32 * b, y, bar);
            } else {
                for (int b = 0; b < 2; ++b) tma_load_2d(st + 16384 * b, &maps.h0, 64 * b, y, bar);
            }
        };
        auto state_store = [&](int k) {
            const uint8_t* st = stages + (k & 1) * kShortStage;
            const int y = (int)(chain_of(k) * kD) + (kFp32 ? 64 * group : 0);
            if constexpr (kFp32) {
                for (int b = 0; b < 4; ++b) tma_store_2d(&maps.hT, 32 * b, y, st + 8192 * b);
            } else {
                for (int b = 0; b < 2; ++b) tma_store_2d(&maps.hT, 64 * b, y, st + 16384 * b);
            }
            bulk_commit_group();
        };
        int loads = 0;   // (leader) items whose load has been issued
        if (leader && has_in)
            for (; loads < 2 && loads < n_items; ++loads) state_load(loads);
        WalkState<kMt> w;
        WalkHead<kMt> hd;
        auto wait_all = [&](uint64_t* bar, uint32_t ph) { return __all_sync(0xffffffffu, mbar_wait_bounded(bar, ph, abort_flag, a.wait_ns)) != 0; };
#pragma unroll 1
        for (int k = 0; k < n_items; ++k) {
            const int i = first + k * per, slot = i % kShortSlots;
            const int64_t chain = chain_of(k), n = chain / a.H;
            const int h = (int)(chain - n * a.H);
            const uint32_t stage = smem_u32(stages + (k & 1) * kShortStage);
            if (has_in) {
                if (!wait_all(&ctl.sfull[group][k & 1], (uint32_t)((k >> 1) & 1))) { failed = true; break; }
                short_get<kMt, kFp32>(w.s, stage, row, lane);
            } else {
                w.clear();
            }
            if (leader && k > 0) {
                // the other stage's rows have left (their store was issued an item ago): refill it
                bulk_wait_group_read<0>();
                if (has_in && loads < n_items) state_load(loads++);
            }
            __syncwarp();
            if (!wait_all(&ctl.full[slot], (uint32_t)((i / kShortSlots) & 1))) { failed = true; break; }
            const uint32_t rec = rec0 + slot * kTcRecord;
            const int len = ctl.len[slot];
            w.first(rec, wl);
            hd.fetch(rec, wl);
#pragma unroll
            for (int mt = 0; mt < kMt; ++mt) ldmatrix_x4_t(hd.v[mt][0], hd.v[mt][1], hd.v[mt][2], hd.v[mt][3], v_off[mt] + slot * kShortVTile);
            hd.mask(len, lane & 3);
            const int64_t t0 = kRagged ? a.cu_seqlens[n] : n * a.T;
            __nv_bfloat16* og = a.out + (t0 + (lane >> 1)) * a.token_stride + (int64_t)h * kD + vrow + 8 * (lane & 1);
            uint32_t o[kMt][4];
            uint4 orow[kMt];
            w.template chunk<false>(rec, rec, wl, hd, o, [&](int j) {
                if (j == 3) {   // the out rows: fragments through a 512-byte tile, 32 contiguous bytes per token to global memory
#pragma unroll
                    for (int mt = 0; mt < kMt; ++mt) stmatrix_x4_t(o_frag + mt * 512, o[mt][0], o[mt][1], o[mt][2], o[mt][3]);
                    __syncwarp();
                }
                if (j == 4) {
#pragma unroll
                    for (int mt = 0; mt < kMt; ++mt) orow[mt] = lds_u4(o_row + mt * 512);
                }
                if (j == 6 && (lane >> 1) < len) {
#pragma unroll
                    for (int mt = 0; mt < kMt; ++mt) *reinterpret_cast<uint4*>(og + mt * 16) = orow[mt];
                }
            });
            __syncwarp();
            mbar_arrive_lane0(&ctl.empty[slot], lane);   // (my warp's last reads of this slot are done)
            // All warps are done with item k - 1: otherwise an arrival of mine below could count for that item, and the store of
            // item k - 2, which the leader sees off before its own arrival for item k - 1, could still be reading the stage.
            // (Of six ways to order this, among them a barrier per stage, and all warps waiting for item k itself: 154 us
            // for 12 288 chains of 5 tokens with bf16 states, the others 154 to 167.)
            if (k > 0 && !wait_all(&ctl.sdone[group], (uint32_t)((k - 1) & 1))) { failed = true; break; }
            if (kRagged && len == 0) {   // an empty sequence: its state passes through, whatever the record holds
                if (has_in) short_get<kMt, kFp32>(w.s, stage, row, lane);
                else w.clear();
            }
            if (has_out) {
                short_put<kMt, kFp32>(w.s, stage, row, lane);
                fence_proxy_async_smem();
            }
            __syncwarp();
            mbar_arrive_lane0(&ctl.sdone[group], lane);   // my rows are back in the stage
            if (leader) {
                if (!mbar_wait_bounded(&ctl.sdone[group], (uint32_t)(k & 1), abort_flag, a.wait_ns)) failed = true;
                else if (has_out) state_store(k);
            }
            failed = __any_sync(0xffffffffu, failed) != 0;
            if (failed) break;
        }
        if (failed) *abort_flag = 1;
        if (leader) {
            if (failed && has_in)   // loads in flight land before this CTA's shared memory goes
                for (int k = max(0, loads - 2); k < loads; ++k)
                    mbar_wait_bounded(&ctl.sfull[group][k & 1], (uint32_t)((k >> 1) & 1), nullptr, 100000000ull);
            bulk_wait_group<0>();   // the states are written
        }
    }
    if (failed) {
        *abort_flag = 1;
        if (a.status != nullptr) atomicExch(a.status, FKDA_ERR_DEVICE_STATUS);
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------
static bool whole_forward(const fkda_fwd_params& p) {
    return p.phase_mask == 0 || p.phase_mask == (FKDA_PHASE_PREPARE | FKDA_PHASE_RECURRENCE);
}

// A fixed batch of 2 .. 16 tokens per sequence, or a decode step (one token) with more chains than the decode kernel is for.
bool short_eligible(const fkda_fwd_params& p) {
    if (p.cu_seqlens != nullptr || p.T < 1 || p.T > kChunk || p.chunk_states != nullptr || !whole_forward(p)) return false;
    if (p.flags & FKDA_FLAG_NO_SHORT) return false;
    return p.T > 1 || (p.N * p.H > decode_max_chains(p) && !(p.flags & FKDA_FLAG_NO_DECODE));
}
// A decode step of a fixed batch for the decode kernel.
bool decode_eligible(const fkda_fwd_params& p) {
    return p.cu_seqlens == nullptr && p.T == 1 && p.chunk_states == nullptr && whole_forward(p) && !(p.flags & FKDA_FLAG_NO_DECODE) &&
           (p.N * p.H <= decode_max_chains(p) || (p.flags & FKDA_FLAG_NO_SHORT));
}

bool short_ragged_candidate(const fkda_fwd_params& p) {
    // tokens <= 16 per sequence on average is necessary for "no sequence longer than a chunk"; a handful of chains is
    // not worth two extra launches
    return p.cu_seqlens != nullptr && p.N > 0 && p.T > 0 && p.B * p.T <= kChunk * p.N && p.N * p.H >= 64 &&
           p.chunk_states == nullptr && whole_forward(p);
}

template <bool kFp32>
static int launch_short_typed(const fkda_fwd_params& p, const TwoPassArgs& a, int sms, cudaStream_t stream) {
    const int64_t chains = p.N * p.H;
    ShortMaps maps;
    memset(&maps, 0, sizeof(maps));
    if (!encode_v_map(&maps.v, p)) return FKDA_ERR_LAUNCH;
    if (p.initial_state != nullptr && !encode_state_map(&maps.h0, p.initial_state, chains, kFp32)) return FKDA_ERR_LAUNCH;
    if (p.final_state != nullptr && !encode_state_map(&maps.hT, p.final_state, chains, kFp32)) return FKDA_ERR_LAUNCH;
    const int64_t ctas = chains < sms ? chains : sms;
    if (a.short_flag != nullptr) {   // behind the prefix kernel
        if (!allow_smem<short_kernel<kFp32, true>>(kShortSmemBytes)) return FKDA_ERR_LAUNCH;
        return launch_dependent(short_kernel<kFp32, true>, ctas, kShortThreads, kShortSmemBytes, stream, a, maps) ? FKDA_OK : FKDA_ERR_LAUNCH;
    }
    if (!allow_smem<short_kernel<kFp32, false>>(kShortSmemBytes)) return FKDA_ERR_LAUNCH;
    return launch_dependent(short_kernel<kFp32, false>, ctas, kShortThreads, kShortSmemBytes, stream, a, maps) ? FKDA_OK : FKDA_ERR_LAUNCH;
}

int launch_short_ragged(const fkda_fwd_params& p, const TwoPassArgs& a, cudaStream_t stream) {
    // (state rows are counted in 32 bits: half a terabyte of states)
    if (p.N * p.H > 0xffffff && (p.initial_state != nullptr || p.final_state != nullptr)) return FKDA_ERR_BAD_SHAPE;
    const int sms = device_sm_count();
    return a.state_fp32 ? launch_short_typed<true>(p, a, sms, stream) : launch_short_typed<false>(p, a, sms, stream);
}

int launch_short(const fkda_fwd_params& p, cudaStream_t stream, int* n_launches) {
    TwoPassArgs a;
    fill_args(p, &a);
    const int rc = launch_short_ragged(p, a, stream);
    if (rc == FKDA_OK) *n_launches = 1;
    return rc;
}

}  // namespace fkda
