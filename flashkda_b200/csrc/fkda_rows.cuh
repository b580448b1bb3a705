// Recurrence over chunk records in HBM / L2, row slices: a (sequence, head) chain is walked by kRowSplit CTAs of
// kRowWarps warps, each warp with 16 (kMt = 2: 32) of the 128 state rows in registers (fkda_walk.cuh).  The warps of a chain share nothing
// but the records they read, so a chunk step has no barrier in it: every warp waits for the stage of its next chunk, walks
// it, and tells the control warp that it is done with the stage.
//
// Why this shape: with few chains the forward is a serial walk, (number of chunks) x (latency of a step).  A step is about
// 115 cycles of dependent latency (u', U, the first update) plus the products of one warp, 52 x 8.5 cycles of its scheduler's
// tensor pipe, and at most one warp walks on a scheduler.  The tcgen05 form of the same step (control warp, accumulators in
// tensor memory) took 2 100 cycles, of which 1 300 were hand-overs: tensor-memory loads and stores, commits, mbarriers.  With
// only the out term's S . qd^T on tcgen05 (the state put into tensor memory block by block, the product started by the control
// warp, a chunk's out rows stored during the next chunk) a step took 0.46 us against 0.43: eight tcgen05 products and their
// wait take 300 cycles and slow the mma.sync ones beside them from 8.5 to 10.6 cycles.
//
// A stage holds two chunks where shared memory allows it (kPair), which halves the waits, arrivals and branches between chunks
// (230 of 980 cycles per step were spent there): 131 072 tokens, 32 heads 4.21 -> 3.88 ms together with predicated stores and
// arrivals and the next chunk's first fragments fetched ahead; 3.75 with products and update strung together (fkda_walk.cuh).
// Included by fkda_tc.cu.
#pragma once

#include "fkda_walk.cuh"

namespace fkda {

// kWarps walking warps per CTA, kMt row tiles of 16 state rows each: 8 / (kWarps kMt) CTAs per chain
__host__ __device__ constexpr int row_split(int warps, int mt) { return kD / (16 * mt * warps); }
__host__ __device__ constexpr int row_threads(int warps) { return (warps + 1) * 32; }
constexpr int kRowVCols = kD / 2;                               // value columns of a tile: a CTA reads one half of a value row, or both
constexpr int kRowVTile = kChunk * kRowVCols * 2;               // value tile [16 tokens][64] bf16, 128-byte swizzle
static_assert(kRowVTile % 1024 == 0, "tile alignments");

// Shared memory of a CTA with kStages groups of kPair chunks in flight
template <int kMt, int kRowWarps, int kStages, int kPair>
struct RowSmem {
    static constexpr int kRowVBytes = (16 * kMt * kRowWarps > kRowVCols ? 2 : 1) * kRowVTile;   // value tiles of a chunk
    static constexpr int kV = 0;                                        // value tiles (1024-byte aligned for the swizzle)
    static constexpr int kOut = kV + kStages * kPair * kRowVBytes;      // per warp an out tile [16 tokens][16 kMt] bf16
    static constexpr int kRec = kOut + kRowWarps * kMt * 512;             // chunk records
    static constexpr int kStaging = kRec + kStages * kPair * kTcRecord;   // per warp one staging tile for states
    static constexpr int kCtrl = kStaging + kRowWarps * kWalkStageBytes;
    struct Ctrl {
        uint64_t full[kStages];    // operands of a group of chunks have landed (transaction bytes)
        uint64_t empty[kStages];   // a stage has been read by all walking warps
        int32_t abort_flag;
    };
    static constexpr int kBytes = kCtrl + (int)sizeof(Ctrl) + 1024;
    static_assert(kOut % 256 == 0 && kRec % 16 == 0 && kStaging % 16 == 0 && kCtrl % 8 == 0, "tile alignments");
};

// kExport: the states before every cs_every-th chunk are written out as well.  kLoop: a CTA takes several slices in turn
// (for launches that mostly return at once, see launch_tc; the loop alone makes a step 15 % longer).  kRowStages, kPair: 4 stages
// of two chunks when every slice has an SM of its own (with the prepare stage of the next slab loading the memory, records arrive
// up to four steps late: 131 072 tokens, 32 heads: 4.58 -> 4.31 ms with 8 chunks in flight against 4), otherwise of one, so that
// two CTAs fit an SM (with 2 stages of two: 300 + 1 + 211 + 512 tokens of 32 heads 57 us against 51).
template <bool kExport, bool kLoop, int kMt, int kRowWarps, int kRowStages, int kPair>
__global__ void __launch_bounds__(row_threads(kRowWarps), kMt == 1 ? 2 : 1)
recurrence_rows_kernel(const __grid_constant__ TwoPassArgs a, const __grid_constant__ VMap map) {
    extern __shared__ uint8_t smem_dyn[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    static_assert(!kLoop || kPair == 1, "slices in turn: a stage of one chunk");
    constexpr int kRowSplit = row_split(kRowWarps, kMt), kRowCols = 16 * kMt * kRowWarps;
    using L = RowSmem<kMt, kRowWarps, kRowStages, kPair>;
    constexpr int kRowVBytes = L::kRowVBytes;
    typename L::Ctrl& ctl = *reinterpret_cast<typename L::Ctrl*>(sm + L::kCtrl);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    volatile int* abort_flag = &ctl.abort_flag;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kRowStages; ++s) {
            mbar_init(&ctl.full[s], 1);
            mbar_init(&ctl.empty[s], kRowWarps);
        }
        ctl.abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_map(&map.v);
    }
    grid_dep_wait();
    // (a ragged batch that a one-kernel path has served: nothing to do)
    if (a.short_flag != nullptr && *a.short_flag != 0) return;
    __syncthreads();

    const int64_t n_items = a.N * a.H * kRowSplit;
    bool failed = false;
    int k0 = 0;   // groups of the items before: the stages and their phases run on from item to item
    for (int64_t item = blockIdx.x; item < n_items && !failed; item = kLoop ? item + gridDim.x : n_items) {
    // chains come longest first; the second layer of CTAs runs backwards, so that the SMs with the longest chains get the
    // shortest ones beside them (or none)
    const int64_t place = !kLoop && a.layer > 0 && item >= a.layer ? n_items - 1 - (item - a.layer) : item;
    const int64_t chain = place / kRowSplit;
    const int slice = (int)(place % kRowSplit);
    const TcChain ch = tc_locate_chain(a, chain);
    const int h = ch.h;
    // chunk range of this launch: all chunks, or one slab of a pipelined forward (fixed batches)
    const int c0 = a.slab_chunks > 0 ? a.slab_c0 : 0;
    const int c1 = (a.slab_chunks > 0 && c0 + a.slab_chunks < ch.n_chunks) ? c0 + a.slab_chunks : ch.n_chunks;
    if (warp == kRowWarps) {
        // =========================== control warp: keeps the stages filled ===========================
        if (elect_one()) {
            const int n_groups = (c1 - c0 + kPair - 1) / kPair;
            int p = 0;
            for (; p < n_groups; ++p) {
                const int k = k0 + p, s = k % kRowStages, t = c0 + kPair * p, m = min(kPair, c1 - t);
                if (k >= kRowStages && !mbar_wait_bounded(&ctl.empty[s], (uint32_t)((k / kRowStages - 1) & 1), abort_flag, a.wait_ns)) {
                    failed = true;
                    break;
                }
                mbar_arrive_expect_tx(&ctl.full[s], (uint32_t)(m * (kTcRecord + kRowVBytes)));
                bulk_g2s(sm + L::kRec + s * kPair * kTcRecord, ch.rec_base + (int64_t)t * kTcRecord, m * kTcRecord, &ctl.full[s]);
                // rows past the end of the tensor arrive as zeros; rows of the next sequence are never used
                for (int e = 0; e < m; ++e)
                    for (int half = 0; half < kRowVBytes / kRowVTile; ++half)
                        tma_load_3d(sm + L::kV + (s * kPair + e) * kRowVBytes + half * kRowVTile, &map.v, slice * kRowCols / kRowVCols * kRowVCols + half * kRowVCols, h,
                                    (int)(ch.bos + (int64_t)(t + e) * kChunk), &ctl.full[s]);
            }
            if (failed) {   // the copies in flight land before this CTA's shared memory goes
                *abort_flag = 1;
                for (int k = max(0, k0 + p - kRowStages); k < k0 + p; ++k)
                    mbar_wait_bounded(&ctl.full[k % kRowStages], (uint32_t)((k / kRowStages) & 1), nullptr, 100000000ull);
            }
        }
        failed = __any_sync(0xffffffffu, failed) != 0;
    } else {
        // =========================== walking warps ===========================
        const int row0 = slice * kRowCols + warp * 16 * kMt;   // my first state row
        const WalkLane wl = walk_lane(lane);
        uint8_t* stage_tile = sm + L::kStaging + warp * kWalkStageBytes;
        const uint32_t rec0 = smem_u32(sm + L::kRec);
        // my value columns in the [16 tokens][64] tiles: token (lane & 7) + 8 (lane / 16), 16-byte piece (my first column) / 8 + (lane / 8) % 2
        const int o_tok = (lane & 7) + 8 * (lane >> 4);
        uint32_t v_off[kMt];
#pragma unroll
        for (int mt = 0; mt < kMt; ++mt) {
            const int col = row0 + 16 * mt - slice * kRowCols / kRowVCols * kRowVCols;
            v_off[mt] = smem_u32(sm + L::kV) + (uint32_t)(col / kRowVCols * kRowVTile + o_tok * 128 + (((col % kRowVCols / 8 + ((lane >> 3) & 1)) ^ (lane & 7)) << 4));
        }
        // out tile of my warp, [16 tokens][16 kMt]: 32 bytes per token with the two 16-byte pieces swapped in every other group of four
        // tokens, or 64 bytes per token as in fused_kernel; rows out 16 / kMt tokens at a time (token lane / (2 kMt), piece lane % (2 kMt))
        const uint32_t o_tile = smem_u32(sm + L::kOut + warp * kMt * 512);
        auto o_piece = [&](int tok, int piece) {
            return o_tile + (uint32_t)(tok * 32 * kMt + ((piece ^ (kMt == 1 ? (tok >> 2) & 1 : (tok >> 1) & 3)) << 4));
        };
        uint32_t o_frag[kMt];
#pragma unroll
        for (int mt = 0; mt < kMt; ++mt) o_frag[mt] = o_piece(o_tok, 2 * mt + ((lane >> 3) & 1));
        const int my_tok = lane / (2 * kMt), my_piece = lane % (2 * kMt);
        const uint32_t o_row = o_piece(my_tok, my_piece);   // (kMt == 2: tokens 8 .. 15 are 512 bytes further, the same permutation)
        const int64_t o_step = kChunk * a.token_stride;
        __nv_bfloat16* og = a.out + (ch.bos + (int64_t)c0 * kChunk + my_tok) * a.token_stride + (int64_t)h * kD + row0 + 8 * my_piece;
        const int64_t st_base = ((ch.n * a.H + h) * (int64_t)kD + row0) * (int64_t)kD;   // element (row0, 0) of my rows
        uint4* const handover = reinterpret_cast<uint4*>(a.seg_state) + (chain * 8 + row0 / 16) * 256 + lane;   // + (8 mt + j) * 32

        WalkState<kMt, true> w;
        if (c0 > 0) {                       // handed over by the previous slab
#pragma unroll
            for (int mt = 0; mt < kMt; ++mt)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint4 x = __ldcg(handover + (8 * mt + j) * 32);
                    w.s[mt][j][0] = x.x; w.s[mt][j][1] = x.y; w.s[mt][j][2] = x.z; w.s[mt][j][3] = x.w;
                }
        } else if (a.initial_state != nullptr) {
            if (a.state_fp32) walk_load_tiles<kMt, true>(w.s, stage_tile, reinterpret_cast<const float*>(a.initial_state) + st_base, lane);
            else walk_load_tiles<kMt, false>(w.s, stage_tile, reinterpret_cast<const unsigned short*>(a.initial_state) + st_base, lane);
        } else {
            w.clear();
        }
        auto full_phase = [&](int p) { return (uint32_t)(((k0 + p) / kRowStages) & 1); };   // group p of this item
        WalkHead<kMt> hd;
        int left = (int)min((int64_t)0x7fffffff, ch.seq_len - (int64_t)c0 * kChunk);   // tokens from the current chunk on
        auto fetch_head = [&](int slot) {   // slot: kPair * stage + chunk of the stage
            hd.fetch(rec0 + slot * kTcRecord, wl);
#pragma unroll
            for (int mt = 0; mt < kMt; ++mt) ldmatrix_x4_t(hd.v[mt][0], hd.v[mt][1], hd.v[mt][2], hd.v[mt][3], v_off[mt] + slot * kRowVBytes);
        };
        const int n = c1 - c0;
        int s = k0 % kRowStages;   // stage of the current group
        if (n > 0) {
            if (__all_sync(0xffffffffu, mbar_wait_bounded(&ctl.full[s], full_phase(0), abort_flag, a.wait_ns)) == 0) failed = true;
            else {
                w.first(rec0 + s * kPair * kTcRecord, wl);
                fetch_head(s * kPair);
                hd.mask(left, lane & 3);
            }
        }
        bool ready = false;   // the next group's operands have been seen
        // Chunk i of the walk, in slot `slot`; `next`: the slot of the chunk after it, or `slot` where there is none.
        auto step = [&](int i, int slot, int next, auto&& look) {
            if (kExport && (c0 + i) % a.cs_every == 0) {   // the state before this group of chunks
                __nv_bfloat16* dst = a.chunk_states + ((ch.cs_slot0 + (c0 + i) / a.cs_every) * a.H + h) * (int64_t)(kD * kD) + (int64_t)row0 * kD;
#pragma unroll
                for (int mt = 0; mt < kMt; ++mt) walk_store_tile(w.s[mt], stage_tile, dst + mt * 16 * kD, false, lane);
            }
            uint32_t o[kMt][4];
            uint4 orow[kMt];
            const WalkHead<kMt> cur = hd;
            w.chunk(rec0 + slot * kTcRecord, rec0 + next * kTcRecord, wl, cur, o, [&](int j) {
                if (j == 3) fetch_head(next);
                if (j == 4) look();
                // the out rows: fragments through the warp's tile, 32 kMt contiguous bytes per token to global memory
                if (j == 3) {
#pragma unroll
                    for (int mt = 0; mt < kMt; ++mt) stmatrix_x4_t(o_frag[mt], o[mt][0], o[mt][1], o[mt][2], o[mt][3]);
                    __syncwarp();
                }
                if (j == 4) {
#pragma unroll
                    for (int e = 0; e < kMt; ++e) orow[e] = lds_u4(o_row + e * 512);
                }
                if (j == 6) {
                    hd.mask(left - kChunk, lane & 3);   // (some blocks behind the loads)
#pragma unroll
                    for (int e = 0; e < kMt; ++e) store_if(my_tok + 8 * e < left, og + e * 8 * a.token_stride, orow[e]);
                }
            });
            left -= kChunk;
            og += o_step;
        };
#pragma unroll 1
        for (int i = 0; i < n && !failed; i += kPair) {
            const int sn = s + 1 == kRowStages ? 0 : s + 1, slot = s * kPair;
            const int p = i / kPair + 1;   // the next group
            auto seen = [&](int st, int g) { return __all_sync(0xffffffffu, mbar_test_wait(&ctl.full[st], full_phase(g))) != 0; };
            const int left_n = n - i;
            const bool has_next = left_n > kPair;
            if constexpr (kPair == 2) {
                step(i, slot, left_n > 1 ? slot + 1 : slot, [&]() { ready = seen(sn, p); });
                __syncwarp();   // (every lane has read its piece of the out tile: the next chunk's rows may go in)
            }
            if (!(has_next & ready)) {   // (one branch that is rarely taken: a branch costs a lone warp some 25 cycles)
                if (kPair == 2 && left_n == 1) break;
                if (has_next && __all_sync(0xffffffffu, mbar_wait_bounded(&ctl.full[sn], full_phase(p), abort_flag, a.wait_ns)) == 0) { failed = true; break; }
            }
            step(i + kPair - 1, slot + kPair - 1, has_next ? sn * kPair : slot + kPair - 1, [&]() {
                if (kPair == 1) ready = seen(sn + 1 == kRowStages ? 0 : sn + 1, p + 1);
            });
            __syncwarp();
            mbar_arrive_lane0(&ctl.empty[s], lane);   // (my warp's last reads of this stage are done)
            s = sn;
        }
        if (!failed) {
            if (c1 < ch.n_chunks) {         // not the last slab
#pragma unroll
                for (int mt = 0; mt < kMt; ++mt)
#pragma unroll
                    for (int j = 0; j < 8; ++j) handover[(8 * mt + j) * 32] = make_uint4(w.s[mt][j][0], w.s[mt][j][1], w.s[mt][j][2], w.s[mt][j][3]);
            } else if (a.final_state != nullptr) {
#pragma unroll
                for (int mt = 0; mt < kMt; ++mt)
                    walk_store_tile(w.s[mt], stage_tile,
                                    a.state_fp32 ? (void*)(reinterpret_cast<float*>(a.final_state) + st_base + mt * 16 * kD)
                                                 : (void*)(reinterpret_cast<unsigned short*>(a.final_state) + st_base + mt * 16 * kD),
                                    a.state_fp32, lane);
            }
        } else {
            *abort_flag = 1;   // the other warps leave their waits
        }
    }
    if constexpr (kLoop) k0 += (max(0, c1 - c0) + kPair - 1) / kPair;
    }
    if (failed) atomicExch(a.status, FKDA_ERR_DEVICE_STATUS);
    __syncthreads();   // shared memory stays until every warp, and every copy of the control warp, is done with it
}

}  // namespace fkda
