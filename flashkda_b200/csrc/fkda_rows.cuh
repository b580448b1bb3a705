// Recurrence over chunk records in HBM / L2, row slices: a (sequence, head) chain is walked by kRowSplit CTAs of
// kRowWarps warps, each warp with 16 of the 128 state rows in registers (fkda_walk.cuh).  The warps of a chain share nothing
// but the records they read, so a chunk step has no barrier in it: every warp waits for the stage of its next chunk, walks
// it, and tells the control warp that it is done with the stage.
//
// Why this shape: with few chains the forward is a serial walk, (number of chunks) x (latency of a step).  A step is about
// 115 cycles of dependent latency (u', U, the first update) plus the products of one warp, 52 x 8 cycles of its scheduler's
// tensor pipe, and four warps put one on each scheduler.  The tcgen05 form of the same step (control warp, accumulators in
// tensor memory) took 2 100 cycles, of which 1 300 were hand-overs: tensor-memory loads and stores, commits, mbarriers.
// Included by fkda_tc.cu.
#pragma once

#include "fkda_walk.cuh"

namespace fkda {

constexpr int kRowWarps = 4;                      // walking warps per CTA, 16 state rows each
constexpr int kRowSplit = kD / (16 * kRowWarps);  // CTAs per chain
constexpr int kRowCols = 16 * kRowWarps;          // value columns (= state rows) of a CTA
constexpr int kRowThreads = (kRowWarps + 1) * 32;
constexpr int kRowVBytes = kChunk * kRowCols * 2;              // value tile [16 tokens][64] bf16, 128-byte swizzle
static_assert(kRowCols == 64 && kRowVBytes % 1024 == 0, "tile alignments");

// Shared memory of a CTA with kStages chunks in flight
template <int kStages>
struct RowSmem {
    static constexpr int kV = 0;                                        // value tiles (1024-byte aligned for the swizzle)
    static constexpr int kOut = kV + kStages * kRowVBytes;              // per warp an out tile [16 tokens][16] bf16
    static constexpr int kRec = kOut + kRowWarps * 512;                 // chunk records
    static constexpr int kStaging = kRec + kStages * kTcRecord;         // per warp one staging tile for states
    static constexpr int kCtrl = kStaging + kRowWarps * kWalkStageBytes;
    struct Ctrl {
        uint64_t full[kStages];    // operands of a chunk have landed (transaction bytes)
        uint64_t empty[kStages];   // a stage has been read by all walking warps
        int32_t abort_flag;
    };
    static constexpr int kBytes = kCtrl + (int)sizeof(Ctrl) + 1024;
    static_assert(kOut % 256 == 0 && kRec % 16 == 0 && kStaging % 16 == 0 && kCtrl % 8 == 0, "tile alignments");
};

// kExport: the states before every cs_every-th chunk are written out as well.  kLoop: a CTA takes several slices in turn
// (for launches that mostly return at once, see launch_tc; the loop alone makes a step 15 % longer).  kRowStages: 8 when every
// slice has an SM of its own (with the prepare stage of the next slab loading the memory, records arrive up to four steps
// late: 131 072 tokens, 32 heads: 4.58 -> 4.31 ms against 4 stages), otherwise 4, so that two CTAs fit an SM.
template <bool kExport, bool kLoop, int kRowStages>
__global__ void __launch_bounds__(kRowThreads, 2)
recurrence_rows_kernel(const __grid_constant__ TwoPassArgs a, const __grid_constant__ VMap map) {
    extern __shared__ uint8_t smem_dyn[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    using L = RowSmem<kRowStages>;
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
    }
    grid_dep_wait();
    // (a ragged batch that a one-kernel path has served: nothing to do)
    if (a.short_flag != nullptr && *a.short_flag != 0) return;
    __syncthreads();

    const int64_t n_items = a.N * a.H * kRowSplit;
    bool failed = false;
    int k0 = 0;   // chunks of the items before: the stages and their phases run on from item to item
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
            int t = c0;
            for (; t < c1; ++t) {
                const int k = k0 + t - c0, s = k % kRowStages;
                if (k >= kRowStages && !mbar_wait_bounded(&ctl.empty[s], (uint32_t)((k / kRowStages - 1) & 1), abort_flag, a.wait_ns)) {
                    failed = true;
                    break;
                }
                mbar_arrive_expect_tx(&ctl.full[s], (uint32_t)(kTcRecord + kRowVBytes));
                bulk_g2s(sm + L::kRec + s * kTcRecord, ch.rec_base + (int64_t)t * kTcRecord, kTcRecord, &ctl.full[s]);
                // rows past the end of the tensor arrive as zeros; rows of the next sequence are never used
                tma_load_3d(sm + L::kV + s * kRowVBytes, &map.v, slice * kRowCols, h, (int)(ch.bos + (int64_t)t * kChunk), &ctl.full[s]);
            }
            if (failed) {   // the copies in flight land before this CTA's shared memory goes
                *abort_flag = 1;
                for (int k = max(0, k0 + t - c0 - kRowStages); k < k0 + t - c0; ++k)
                    mbar_wait_bounded(&ctl.full[k % kRowStages], (uint32_t)((k / kRowStages) & 1), nullptr, 100000000ull);
            }
        }
        failed = __any_sync(0xffffffffu, failed) != 0;
    } else {
        // =========================== walking warps ===========================
        const int row0 = slice * kRowCols + warp * 16;   // my first state row
        const WalkLane wl = walk_lane(lane);
        uint8_t* stage_tile = sm + L::kStaging + warp * kWalkStageBytes;
        const uint32_t rec0 = smem_u32(sm + L::kRec);
        // my value columns in the [16 tokens][64] tile: token (lane & 7) + 8 (lane / 16), 16-byte piece 2 warp + (lane / 8) % 2
        const uint32_t v_off = smem_u32(sm + L::kV) + (uint32_t)(((lane & 7) + 8 * (lane >> 4)) * 128 + (((2 * warp + ((lane >> 3) & 1)) ^ (lane & 7)) << 4));
        // out tile of my warp, [16 tokens][16] with the two 16-byte pieces of a token swapped in every other group of four:
        // fragments in (token (lane & 7) + 8 (lane / 16), piece (lane / 8) % 2), rows out (token lane / 2, piece lane % 2)
        const int o_tok = (lane & 7) + 8 * (lane >> 4);
        const uint32_t o_tile = smem_u32(sm + L::kOut + warp * 512);
        const uint32_t o_frag = o_tile + (uint32_t)(o_tok * 32 + ((((lane >> 3) & 1) ^ ((o_tok >> 2) & 1)) << 4));
        const uint32_t o_row = o_tile + (uint32_t)((lane >> 1) * 32 + (((lane & 1) ^ ((lane >> 3) & 1)) << 4));
        const int64_t o_step = kChunk * a.token_stride;
        __nv_bfloat16* og = a.out + (ch.bos + (int64_t)c0 * kChunk + (lane >> 1)) * a.token_stride + (int64_t)h * kD + row0 + 8 * (lane & 1);
        const int64_t st_base = ((ch.n * a.H + h) * (int64_t)kD + row0) * (int64_t)kD;   // element (row0, 0) of my rows
        uint4* const handover = reinterpret_cast<uint4*>(a.seg_state) + (chain * 8 + slice * kRowWarps + warp) * 256 + lane;   // + j * 32

        WalkState<1> w;
        if (c0 > 0) {                       // handed over by the previous slab
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint4 x = __ldcg(handover + j * 32);
                w.s[0][j][0] = x.x; w.s[0][j][1] = x.y; w.s[0][j][2] = x.z; w.s[0][j][3] = x.w;
            }
        } else if (a.initial_state != nullptr) {
            if (a.state_fp32) walk_load_tiles<1, true>(w.s, stage_tile, reinterpret_cast<const float*>(a.initial_state) + st_base, lane);
            else walk_load_tiles<1, false>(w.s, stage_tile, reinterpret_cast<const unsigned short*>(a.initial_state) + st_base, lane);
        } else {
            w.clear();
        }
        auto full_bar = [&](int i) { return &ctl.full[(k0 + i) % kRowStages]; };
        auto full_phase = [&](int i) { return (uint32_t)(((k0 + i) / kRowStages) & 1); };
        auto wait_full = [&](int i) {
            return __all_sync(0xffffffffu, mbar_wait_bounded(full_bar(i), full_phase(i), abort_flag, a.wait_ns)) != 0;
        };
        WalkHead<1> hd;
        int left = (int)min((int64_t)0x7fffffff, ch.seq_len - (int64_t)c0 * kChunk);   // tokens from the current chunk on
        auto fetch_head = [&](int s, int tokens) {
            hd.fetch(rec0 + s * kTcRecord, wl);
            ldmatrix_x4_t(hd.v[0][0], hd.v[0][1], hd.v[0][2], hd.v[0][3], v_off + s * kRowVBytes);
            hd.mask(tokens, lane & 3);
        };
        const int n = c1 - c0;
        if (n > 0) {
            if (!wait_full(0)) failed = true;
            else {
                w.first(rec0 + k0 % kRowStages * kTcRecord, wl);
                fetch_head(k0 % kRowStages, left);
            }
        }
        int s = k0 % kRowStages;   // stage of the current chunk
        bool ready = false;   // the next chunk's operands have been seen
        for (int i = 0; i < n && !failed; ++i) {
            if (kExport && (c0 + i) % a.cs_every == 0)   // the state before this group of chunks
                walk_store_tile(w.s[0], stage_tile, a.chunk_states + ((ch.cs_slot0 + (c0 + i) / a.cs_every) * a.H + h) * (int64_t)(kD * kD) + (int64_t)row0 * kD,
                                false, lane);
            const uint32_t rec = rec0 + s * kTcRecord;
            const int sn = s + 1 == kRowStages ? 0 : s + 1;
            const bool has_next = i + 1 < n;
            if (has_next && !ready && !wait_full(i + 1)) { failed = true; break; }
            uint32_t o[1][4];
            uint4 orow;
            const WalkHead<1> cur = hd;
            w.chunk(rec, has_next ? rec0 + sn * kTcRecord : rec, wl, cur, o, [&](int j) {
                if (j == 3) fetch_head(has_next ? sn : s, left - kChunk);
                if (j == 4) ready = __all_sync(0xffffffffu, mbar_test_wait(full_bar(i + 2), full_phase(i + 2))) != 0;
                // the out rows: fragments through a 512-byte tile, 32 contiguous bytes per token to global memory
                if (j == 3) {
                    stmatrix_x4_t(o_frag, o[0][0], o[0][1], o[0][2], o[0][3]);
                    __syncwarp();
                }
                if (j == 4) orow = lds_u4(o_row);
                if (j == 6 && (lane >> 1) < left) *reinterpret_cast<uint4*>(og) = orow;
            });
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl.empty[s]);   // (my warp's last reads of this stage are done)
            s = sn;
            left -= kChunk;
            og += o_step;
        }
        if (!failed) {
            if (c1 < ch.n_chunks) {         // not the last slab
#pragma unroll
                for (int j = 0; j < 8; ++j) handover[j * 32] = make_uint4(w.s[0][j][0], w.s[0][j][1], w.s[0][j][2], w.s[0][j][3]);
            } else if (a.final_state != nullptr) {
                walk_store_tile(w.s[0], stage_tile,
                                a.state_fp32 ? (void*)(reinterpret_cast<float*>(a.final_state) + st_base)
                                             : (void*)(reinterpret_cast<unsigned short*>(a.final_state) + st_base),
                                a.state_fp32, lane);
            }
        } else {
            *abort_flag = 1;   // the other warps leave their waits
        }
    }
    if constexpr (kLoop) k0 += max(0, c1 - c0);
    }
    if (failed) atomicExch(a.status, FKDA_ERR_DEVICE_STATUS);
    __syncthreads();   // shared memory stays until every warp, and every copy of the control warp, is done with it
}

}  // namespace fkda
