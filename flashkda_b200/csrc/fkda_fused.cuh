// The whole forward in one persistent kernel, for batches with enough chains to fill the GPU: every SM walks one
// (sequence, head) chain at a time and prepares that chain's chunk operands itself, so that no chunk record ever leaves the SM
// (through HBM the records cost 1.8 KB per token and head on top of the 1.3 KB that the path cannot do without).
//
// Roles of a CTA (12 warps):
//   * warpgroup 0: four walking warps, 32 state rows each in registers (fkda_walk.cuh), one per scheduler.  Two row tiles per
//     warp halve the shared-memory reads of the chunk operands, which would otherwise be the limit;
//   * warpgroups 1, 2: eight preparing warps; warp w builds the records of the CTA's chunks w, w + 8, ... in a ring of
//     kFusedSlots blocks (fkda_prep.cuh), asks for the value tile and leaves a note on where the chunk belongs, so that the
//     walking warps spend nothing on addresses.  Chunks are handed over through mbarriers, slot by slot.
// Register shares: the walkers keep 232 registers per thread, the preparing warps 136 (128 x 232 + 256 x 136 = 384 x 168, what
// the CTA is launched with; 216 and 144: 1 % slower, 240 and 128: 2 to 3 %, 200 and 152: 1 to 3 %, 184 and 160: 12 %).  The build spills
// 20 bytes (76 of loads).
//
// Work split: the chunks of all chains form one line, chain after chain, cut into ranges of equal cost, one per CTA.  (Equal
// numbers of chunks leave the ranges with many short chains far behind: 640 chains of 1 to 16 chunks 110 us against 64, 3 200
// chains of 1 to 32 chunks 825 us against 506.)  A range that
// starts or ends inside a chain hands the chain's state over: a CTA walks the beginning of the chain that it shares
// with the CTA after it FIRST, then its whole chains, and last the end of the chain it shares with the CTA before it,
// whose state has then long been published.  Ranges are numbered by a ticket that a CTA draws when it starts, and a CTA waits
// only for the range before its own, i.e. for a CTA that is already running and whose first piece waits for nothing
// (or, with a chain longer than a range, for the range before that, and so on): no waiter depends on a CTA that has not
// started.  A chain longer than a range is walked range after range from time zero, which is its critical path.
//
// Bound by the latency of both roles beside each other: 0.57 instructions per cycle and scheduler, 64 % of the L1's wavefronts, tensor
// pipe 44 % (148 chains of 256 chunks, 0.30 ms); a chunk step takes 1.1 us.  In long runs the power cap takes the clock to 1.8 GHz.
// Included by fkda_tc.cu.
#pragma once

#include "fkda_prep.cuh"
#include "fkda_walk.cuh"

namespace fkda {

constexpr int kFusedWalkers = 4, kFusedMt = 2;             // walking warps, row tiles of 16 per warp
constexpr int kFusedPrep = 8;                              // preparing warps
constexpr int kFusedThreads = (kFusedWalkers + kFusedPrep) * 32;
constexpr int kFusedSlots = 11;                            // chunks in the ring: a record block and a value tile each
constexpr int kFusedCols = 16 * kFusedMt;                  // value columns (= state rows) of a walking warp
constexpr int kFusedVTile = kChunk * kD * 2;               // value tile: two halves [16 tokens][64] bf16, 128-byte swizzle
constexpr int kFusedV = 0;                                                         // 1024-byte aligned tiles
constexpr int kFusedOut = kFusedV + kFusedSlots * kFusedVTile;                     // per warp kFusedMt out tiles [16][16]
constexpr int kFusedStaging = kFusedOut + kFusedWalkers * kFusedMt * 512;          // per warp one staging tile for states
constexpr int kFusedRec = kFusedStaging + kFusedWalkers * kWalkStageBytes;         // the ring of records
constexpr int kFusedCtrl = kFusedRec + kFusedSlots * kTcRecord;

// The line of chunks: [lo, hi) is this CTA's range, walked as [b0, hi), [a1, b0), [lo, a1).
struct FusedRange {
    int64_t lo, hi, a1, b0;
    int64_t before;       // chunks of the chain at lo that other ranges walk first
    // position of unit u and the end of its run of consecutive positions
    __device__ __forceinline__ int64_t position(int u, int64_t* end) const {
        const int n1 = (int)(hi - b0), n2 = (int)(b0 - a1);
        if (u < n1) { *end = hi; return b0 + u; }
        if (u < n1 + n2) { *end = b0; return a1 + (u - n1); }
        *end = a1;
        return lo + (u - n1 - n2);
    }
};

// Chunks of each chain of a fixed batch; kSlab: of this launch, which walks only the first a.slab_chunks of them.
template <bool kSlab>
__device__ __forceinline__ int64_t fused_chunks(const TwoPassArgs& a) { return kSlab ? a.slab_chunks : (a.T + kChunk - 1) / kChunk; }

// The sequence that holds a position: its chunks of all heads are [begin, end) on the line, head after head.
struct FusedSeq {
    int64_t begin, end, bos, seq_len;
    int n, n_chunks;      // sequence; chunks of each of its chains
};
template <bool kSlab>
__device__ __forceinline__ FusedSeq fused_seq(const TwoPassArgs& a, int64_t p) {
    FusedSeq s;
    if (a.cu_seqlens != nullptr) {
        const int32_t* pre = a.tile_prefix;   // the chunks of sequence n start at position H * pre[n]
        const int64_t q = p / a.H;
        int64_t lo = 0, hi = a.N;             // the last n with pre[n] <= q (sequences without chunks drop out)
        while (hi - lo > 1) {
            const int64_t mid = (lo + hi) >> 1;
            if (pre[mid] <= q) lo = mid; else hi = mid;
        }
        s.n = (int)lo;
        s.n_chunks = pre[lo + 1] - pre[lo];
        s.begin = a.H * (int64_t)pre[lo];
        s.bos = a.cu_seqlens[lo];
        s.seq_len = a.cu_seqlens[lo + 1] - s.bos;
    } else {
        s.n_chunks = (int)fused_chunks<kSlab>(a);
        const int64_t per = a.H * s.n_chunks;
        s.n = (int)(p / per);
        s.begin = s.n * per;
        s.bos = s.n * a.T;
        s.seq_len = a.T;
    }
    s.end = s.begin + a.H * s.n_chunks;
    return s;
}
// Where range `range` starts.  The ranges are equal in cost, not in chunks: a chain counts a.chain_weight chunks more than it
// has, in front of its first one (a cut that falls there is a cut at the start of the chain).
template <bool kSlab>
__device__ __forceinline__ int64_t fused_bound(const TwoPassArgs& a, int range) {
    const int64_t w = a.chain_weight;
    const int64_t fixed = fused_chunks<kSlab>(a);
    const int64_t total = a.cu_seqlens != nullptr ? a.H * (a.tile_prefix[a.N] + w * a.N) : a.N * a.H * (fixed + w);
    const int64_t x = total * range / gridDim.x;
    if (a.cu_seqlens == nullptr) return x / (fixed + w) * fixed + max((int64_t)0, x % (fixed + w) - w);
    const int32_t* pre = a.tile_prefix;
    const int64_t q = x / a.H;
    int64_t lo = 0, hi = a.N;   // the last n whose chains start at or before x
    while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (pre[mid] + w * mid <= q) lo = mid; else hi = mid;
    }
    const int64_t n_chunks = pre[lo + 1] - pre[lo];
    const int64_t at = x - a.H * (pre[lo] + w * lo);
    return a.H * (int64_t)pre[lo] + min(a.H, at / (n_chunks + w)) * n_chunks + (at < a.H * (n_chunks + w) ? max((int64_t)0, at % (n_chunks + w) - w) : 0);
}
template <bool kSlab>
__device__ __forceinline__ FusedRange fused_range(const TwoPassArgs& a, int range) {
    FusedRange r;
    r.lo = fused_bound<kSlab>(a, range);
    r.hi = fused_bound<kSlab>(a, range + 1);
    r.a1 = r.lo;
    r.before = 0;
    r.b0 = r.hi;
    if (r.lo < r.hi) {
        const FusedSeq f = fused_seq<kSlab>(a, r.lo), l = fused_seq<kSlab>(a, r.hi - 1);
        const int64_t first = r.lo - (r.lo - f.begin) % f.n_chunks;            // starts of the chains that hold the ends
        const int64_t last = r.hi - 1 - (r.hi - 1 - l.begin) % l.n_chunks;
        r.before = r.lo - first;
        if (first < r.lo) r.a1 = min(r.hi, first + f.n_chunks);
        if (r.hi < last + l.n_chunks) r.b0 = max(r.a1, last);
    }
    return r;
}

// What the walking warps need to know about a chunk, left beside its record by the warp that prepared it.
struct FusedInfo {
    int64_t tok0;         // first token
    int n, h;             // sequence, head
    int chunk;            // index in the chain
    int left;             // tokens of the chain from this chunk on
    int rest;             // chunks from this one to the end of the piece (a run of chunks of one chain inside a range)
    int last;             // whether the piece ends with the chain
};

struct FusedCtrl {
    uint64_t full[kFusedSlots];    // a record is complete and its value tile has landed
    uint64_t empty[kFusedSlots];   // a slot has been read by all walking warps
    FusedInfo info[kFusedSlots];
    int32_t range;
    int32_t abort_flag;
};
constexpr int kFusedSmemBytes = kFusedCtrl + (int)sizeof(FusedCtrl) + 1024;
// Two producers may wait on one slot, for units a whole round apart, but the later one only after the unit before the earlier
// one's was consumed (it had to be, for the later one's previous unit to get its slot): with more producers than slots that
// no longer holds and the parities of the rounds become ambiguous.
static_assert(kFusedPrep <= kFusedSlots, "no more preparing warps than slots");
static_assert(kFusedVTile == 4096 && kFusedWalkers * kFusedCols == kD && kFusedOut % 256 == 0 && kFusedStaging % 16 == 0 &&
              kFusedRec % 16 == 0 && kFusedCtrl % 8 == 0 && kFusedSmemBytes <= 232448, "shared-memory layout");

template <int kRegs>
__device__ __forceinline__ void reg_alloc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs)); }
template <int kRegs>
__device__ __forceinline__ void reg_dealloc() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs)); }

__device__ __forceinline__ int load_acquire(const int32_t* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// kExport: the states before every cs_every-th chunk are written out as well.  kSlab: only the first a.slab_chunks chunks of every
// chain are walked, one chain per CTA, and the states handed on to the row-slice kernel (see launch_mid)
template <bool kExport, bool kSlab>
__global__ void __launch_bounds__(kFusedThreads, 1)
fused_kernel(const __grid_constant__ TwoPassArgs a, const __grid_constant__ VMap map) {
    extern __shared__ uint8_t smem_dyn[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    FusedCtrl& ctl = *reinterpret_cast<FusedCtrl*>(sm + kFusedCtrl);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    volatile int* abort_flag = &ctl.abort_flag;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kFusedSlots; ++s) {
            mbar_init(&ctl.full[s], 2);
            mbar_init(&ctl.empty[s], kFusedWalkers);
        }
        ctl.abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_map(&map.v);
    }
    grid_dep_wait();
    if (threadIdx.x == 0) ctl.range = atomicAdd(a.queue, 1);
    __syncthreads();
    const int range = ctl.range;
    const FusedRange r = fused_range<kSlab>(a, range);
    const int n_units = (int)(r.hi - r.lo);
    // The chain at lo reaches this range when the ranges before have walked its beginning, at a microsecond per chunk: with a
    // chain much longer than a range that alone may take longer than the limit of a wait, which is for what never comes.
    const uint64_t wait_ns = a.wait_ns + 8000ull * (uint64_t)r.before;
    bool failed = false;

    if (warp >= kFusedWalkers) {
        // =========================== preparing warps ===========================
        reg_dealloc<136>();
        FusedSeq sq;          // the sequence of the current unit
        sq.begin = sq.end = sq.n_chunks = -1;
        int h = 0, t = 0;     // its head and chunk
        int64_t p = 0, end = 0;   // its position and the end of the run of positions it belongs to
        for (int u = warp - kFusedWalkers; u < n_units; u += kFusedPrep) {
            p += kFusedPrep;
            t += kFusedPrep;
            if (t >= sq.n_chunks || p >= end) {   // another chain, or another run
                p = r.position(u, &end);
                if (p < sq.begin || p >= sq.end) sq = fused_seq<kSlab>(a, p);
                const int at = (int)(p - sq.begin);
                h = at / sq.n_chunks;
                t = at - h * sq.n_chunks;
            }
            const int64_t t0 = sq.bos + (int64_t)t * kChunk;
            const int len = (int)min((int64_t)kChunk, sq.seq_len - (int64_t)t * kChunk);
            if (t == 0 && a.initial_state != nullptr) {   // the state that the walking warps will load in a while
                const int bytes = kD * kD * (a.state_fp32 ? 4 : 2);
                const char* st = reinterpret_cast<const char*>(a.initial_state) + ((int64_t)sq.n * a.H + h) * bytes;
                for (int off = lane * 128; off < bytes; off += 32 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(st + off));
            }
            PrepHead x;
            const PrepSrc src = prep_src(a, t0, len, h, lane);
            prep_load(a, src, t0, len, h, lane, x);
            const int slot = u % kFusedSlots;
            const uint32_t phase = 1u ^ ((u / kFusedSlots) & 1);   // of empty[slot]: the first round finds the slots free
            uint8_t* rec = sm + kFusedRec + slot * kTcRecord;
            auto acquire = [&]() {   // the slot is free: leave the note and ask for the value tile
                if (__all_sync(0xffffffffu, mbar_wait_bounded(&ctl.empty[slot], phase, abort_flag, wait_ns)) == 0) return false;
                if (lane == 0) {
                    FusedInfo& f = ctl.info[slot];
                    f.tok0 = t0;
                    f.n = sq.n; f.h = h; f.chunk = t;
                    f.left = (int)min((int64_t)0x7fffffff, sq.seq_len - (int64_t)t * kChunk);
                    f.rest = (int)min(end - p, (int64_t)(sq.n_chunks - t));
                    f.last = f.rest == sq.n_chunks - t;
                    // rows past the end of the tensor arrive as zeros; rows of the next sequence are never used
                    mbar_arrive_expect_tx(&ctl.full[slot], kFusedVTile);
                    tma_load_3d(sm + kFusedV + slot * kFusedVTile, &map.v, 0, h, (int)t0, &ctl.full[slot]);
                    tma_load_3d(sm + kFusedV + slot * kFusedVTile + kFusedVTile / 2, &map.v, kD / 2, h, (int)t0, &ctl.full[slot]);
                }
                __syncwarp();
                return true;
            };
            if (!prep_compute<false, false>(a, src, len, rec, lane, x, acquire, [] {})) {
                failed = true;
                *abort_flag = 1;
                // my value tiles in flight (of my last units, as many as there are slots) land before this CTA's shared memory goes
                for (int v = u - kFusedPrep; v >= 0 && v > u - kFusedSlots - kFusedPrep; v -= kFusedPrep)
                    mbar_wait_bounded(&ctl.full[v % kFusedSlots], (uint32_t)((v / kFusedSlots) & 1), nullptr, 100000000ull);
                break;
            }
            mbar_arrive_lane0(&ctl.full[slot], lane);
        }
    } else {
        // =========================== walking warps ===========================
        reg_alloc<232>();
        const int row0 = warp * kFusedCols;   // my first state row
        const WalkLane wl = walk_lane(lane);
        uint8_t* stage_tile = sm + kFusedStaging + warp * kWalkStageBytes;
        const uint32_t rec0 = smem_u32(sm + kFusedRec);
        // my value columns: token (lane & 7) + 8 (lane / 16), 16-byte piece 4 (warp & 1) + 2 mt + (lane / 8) % 2 of half warp / 2
        uint32_t v_off[kFusedMt];
        const int v_tok = (lane & 7) + 8 * (lane >> 4);
#pragma unroll
        for (int mt = 0; mt < kFusedMt; ++mt)
            v_off[mt] = smem_u32(sm + kFusedV) + (uint32_t)((warp >> 1) * (kFusedVTile / 2) + v_tok * 128 +
                                                            (((4 * (warp & 1) + 2 * mt + ((lane >> 3) & 1)) ^ (lane & 7)) << 4));
        // out tile of my warp, [16 tokens][32], 64 bytes per token with its 16-byte pieces permuted by the token: fragments of row tile
        // mt in (token v_tok, piece 2 mt + (lane / 8) % 2), rows out eight tokens at a time (token lane / 4, piece lane % 4), so that a
        // store touches eight lines, not sixteen (each takes a pass through the L1 of its own)
        const uint32_t o_tile = smem_u32(sm + kFusedOut + warp * kFusedMt * 512);
        auto o_piece = [&](int tok, int piece) { return o_tile + (uint32_t)(tok * 64 + ((piece ^ ((tok >> 1) & 3)) << 4)); };
        uint32_t o_frag[kFusedMt];
#pragma unroll
        for (int mt = 0; mt < kFusedMt; ++mt) o_frag[mt] = o_piece(v_tok, 2 * mt + ((lane >> 3) & 1));
        const uint32_t o_row = o_piece(lane >> 2, lane & 3);   // tokens 8 .. 15: 512 bytes further (the same permutation)
        const int64_t o_step = kChunk * a.token_stride;

        WalkState<kFusedMt> w;
        WalkHead<kFusedMt> hd;
        int slot = 0;             // ring slot of the current unit
        uint32_t phase = 0;       // of full[slot]
        auto wait_full = [&](int sl, uint32_t ph) { return __all_sync(0xffffffffu, mbar_wait_bounded(&ctl.full[sl], ph, abort_flag, wait_ns)) != 0; };
        FusedInfo pc;   // of the first chunk of the current piece
        for (int u = 0; u < n_units; u += pc.rest) {
            if (!wait_full(slot, phase)) { failed = true; break; }
            pc = ctl.info[slot];
            const int64_t st_base = ((pc.n * a.H + pc.h) * (int64_t)kD + row0) * (int64_t)kD;   // element (row0, 0) of my rows
            // ---- the state this piece starts from ----
            if (pc.chunk > 0) {   // published by the range before this one (the last one that holds any chunks)
                int before = range - 1;
                while (before > 0 && fused_bound<kSlab>(a, before) == r.lo) --before;
                const uint64_t begin = global_timer_ns();
                uint32_t spins = 0;
                while (load_acquire(a.range_flags + before) < kFusedWalkers) {
                    if ((++spins & 15u) == 0 && (*abort_flag != 0 || global_timer_ns() - begin > wait_ns)) { failed = true; break; }
                    __nanosleep(100);
                }
                if (__any_sync(0xffffffffu, failed)) { failed = true; break; }
                const uint4* src = reinterpret_cast<const uint4*>(a.seg_state) + ((int64_t)before * kFusedWalkers + warp) * (kFusedMt * 256) + lane;
#pragma unroll
                for (int mt = 0; mt < kFusedMt; ++mt)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint4 x = __ldcg(src + (mt * 8 + j) * 32);
                        w.s[mt][j][0] = x.x; w.s[mt][j][1] = x.y; w.s[mt][j][2] = x.z; w.s[mt][j][3] = x.w;
                    }
            } else if (a.initial_state != nullptr) {
                if (a.state_fp32) walk_load_tiles<kFusedMt, true>(w.s, stage_tile, reinterpret_cast<const float*>(a.initial_state) + st_base, lane);
                else walk_load_tiles<kFusedMt, false>(w.s, stage_tile, reinterpret_cast<const unsigned short*>(a.initial_state) + st_base, lane);
            } else {
                w.clear();
            }
            // ---- the piece's chunks ----
            const int64_t cs_slot0 = kExport ? cs_first_slot(a, pc.n) : 0;
            int left = pc.left;   // tokens from the current chunk on
            __nv_bfloat16* og = a.out + (pc.tok0 + (lane >> 2)) * a.token_stride + (int64_t)pc.h * kD + row0 + 8 * (lane & 3);
            auto fetch_head = [&](int sl, int tokens) {
                hd.fetch(rec0 + sl * kTcRecord, wl);
#pragma unroll
                for (int mt = 0; mt < kFusedMt; ++mt)
                    ldmatrix_x4_t(hd.v[mt][0], hd.v[mt][1], hd.v[mt][2], hd.v[mt][3], v_off[mt] + sl * kFusedVTile);
                hd.mask(tokens, lane & 3);
            };
            w.first(rec0 + slot * kTcRecord, wl);
            fetch_head(slot, left);
            bool ready = false;   // the next chunk's slot has been seen complete
#pragma unroll 1
            for (int i = 0; i < pc.rest; ++i) {
                if (kExport && (pc.chunk + i) % a.cs_every == 0) {   // the state before this group of chunks
                    __nv_bfloat16* dst = a.chunk_states + ((cs_slot0 + (pc.chunk + i) / a.cs_every) * a.H + pc.h) * (int64_t)(kD * kD) + (int64_t)row0 * kD;
#pragma unroll
                    for (int mt = 0; mt < kFusedMt; ++mt) walk_store_tile(w.s[mt], stage_tile, dst + mt * 16 * kD, false, lane);
                }
                const uint32_t rec = rec0 + slot * kTcRecord;
                int sn = slot + 1;
                uint32_t pn = phase;
                if (sn == kFusedSlots) { sn = 0; pn ^= 1u; }
                const bool has_next = i + 1 < pc.rest;
                if (has_next && !ready && !wait_full(sn, pn)) { failed = true; break; }
                int s2 = sn + 1;   // the slot after the next one
                uint32_t p2 = pn;
                if (s2 == kFusedSlots) { s2 = 0; p2 ^= 1u; }
                uint32_t o[kFusedMt][4];
                uint4 orow[2];
                const WalkHead<kFusedMt> cur = hd;
                w.chunk(rec, has_next ? rec0 + sn * kTcRecord : rec, wl, cur, o, [&](int j) {
                    if (j == 3) {
                        fetch_head(has_next ? sn : slot, left - kChunk);
                        // the out rows: fragments through the tile, 64 contiguous bytes per token to global memory
#pragma unroll
                        for (int mt = 0; mt < kFusedMt; ++mt) stmatrix_x4_t(o_frag[mt], o[mt][0], o[mt][1], o[mt][2], o[mt][3]);
                        __syncwarp();
                    }
                    if (j == 4) {
                        ready = __all_sync(0xffffffffu, mbar_test_wait(&ctl.full[s2], p2)) != 0;
#pragma unroll
                        for (int i = 0; i < 2; ++i) orow[i] = lds_u4(o_row + i * 512);
                    }
                    if (j == 6) {
#pragma unroll
                        for (int i = 0; i < 2; ++i) store_if((lane >> 2) + 8 * i < left, og + i * 8 * a.token_stride, orow[i]);
                    }
                });
                __syncwarp();
                mbar_arrive_lane0(&ctl.empty[slot], lane);   // (my warp's last reads of this slot are done)
                slot = sn;
                phase = pn;
                left -= kChunk;
                og += o_step;
            }
            if (failed) break;
            // ---- the state leaves: to the next range, or as the final state ----
            if (!pc.last) {
                uint4* dst = reinterpret_cast<uint4*>(a.seg_state) + ((int64_t)range * kFusedWalkers + warp) * (kFusedMt * 256) + lane;
#pragma unroll
                for (int mt = 0; mt < kFusedMt; ++mt)
#pragma unroll
                    for (int j = 0; j < 8; ++j) dst[(mt * 8 + j) * 32] = make_uint4(w.s[mt][j][0], w.s[mt][j][1], w.s[mt][j][2], w.s[mt][j][3]);
                __threadfence();
                __syncwarp();
                if (lane == 0 && !a.test_drop_push) atomicAdd(a.range_flags + range, 1);
            } else if (kSlab) {
                uint4* dst = reinterpret_cast<uint4*>(a.seg_state) + ((pc.n * a.H + pc.h) * 8 + row0 / 16) * 256 + lane;
#pragma unroll
                for (int mt = 0; mt < kFusedMt; ++mt)
#pragma unroll
                    for (int j = 0; j < 8; ++j) dst[(mt * 8 + j) * 32] = make_uint4(w.s[mt][j][0], w.s[mt][j][1], w.s[mt][j][2], w.s[mt][j][3]);
            } else if (a.final_state != nullptr) {
#pragma unroll
                for (int mt = 0; mt < kFusedMt; ++mt)
                    walk_store_tile(w.s[mt], stage_tile,
                                    a.state_fp32 ? (void*)(reinterpret_cast<float*>(a.final_state) + st_base + mt * 16 * kD)
                                                 : (void*)(reinterpret_cast<unsigned short*>(a.final_state) + st_base + mt * 16 * kD),
                                    a.state_fp32, lane);
            }
        }
        // sequences without tokens are not on the line: their state passes through (rounded to bf16, as everywhere)
        if (!failed && a.cu_seqlens != nullptr && a.final_state != nullptr) {
            for (int64_t n = blockIdx.x; n < a.N; n += gridDim.x) {
                if (a.cu_seqlens[n + 1] > a.cu_seqlens[n]) continue;
                for (int h = 0; h < (int)a.H; ++h) {
                    const int64_t at = ((n * a.H + h) * (int64_t)kD + row0) * (int64_t)kD;
                    if (a.initial_state == nullptr)
                        w.clear();
                    else if (a.state_fp32)
                        walk_load_tiles<kFusedMt, true>(w.s, stage_tile, reinterpret_cast<const float*>(a.initial_state) + at, lane);
                    else
                        walk_load_tiles<kFusedMt, false>(w.s, stage_tile, reinterpret_cast<const unsigned short*>(a.initial_state) + at, lane);
#pragma unroll
                    for (int mt = 0; mt < kFusedMt; ++mt)
                        walk_store_tile(w.s[mt], stage_tile, a.state_fp32 ? (void*)(reinterpret_cast<float*>(a.final_state) + at + mt * 16 * kD)
                                                                          : (void*)(reinterpret_cast<unsigned short*>(a.final_state) + at + mt * 16 * kD),
                                        a.state_fp32, lane);
                }
            }
        }
    }
    if (failed) {
        *abort_flag = 1;
        atomicExch(a.status, FKDA_ERR_DEVICE_STATUS);
    }
    __syncthreads();
}

}  // namespace fkda
