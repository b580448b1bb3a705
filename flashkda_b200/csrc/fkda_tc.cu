// Tensor-core KDA forward for sm_100a: dispatch and launches.
//
// The forms of the forward, all on the same chunk operands (a 14 656-byte record per (chunk, head), fkda_common.cuh), the same
// chunk step on mma.sync with the state in registers (fkda_walk.cuh), and with bit-identical results:
//   * fkda_fused.cuh: one persistent kernel whose CTAs prepare the records in shared memory and walk them, for batches with
//     enough chains to fill the GPU: no record ever reaches HBM;
//   * fkda_prepare_warp.cuh + fkda_rows.cuh: a prepare kernel writes the records to the workspace, a recurrence kernel walks
//     row slices of the chains; the slices of few chains spread over more SMs than there are chains, and the prepare stage of
//     later chunks runs on the SMs that are left (the slab pipeline below);
//   * both, for chains that leave SMs idle in the first form and have none for slices (launch_mid).
// An earlier form of both recurrences ran the products on tcgen05 with accumulators in tensor memory: the hand-overs between
// registers and tensor memory (a store takes 180 cycles, a commit and its wait as long) cost more than products that are 16 to
// 128 columns wide and 16 deep take on mma.sync (a chunk step of one chain per SM: 1.11 us against 0.52).
//
// Numerics: steps B1-B7 of the reference's contract (tests/torch_ref.py:231-251; the reference's own recurrence is
// csrc/smxx/fwd_kernel2.cuh:434-742).
#include <cuda.h>
#include <string.h>

#include <mutex>

#include "fkda_common.cuh"
#include "fkda_internal.h"
#include "fkda_prepare_warp.cuh"
#include "fkda_sm100.cuh"

namespace fkda {

using namespace sm100;

// Where the tokens and records of one (sequence, head) chain live.
struct TcChain {
    int64_t n;        // sequence
    int h;            // head
    int64_t bos;      // first token
    int64_t seq_len;
    int n_chunks;
    const uint8_t* rec_base;  // record of the chain's chunk 0
    int64_t cs_slot0;         // first state-export slot of the sequence (valid when chunk_states is given)
};
__device__ __forceinline__ TcChain tc_locate_chain(const TwoPassArgs& a, int64_t chain) {
    TcChain c;
    const int64_t s = chain / a.H;  // position in the order the chains are started in
    c.h = (int)(chain - s * a.H);
    c.n = a.seq_order != nullptr ? a.seq_order[s] : s;
    int64_t tile_base;
    if (a.cu_seqlens != nullptr) {
        c.bos = a.cu_seqlens[c.n];
        c.seq_len = a.cu_seqlens[c.n + 1] - c.bos;
        if (c.seq_len < 0) c.seq_len = 0;
        tile_base = a.tile_prefix[c.n];
    } else {
        c.bos = c.n * a.T;
        c.seq_len = a.T;
        tile_base = c.n * ((a.T + kChunk - 1) / kChunk);
    }
    c.n_chunks = (int)((c.seq_len + kChunk - 1) / kChunk);
    c.rec_base = a.workspace + ((int64_t)c.h * a.total_tiles + tile_base) * (int64_t)kTcRecord;
    c.cs_slot0 = a.chunk_states != nullptr ? cs_first_slot(a, c.n) : 0;
    return c;
}

}  // namespace fkda

#include "fkda_fused.cuh"
#include "fkda_rows.cuh"

namespace fkda {

// ---------------------------------------------------------------------------------
// SM count of the current device (B200: 148), cached per device; 148 when no device can be asked (sizing calls
// on a machine without a GPU).
int device_sm_count() {
    static int cache[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (cache[dev] == 0) {
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 148;
        cache[dev] = sms;
    }
    return cache[dev];
}

constexpr int kRowSplit = row_split(4, 1);   // CTAs per chain of the row-slice kernel, unless there are SMs for more
constexpr size_t kStateBytes = (size_t)kD * kD * 2;   // a chain's state as bf16 (hand-over buffers)

// Few chains on a fixed batch may run as a slab pipeline (see launch_tc): at least 32 SMs are left beside the row slices.
static bool slabs_possible(int64_t chains, int sms) { return chains * kRowSplit <= sms - 32; }

// The one-kernel forward serves whole forwards with more than one chunk per chain on average and more row slices than SMs.
// While every slice has an SM of its own, a step of the row-slice kernel takes 0.45 us against 1.1 us here, which pays for the
// prepare kernel in front of it (chains of 512 chunks, one prepare and one recurrence kernel against this: 64 chains 395 us, 567;
// 74 chains 421, 568; 80 chains 627, 568; 96 chains 667, 568).  A ragged batch whose lengths the host does not know may consist of
// a few long chains, whose walk is then the whole time (128 chains of 1 to 32 chunks: 45.5 us in two kernels against 52.8): it needs
// two chains per SM, or 1.6 with more than ten chunks per sequence on average (256 and 288 chains of even lengths: 16 chunks 67, 68
// us in two kernels against 52, 57; 256 chunks 756, 804 against 504, 565; the 4 chunks per sequence that the line keeps out are as fast
// here by now, 28.4, 29.7 against 25.8, 28.8).  With fp32 states to load and to store, which nothing hides here, it needs more than
// four chunks per sequence on average (3 840 chains of 2 chunks 199 us in two kernels against 215, of 4 chunks 277 against 268, of 5
// chunks 319 against 298).
static bool fused_eligible(const fkda_fwd_params& p, int sms) {
    if (p.phase_mask != 0 || p.B * p.T <= kChunk * p.N) return false;
    if (p.flags & FKDA_FLAG_NO_WIDE) return true;
    const int64_t chains = p.N * p.H, tokens = p.B * p.T;
    if (p.state_dtype == FKDA_STATE_FP32 && p.initial_state != nullptr && p.final_state != nullptr && tokens <= 4 * kChunk * p.N) return false;
    if (p.cu_seqlens == nullptr) return chains * kRowSplit > sms;
    return chains >= 2 * sms || (5 * chains >= 8 * sms && tokens > 10 * kChunk * p.N);
}
static size_t fused_flag_bytes(int sms) { return (size_t)(sms * 4 + 255) / 256 * 256; }
// header | prefix tables | one flag and one hand-over state per range
static size_t fused_bytes(int64_t N, int sms) { return kWsHeaderBytes + ws_prefix_bytes(N) + fused_flag_bytes(sms) + (size_t)sms * kStateBytes; }

// The two-kernel form: header | prefix tables | hand-over states of the slab pipeline | records.  A function of the shapes
// only, not of phase_mask or flags, so that calls which share a workspace find the records in the same place.
struct TcCarve {
    size_t states, records;
};
static TcCarve tc_carve(const fkda_fwd_params& p, int sms) {
    const int64_t chains = p.N * p.H;
    const bool varlen = p.cu_seqlens != nullptr;
    TcCarve c;
    c.states = !varlen && slabs_possible(chains, sms) ? (size_t)chains * kStateBytes : 0;
    const int64_t tiles = varlen ? ws_tiles_upper_bound(p.B * p.T, p.N) : p.N * ((p.T + kChunk - 1) / kChunk);
    c.records = (size_t)p.H * (size_t)tiles * (size_t)kTcRecord;
    return c;
}

// Fewer chains than SMs, but too many for two SMs each: launch_mid, while its records take no more than a gigabyte.  The three kernel
// boundaries cost some 12 us, and what is won grows with the chunks and with the idle SMs: the line lies where the two meet (time of
// the one kernel over this, 75 to 124 chains by chunks x idle SMs, without exported states: 4 650 .. 4 700: 0.98 to 1.015, 5 200:
// 1.00 to 1.03, 7 000: 1.01 to 1.08, 8 800: 1.025 to 1.12).  With exported states the line lies higher: the stores of a state hold a walking
// warp up in both, in the one kernel partly while it would wait for its preparing warps (4 650 .. 4 850: 0.94 to 0.98, 5 800: 0.98 to
// 0.99, 7 000: 0.99 to 1.03, 9 200: 1.00 to 1.07, from every chunk to every 16th exported).
constexpr size_t kMidBytesMost = (size_t)1 << 30;
static size_t mid_bytes(const fkda_fwd_params& p, int sms) {
    const int64_t chains = p.N * p.H, tps = (p.T + kChunk - 1) / kChunk;
    return kWsHeaderBytes + ws_prefix_bytes(p.N) + fused_flag_bytes(sms) + (size_t)chains * kStateBytes + (size_t)(chains * tps) * kTcRecord;
}
static bool mid_eligible(const fkda_fwd_params& p, int sms) {
    const int64_t chains = p.N * p.H;
    return p.cu_seqlens == nullptr && p.phase_mask == 0 && !(p.flags & (FKDA_FLAG_NO_WIDE | FKDA_FLAG_NO_SLABS)) && chains * kRowSplit > sms &&
           chains + 24 <= sms && p.T > 63 * kChunk && (p.T + kChunk - 1) / kChunk * (sms - chains) >= (p.chunk_states == nullptr ? 4608 : 6912) &&
           mid_bytes(p, sms) <= kMidBytesMost;
}

// Names the records that a call writes or expects: everything that decides where each of them lies.
static uint64_t records_tag(const fkda_fwd_params& p) {
    uint64_t x = p.cu_seqlens != nullptr ? 2 : 1;
    for (const int64_t y : {p.B, p.T, p.H, p.N}) x = (x ^ (uint64_t)y) * 0x9e3779b97f4a7c15ull, x ^= x >> 29;
    return x | 1;
}

// Upper bound over every call with these totals (the caller may not know yet whether the batch is ragged).
size_t tc_workspace_bytes(int64_t T_total, int64_t H, int64_t N) {
    const int sms = device_sm_count();
    const size_t two_pass = kWsHeaderBytes + ws_prefix_bytes(N) + (H * N < sms ? fused_flag_bytes(sms) + (size_t)(H * N) * kStateBytes : 0) +
                            (size_t)H * (size_t)ws_tiles_upper_bound(T_total, N) * (size_t)kTcRecord;
    const size_t fused = fused_bytes(N, sms);
    return two_pass > fused ? two_pass : fused;
}

// What one particular call needs.
size_t tc_workspace_bytes_for(const fkda_fwd_params& p) {
    if (decode_eligible(p) || short_eligible(p)) return 0;   // one kernel, nothing staged
    const int sms = device_sm_count();
    if (fused_eligible(p, sms)) return fused_bytes(p.N, sms);
    const TcCarve c = tc_carve(p, sms);
    return kWsHeaderBytes + ws_prefix_bytes(p.N) + c.states + c.records;
}

// What a call makes use of: more than it needs where records of the later chunks make it faster.
size_t tc_workspace_bytes_wanted(const fkda_fwd_params& p) {
    const int sms = device_sm_count();
    const size_t need = tc_workspace_bytes_for(p);
    return need > 0 && mid_eligible(p, sms) && mid_bytes(p, sms) > need ? mid_bytes(p, sms) : need;
}

// Calls that a host thread makes on the library's own streams concern no stream of the caller: another thread's capture in the
// strict mode does not forbid them.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Side stream and events, one set per device for the slab pipeline and one for launch_mid, created on first use.
constexpr int kMaxSlabs = 4;
enum SideUse { kSideSlabs, kSideMid, kSideUses };
struct SlabStreams {
    std::mutex launch_mu;  // one call at a time is ENQUEUED per set (event record / wait pairs stay paired)
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, done[kMaxSlabs] = {nullptr, nullptr, nullptr, nullptr};
    unsigned long long user = 0;   // id of the stream whose call was the last to put work on the side stream (side_free)
    bool ready = false;
};
static SlabStreams* slab_streams(int dev, SideUse use) {
    static std::mutex mu;
    static SlabStreams table[64][kSideUses];
    if (dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    SlabStreams& t = table[dev][use];
    if (!t.ready) {
        const RelaxedCapture relaxed;
        if (cudaStreamCreateWithFlags(&t.side, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
        if (cudaEventCreateWithFlags(&t.fork, cudaEventDisableTiming) != cudaSuccess) return nullptr;
        for (int i = 0; i < kMaxSlabs; ++i)
            if (cudaEventCreateWithFlags(&t.done[i], cudaEventDisableTiming) != cudaSuccess) return nullptr;
        t.ready = true;
    }
    return &t;
}

// Whether a call on `stream` gets the side stream to itself (launch_mu is held): not while it belongs to another thread's capture,
// nor while it carries another stream's work, which would put this call behind whatever that stream waits for.
static bool side_free(SlabStreams& t, cudaStream_t stream) {
    auto ok = [](cudaError_t e) { return e == cudaSuccess || (cudaGetLastError(), false); };   // (a refusal here is not the call's)
    cudaStreamCaptureStatus side = cudaStreamCaptureStatusNone, mine = cudaStreamCaptureStatusNone;
    unsigned long long side_id = 0, my_id = 0;
    if (!ok(cudaStreamGetCaptureInfo(t.side, &side, &side_id)) || !ok(cudaStreamGetCaptureInfo(stream, &mine, &my_id))) return false;
    if (side != cudaStreamCaptureStatusNone) return side == cudaStreamCaptureStatusActive && mine == side && my_id == side_id;
    if (mine != cudaStreamCaptureStatusNone) return true;   // (the graph depends on nothing that was enqueued before it)
    unsigned long long user = 0;
    if (!ok(cudaStreamGetId(stream, &user))) return false;
    if (t.user != user) {
        const RelaxedCapture relaxed;
        if (!ok(cudaStreamQuery(t.side))) return false;
        t.user = user;
    }
    return true;
}

// The driver entry point is looked up through the runtime (no link-time dependency on libcuda, so
// the library also loads on a machine without a driver).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

static bool encode_map(CUtensorMap* m, CUtensorMapDataType type, int rank, const void* base, const cuuint64_t* dims,
                       const cuuint64_t* strides, const cuuint32_t* box) {
    EncodeTiledFn encode = encode_tiled_fn();
    if (encode == nullptr) return false;
    const cuuint32_t estr[3] = {1u, 1u, 1u};
    auto encoded = [&]() {
        return encode(m, type, (cuuint32_t)rank, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult rc = encoded();
    if (rc == CUDA_ERROR_INVALID_CONTEXT) {   // the first CUDA work of this host thread: nothing has made the device's context its own yet
        int dev = 0;
        if (cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) rc = encoded();
    }
    return rc == CUDA_SUCCESS;
}
// Map over v viewed as [token][head][128] bf16 with tiles of 16 tokens x 64 columns of one head; the 16-byte pieces of a tile
// row are permuted by the row (128-byte swizzle), so that transposing reads of the tile (8 rows of one piece) do not collide.
bool encode_v_map(CUtensorMap* m, const fkda_fwd_params& p) {
    const cuuint64_t dims[3] = {(cuuint64_t)kD, (cuuint64_t)p.H, (cuuint64_t)(p.B * p.T)};
    const cuuint64_t strides[2] = {(cuuint64_t)kD * 2, (cuuint64_t)p.token_stride * 2};  // bytes, dims 1 and 2
    const cuuint32_t box[3] = {(cuuint32_t)kD / 2, 1u, (cuuint32_t)kChunk};
    return encode_map(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, p.v, dims, strides, box);
}
// Map over states viewed as [chains * 128 rows][128 columns], in tiles 128 bytes wide: 128 rows of 64 bf16 or 64 rows of 32
// fp32 columns (16 or 8 KB), swizzled as above.
bool encode_state_map(CUtensorMap* m, const void* base, int64_t chains, bool fp32) {
    const cuuint64_t dims[2] = {(cuuint64_t)kD, (cuuint64_t)(chains * kD)};
    const cuuint64_t strides[1] = {(cuuint64_t)kD * (fp32 ? 4 : 2)};
    const cuuint32_t box[2] = {fp32 ? 32u : 64u, fp32 ? 64u : 128u};
    return encode_map(m, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box);
}

// What the start and the end of a chain cost a CTA of the one-kernel forward, in chunk steps: the loads and stores of its state,
// which nothing hides (a chain of c chunks takes 1.2 c + 3.9 us with bf16 states in and out and 1.2 c + 5.7 us with fp32
// states).  Measured best among 0 .. 8 on sequences of 1 to 2 u tokens, u = 2 to 64 chunks, 512 to 12 800 chains: 1 without
// states, 3 with bf16 states, 4 with fp32 states (12 800 chains of 4 chunks on average, us by weight 0, 1, 3, 4, 8: no states
// 663, 587, 635, 655, 710; bf16 1115, 962, 853, 872, 925; fp32 1452, 1246, 1038, 1033, 1089).
static int chain_weight(const fkda_fwd_params& p) {
    const int each = p.state_dtype == FKDA_STATE_FP32 ? 3 : 2;
    return (2 + (p.initial_state != nullptr ? each : 0) + (p.final_state != nullptr ? each : 0)) / 2;
}

// One kernel (and the prefix kernel of a ragged batch).
static int launch_fused(const fkda_fwd_params& p, TwoPassArgs& a, int sms, cudaStream_t stream, int* n_launches) {
    const int64_t chains = p.N * p.H;
    a.chain_weight = chain_weight(p);
    // the flags directly behind the header for a fixed batch (it has no prefix tables): one stretch to clear; the prefix
    // kernel clears both for a ragged batch
    uint8_t* base = reinterpret_cast<uint8_t*>(p.workspace) + kWsHeaderBytes;
    uint8_t* flags = base + (p.cu_seqlens != nullptr ? ws_prefix_bytes(p.N) : 0);
    a.range_flags = reinterpret_cast<int32_t*>(flags);
    a.seg_state = reinterpret_cast<uint32_t*>(base + ws_prefix_bytes(p.N) + fused_flag_bytes(sms));
    int launches = 0;
    if (p.cu_seqlens != nullptr) {
        if (!launch_tile_prefix(a, nullptr, false, stream, sms)) return FKDA_ERR_LAUNCH;
        ++launches;
    } else if (cudaMemsetAsync(p.workspace, 0, kWsHeaderBytes + (size_t)sms * 4, stream) != cudaSuccess) {
        return FKDA_ERR_LAUNCH;
    }
    VMap map;
    if (!encode_v_map(&map.v, p)) return FKDA_ERR_LAUNCH;
    const bool exports = a.chunk_states != nullptr;
    if (!(exports ? allow_smem<fused_kernel<true, false>>(kFusedSmemBytes) : allow_smem<fused_kernel<false, false>>(kFusedSmemBytes))) return FKDA_ERR_LAUNCH;
    const auto kernel = exports ? fused_kernel<true, false> : fused_kernel<false, false>;
    const int64_t ctas = chains < sms ? chains : sms;
    if (!launch_dependent(kernel, ctas, kFusedThreads, kFusedSmemBytes, stream, a, map)) return FKDA_ERR_LAUNCH;
    *n_launches = launches + 1;
    return FKDA_OK;
}

// The row-slice kernel for a call.
struct RowsLaunch {
    void (*kernel)(const TwoPassArgs, const VMap);
    int smem, threads, split;
    bool ok;
};
template <bool kExport, bool kLoop, int kMt, int kWarps, int kPair>
static RowsLaunch rows_launch() {
    constexpr int kBytes = RowSmem<kMt, kWarps, 4, kPair>::kBytes;
    static_assert(kBytes <= 232448, "shared memory of an SM");
    constexpr auto kKernel = recurrence_rows_kernel<kExport, kLoop, kMt, kWarps, 4, kPair>;
    return RowsLaunch{kKernel, kBytes, row_threads(kWarps), row_split(kWarps, kMt), allow_smem<kKernel>(kBytes)};
}
// Four CTAs per chain of two warps each instead of two of four, where the SMs last: a step takes 0.43 us against 0.47 (the warps of
// a CTA share one shared-memory pipe, 8 192 tokens of 8 heads 235 us against 254, 777 tokens of 32 heads 37.6 against 38.9; eight CTAs
// of one warp: 237 us).  With the prepare stage of the next slab beside it that takes twice as many SMs more as there are chains
// (8 192 tokens: 16 heads 250 against 257, 32 heads, where the prepare stage comes out of hiding, 380 against 280).
static RowsLaunch rows_select(const TwoPassArgs& a, int64_t chains, int sms, bool slabs) {
    if (a.short_flag != nullptr) return rows_launch<false, true, 1, 4, 1>();   // (such a batch exports no states)
    const bool exports = a.chunk_states != nullptr;
    if (chains * kRowSplit > sms) return exports ? rows_launch<true, false, 1, 4, 1>() : rows_launch<false, false, 1, 4, 1>();
    const bool four = slabs ? 4 * chains + 2 * chains <= sms : 4 * chains <= sms;
    if (four) return exports ? rows_launch<true, false, 1, 2, 2>() : rows_launch<false, false, 1, 2, 2>();
    return exports ? rows_launch<true, false, 1, 4, 2>() : rows_launch<false, false, 1, 4, 2>();
}

// More chains than half the SMs, but fewer than SMs: in the one-kernel form a chain's SM walks and prepares, and the others idle.  Here
// they prepare the records of the later chunks meanwhile (side stream), and once the one-kernel form has walked the first chunks a
// row-slice kernel of one CTA per chain, 32 rows per warp, walks the others without a preparing warp beside it, slab by slab.
// A step takes about 1.11 us in the one and 0.77 us in the other, a record 0.0050 us of the whole GPU (0.0043, which would hide
// nothing, to 0.0061 tried): the slabs follow from that.  8 192 tokens of 96 heads: 568 -> 475 us in runs of some milliseconds, 581 -> 520
// in long ones, where the power cap takes the clock down; of 80 heads 579 -> 444 in the former.
// The one-kernel form needs the caller's stream alone, so a call that finds the side stream in another's hands takes that form.
static int launch_mid(const fkda_fwd_params& p, TwoPassArgs& a, int sms, int dev, cudaStream_t stream, int* n_launches) {
    const int chains = (int)(p.N * p.H), idle = sms - chains, tps = (int)((p.T + kChunk - 1) / kChunk);
    const double records = 0.0050 * sms * chains / idle;   // us for the records of one chunk of every chain
    const int n_slabs = tps >= 256 ? kMaxSlabs : 3;
    double size[kMaxSlabs] = {1.0, 1.11 / records, 0.0, 0.0}, total = 0.0, run = 0.0;
    for (int i = 1; i < n_slabs; ++i) {
        if (i > 1) size[i] = size[i - 1] * 0.77 / records;
        if (size[i] > 4.0 * size[i - 1]) size[i] = 4.0 * size[i - 1];
    }
    for (int i = 0; i < n_slabs; ++i) total += size[i];
    int bounds[kMaxSlabs + 1] = {0};
    for (int i = 0; i < n_slabs; ++i) {
        run += size[i];
        bounds[i + 1] = i + 1 == n_slabs ? tps : (int)(run / total * tps + 1.0) / 2 * 2;
    }
    a.chain_weight = chain_weight(p);
    uint8_t* base = reinterpret_cast<uint8_t*>(p.workspace) + kWsHeaderBytes;
    a.range_flags = reinterpret_cast<int32_t*>(base);
    uint8_t* states = base + ws_prefix_bytes(p.N) + fused_flag_bytes(sms);
    a.seg_state = reinterpret_cast<uint32_t*>(states);
    a.workspace = states + (size_t)chains * kStateBytes;
    VMap map;
    if (!encode_v_map(&map.v, p)) return FKDA_ERR_LAUNCH;
    const bool exports = a.chunk_states != nullptr;
    if (!(exports ? allow_smem<fused_kernel<true, true>>(kFusedSmemBytes) : allow_smem<fused_kernel<false, true>>(kFusedSmemBytes))) return FKDA_ERR_LAUNCH;
    const RowsLaunch rows = exports ? rows_launch<true, false, 2, 4, 2>() : rows_launch<false, false, 2, 4, 2>();
    SlabStreams* ss = slab_streams(dev, kSideMid);
    if (!rows.ok || ss == nullptr) return FKDA_ERR_LAUNCH;
    std::unique_lock<std::mutex> enqueue_lock(ss->launch_mu);
    if (!side_free(*ss, stream)) {   // (same results)
        enqueue_lock.unlock();
        return launch_fused(p, a, sms, stream, n_launches);
    }
    auto slab_args = [&](int i) {
        TwoPassArgs x = a;
        x.slab_c0 = bounds[i];
        x.slab_chunks = bounds[i + 1] - bounds[i];
        return x;
    };
    if (cudaEventRecord(ss->fork, stream) != cudaSuccess || cudaStreamWaitEvent(ss->side, ss->fork, 0) != cudaSuccess) return FKDA_ERR_LAUNCH;
    if (cudaMemsetAsync(p.workspace, 0, kWsHeaderBytes + (size_t)sms * 4, stream) != cudaSuccess) return FKDA_ERR_LAUNCH;
    const auto kernel = exports ? fused_kernel<true, true> : fused_kernel<false, true>;
    kernel<<<(unsigned)chains, kFusedThreads, kFusedSmemBytes, stream>>>(slab_args(0), map);
    int launches = 1;
    for (int i = 1; i < n_slabs; ++i) {
        if (bounds[i + 1] <= bounds[i]) continue;
        if (launch_prepare_warp<true>(slab_args(i), ss->side, idle) != FKDA_OK) return FKDA_ERR_LAUNCH;
        if (cudaEventRecord(ss->done[i], ss->side) != cudaSuccess || cudaStreamWaitEvent(stream, ss->done[i], 0) != cudaSuccess) return FKDA_ERR_LAUNCH;
        rows.kernel<<<(unsigned)chains, rows.threads, rows.smem, stream>>>(slab_args(i), map);
        launches += 2;
    }
    if (cudaGetLastError() != cudaSuccess) return FKDA_ERR_LAUNCH;
    *n_launches = launches;
    return FKDA_OK;
}

int launch_tc(const fkda_fwd_params& p, cudaStream_t stream, int* n_launches) {
    TwoPassArgs a;
    fill_args(p, &a);
    const bool varlen = p.cu_seqlens != nullptr;
    const bool do_prep = p.phase_mask == 0 || (p.phase_mask & FKDA_PHASE_PREPARE);
    const bool do_rec = p.phase_mask == 0 || (p.phase_mask & FKDA_PHASE_RECURRENCE);
    int launches = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return FKDA_ERR_LAUNCH;
    const int sms = device_sm_count();
    const int64_t T_total = p.B * p.T, chains = p.N * p.H;
    if (fused_eligible(p, sms)) {
        if (mid_eligible(p, sms) && p.workspace_bytes >= mid_bytes(p, sms)) return launch_mid(p, a, sms, dev, stream, n_launches);
        return launch_fused(p, a, sms, stream, n_launches);
    }
    if (chains * kRowSplit > 0x7fffffff) return FKDA_ERR_BAD_SHAPE;
    a.records_tag = records_tag(p);
    a.on_demand = do_rec && !do_prep;
    const bool tables = do_prep || do_rec;   // (a phase mask may also name neither)
    // (the header is cleared by the first kernel where there is one: the prefix kernel, or the prepare stage of a fixed batch)
    if (!(varlen ? tables : do_prep && a.total_tiles > 0) && cudaMemsetAsync(p.workspace, 0, 64, stream) != cudaSuccess) return FKDA_ERR_LAUNCH;
    const TcCarve carve = tc_carve(p, sms);
    uint8_t* base = reinterpret_cast<uint8_t*>(p.workspace) + kWsHeaderBytes + ws_prefix_bytes(p.N);
    a.seg_state = reinterpret_cast<uint32_t*>(base);
    a.workspace = base + carve.states;
    VMap map;
    memset(&map, 0, sizeof(map));
    // (an empty batch has no tiles to move: its chains only pass their state through)
    if (do_rec && T_total > 0 && !encode_v_map(&map.v, p)) return FKDA_ERR_LAUNCH;
    // A ragged batch whose sequences MAY all fit one chunk (the host sees only the totals): the prefix kernel decides, the
    // one-chunk kernels and the general kernels are all enqueued and all but one return at once.
    if (short_ragged_candidate(p) && !(p.flags & FKDA_FLAG_NO_SHORT)) a.short_flag = a.queue + 8;
    const int64_t tps = (p.T + kChunk - 1) / kChunk;
    const bool slabs = !varlen && p.phase_mask == 0 && slabs_possible(chains, sms) && tps >= 64 && !(p.flags & FKDA_FLAG_NO_SLABS);
    const RowsLaunch rows = rows_select(a, chains, sms, slabs);
    if (!rows.ok) return FKDA_ERR_LAUNCH;
    a.early_rows = a.short_flag == nullptr && chains * rows.split <= sms;

    // ---- few chains on a fixed batch: the recurrence is a serial walk on 2 x chains SMs and leaves the others
    //      idle, so the forward is cut into slabs of chunks and the prepare stage of slab i+1 runs on the idle SMs
    //      (side stream) while the recurrence walks slab i; the state of a chain travels through seg_state.
    //      Only stream order and events connect the launches: no kernel waits for another one. ----
    if (slabs) {
        const int idle_sms = sms - (int)chains * rows.split;
        SlabStreams* ss = slab_streams(dev, kSideSlabs);
        if (ss == nullptr) return FKDA_ERR_LAUNCH;
        // host threads that call concurrently on one device share the side stream and its events
        std::lock_guard<std::mutex> enqueue_lock(ss->launch_mu);
        // Slab boundaries.  The prepare of slab i+1 (on idle_sms SMs, about 5.8 ns per (chunk, head) on the whole GPU) must
        // be done when the recurrence (0.47 us per chunk, 0.43 with four CTAs per chain) has walked slab i: the slabs grow (or shrink) by the ratio
        // of the two speeds (the factor 1.1 measured: 0.9 .. 1.4 tried).  Two or four slabs: more of them leave less of the prepare stage in front of the first one,
        // unhidden, and cost a hand-over of the states and a launch each, about 5 us.
        const double prep_us = 0.0058 * (double)(chains * tps), walk_us = (rows.split == 4 ? 0.43 : 0.47) * (double)tps;
        const double fit = 1.1 * walk_us * (double)idle_sms / (prep_us * (double)sms);
        const double grow = fit < 0.6 ? 0.6 : (fit > 8.0 ? 8.0 : fit);
        int n_slabs = 2;
        if (tps >= 256) {
            const double first2 = prep_us / (1.0 + grow), first4 = prep_us / (1.0 + grow + grow * grow + grow * grow * grow);
            if (first2 > (first4 > 6.0 ? first4 : 6.0) + 10.0) n_slabs = kMaxSlabs;
        }
        int bounds[kMaxSlabs + 1];
        double total = 0.0, part = 1.0, run = 0.0;
        for (int i = 0; i < n_slabs; ++i, part *= grow) total += part;
        part = 1.0;
        for (int i = 0; i <= n_slabs; ++i, part *= grow) {
            bounds[i] = (int)((int64_t)(run / total * (double)tps + 1.0) / 2 * 2);  // even
            run += part;
        }
        bounds[0] = 0;
        if (bounds[1] < 2) bounds[1] = 2;
        bounds[n_slabs] = (int)tps;
        auto slab_args = [&](int i) {
            TwoPassArgs x = a;
            x.slab_c0 = bounds[i];
            x.slab_chunks = bounds[i + 1] - bounds[i];
            return x;
        };
        // (the side stream forks in front of the first prepare kernel, so that nothing lies between that one and the first walk)
        if (cudaEventRecord(ss->fork, stream) != cudaSuccess || cudaStreamWaitEvent(ss->side, ss->fork, 0) != cudaSuccess) return FKDA_ERR_LAUNCH;
        if (launch_prepare_warp<true>(slab_args(0), stream, 0, true) != FKDA_OK) return FKDA_ERR_LAUNCH;
        const int64_t row_ctas = chains * rows.split;
        if (!launch_dependent(rows.kernel, row_ctas, rows.threads, rows.smem, stream, slab_args(0), map)) return FKDA_ERR_LAUNCH;
        launches += 2;
        for (int i = 1; i < n_slabs; ++i) {
            if (bounds[i + 1] <= bounds[i]) continue;
            if (launch_prepare_warp<true>(slab_args(i), ss->side, idle_sms) != FKDA_OK) return FKDA_ERR_LAUNCH;
            if (cudaEventRecord(ss->done[i], ss->side) != cudaSuccess || cudaStreamWaitEvent(stream, ss->done[i], 0) != cudaSuccess) return FKDA_ERR_LAUNCH;
            rows.kernel<<<(unsigned)row_ctas, rows.threads, rows.smem, stream>>>(slab_args(i), map);
            launches += 2;
        }
        if (cudaGetLastError() != cudaSuccess) return FKDA_ERR_LAUNCH;
        *n_launches = launches;
        return FKDA_OK;
    }

    // as many tokens as sequences: they may have one token each, the decode kernel's case
    const bool try_decode = a.short_flag != nullptr && T_total == p.N && chains <= decode_max_chains(p) && !(p.flags & FKDA_FLAG_NO_DECODE);
    // The recurrence alone takes the records that an earlier call on this workspace left.  That call may have been one that leaves
    // none (the one-kernel forms), so the tables of a ragged batch are made again and the prepare stage is enqueued in any
    // case: it returns at once where the records are there.
    if (varlen && tables) {
        if (!launch_tile_prefix(a, const_cast<int32_t*>(a.seq_order), try_decode, stream)) return FKDA_ERR_LAUNCH;
        ++launches;
    }
    if (try_decode) {
        if (launch_decode_kernel(a, stream) != FKDA_OK) return FKDA_ERR_LAUNCH;
        ++launches;
    }
    if (a.short_flag != nullptr) {
        if (launch_short_ragged(p, a, stream) != FKDA_OK) return FKDA_ERR_LAUNCH;
        ++launches;
    }
    if (a.total_tiles > 0 && tables) {
        if (launch_prepare_warp<true>(a, stream, 0, true) != FKDA_OK) return FKDA_ERR_LAUNCH;
        ++launches;
    }
    if (do_rec) {
        // (behind a device-side decision this launch mostly returns at once: a grid that is resident in one go)
        int64_t ctas = chains * rows.split;
        if (a.seq_order != nullptr && ctas > sms && ctas <= 2 * sms) a.layer = sms;
        if (a.short_flag != nullptr && ctas > 2 * sms) ctas = 2 * sms;
        if (launches > 0) {
            if (!launch_dependent(rows.kernel, ctas, rows.threads, rows.smem, stream, a, map)) return FKDA_ERR_LAUNCH;
        } else {
            rows.kernel<<<(unsigned)ctas, rows.threads, rows.smem, stream>>>(a, map);
        }
        ++launches;
    }
    if (cudaGetLastError() != cudaSuccess) return FKDA_ERR_LAUNCH;
    *n_launches = launches;
    return FKDA_OK;
}

}  // namespace fkda
