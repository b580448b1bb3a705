// Internal host/device declarations shared by the translation units of the library.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stddef.h>

#include <atomic>
#include <stdint.h>

#include "../../include/flashkda_b200.h"

namespace fkda {

// Kernel arguments of the two-pass implementation (passed by value).
struct TwoPassArgs {
    const __nv_bfloat16 *q, *k, *v, *g, *beta;
    __nv_bfloat16* out;
    const float *A_log, *dt_bias;
    const void* initial_state;
    void* final_state;
    const int64_t* cu_seqlens;
    int32_t* tile_prefix;  // [N + 1] chunk-count prefix (varlen only)
    const int32_t* seq_order;  // [N] sequences by decreasing length (varlen with N <= kSeqOrderMaxN, else nullptr)
    uint8_t* workspace;    // [H][total_tiles] per-chunk records
    int32_t* queue;        // header word 0: ticket counter of the one-kernel forward (zeroed per call)
    int32_t* status;       // header word 1: device status, 0 ok, else the code of a bounded wait that gave up
    int32_t* short_flag;   // header word 8, or null: written by the prefix kernel of a ragged batch that MAY consist of
                           // one-chunk sequences; the kernels that can serve the call are all enqueued and all but one
                           // return at once: 2 = every sequence has exactly one token (decode kernel), 1 = no sequence is
                           // longer than one chunk (fused short-sequence kernel), 0 = the general kernels
    uint64_t* records;     // header words 16, 17, or null without a header: which chunk records the workspace holds (records_tag of
                           // the call that wrote them; 0: none, the last forward on this workspace kept them on the SMs)
    uint64_t records_tag;  // of this call
    bool on_demand;        // the recurrence alone was asked for: the records are prepared if the workspace does not hold them
    int32_t* range_flags;  // one-kernel forward: walking warps of each range that have published their rows of its state
    uint32_t* seg_state;   // bf16 states in fragment order, handed from range to range (one-kernel forward) or slab to slab
    int32_t slab_c0, slab_chunks;  // fixed batches only: this launch covers chunks [slab_c0, slab_c0 + slab_chunks) of
                                   // every sequence (slab_chunks == 0: all chunks); a chain's state travels from one
                                   // slab to the next through seg_state
    int32_t layer;         // row slices by decreasing length: CTAs of the first layer (one per SM), 0 = no particular order
    int32_t chain_weight;  // one-kernel forward: what the start and the end of a chain cost, in chunk steps (see chain_weight)
    int64_t T, H, N, total_tiles;
    int64_t token_stride, beta_token_stride;
    float scale, gate_scale;
    __nv_bfloat16* chunk_states;   // optional export of the state before every cs_every-th chunk (see fkda_fwd_params)
    const int32_t* cs_prefix;      // [N] first export slot of every sequence (varlen; fixed batches compute it)
    int32_t cs_every;
    uint64_t wait_ns;      // limit of every bounded device-side wait (mbarrier, range flag)
    bool state_fp32;
    bool early_rows;       // the row slices behind the prepare stage take an SM each: their CTAs may come in while it still runs
    bool test_drop_push;   // test hook (FKDA_FLAG_TEST_DROP_PUSH): ranges do not publish the state they hand over
};

// Workspace layout of both two-pass implementations:
//   [0, 256)  header: int32 ticket counter, device status, word 8: path decision of a ragged batch, words 16, 17: which chunk
//             records are behind it
//   [256, ..) tile prefix (N + 1 int32, padded to 256 B)
//   then      H * total_tiles records
constexpr size_t kWsHeaderBytes = 256;
// (N + 1) chunk-prefix entries, N entries of the length order, N + 1 entries of the state-export prefix
inline size_t ws_prefix_bytes(int64_t N) { return (size_t)(((3 * N + 2) * 4 + 255) / 256 * 256); }
constexpr int64_t kSeqOrderMaxN = 512;  // beyond this the quadratic ranking in the prefix kernel is not worth its time
inline int64_t ws_tiles_upper_bound(int64_t T_total, int64_t N) { return (T_total + 15) / 16 + N; }

size_t twopass_workspace_bytes(int64_t T_total, int64_t H, int64_t N);
int launch_twopass(const fkda_fwd_params& p, cudaStream_t stream, int* n_launches);
size_t tc_workspace_bytes(int64_t T_total, int64_t H, int64_t N);   // upper bound for these totals
size_t tc_workspace_bytes_for(const fkda_fwd_params& p);            // what this particular call needs
size_t tc_workspace_bytes_wanted(const fkda_fwd_params& p);         // what it makes use of
int device_sm_count();
// Device address of the built-in scratch of fkda_fwd_noalloc on the current device, or nullptr before that
// entry point's first call there.
void* noalloc_scratch_or_null();
int launch_tc(const fkda_fwd_params& p, cudaStream_t stream, int* n_launches);
// Decode step (fixed batch, T == 1): one read-modify-write kernel over the states, no workspace records.
// (sequence, head) pairs up to which the decode kernel serves it; beyond, the short-sequence kernel, whose state loads never
// pause.  The line is where the two cross with bf16 states (2 048 pairs: 30.8 us both, 1 024: 14.4 against 16.8, 32 768: 435
// against 373); with fp32 states, where the decode kernel's loads are twice as wide, it is the faster one throughout
// (32 768 pairs: 631 against 671).  The chunk kernel's products are summed in another order: with bf16 states the last bits of a decode
// step depend on which side of the line the batch is (relative difference 6.5e-5), and a state row with an infinity becomes NaN there.
inline int64_t decode_max_chains(const fkda_fwd_params& p) { return p.state_dtype == FKDA_STATE_FP32 ? 0x7fffffff / 4 : 2048; }
bool decode_eligible(const fkda_fwd_params& p);
int launch_decode(const fkda_fwd_params& p, cudaStream_t stream, int* n_launches);
// Short sequences (fixed batch, 2 <= T <= 16): one fused kernel per (sequence, head), no workspace records.
bool short_eligible(const fkda_fwd_params& p);
int launch_short(const fkda_fwd_params& p, cudaStream_t stream, int* n_launches);
// Ragged batches: whether the call MAY consist of sequences of at most one chunk each (the host knows only the totals;
// the prefix kernel decides on the device), and the launch of the fused kernel behind that decision.
bool short_ragged_candidate(const fkda_fwd_params& p);
int launch_short_ragged(const fkda_fwd_params& p, const TwoPassArgs& a, cudaStream_t stream);
// Tensor maps over v and over the states (fkda_tc.cu).
bool encode_v_map(CUtensorMap* m, const fkda_fwd_params& p);
bool encode_state_map(CUtensorMap* m, const void* base, int64_t chains, bool fp32);
int launch_decode_kernel(const TwoPassArgs& a, cudaStream_t stream);   // (a ragged batch: as many tokens as sequences, maybe one each)

// Allows a kernel its dynamic shared memory on the current device.  The attribute belongs to the function and the device,
// so it is set once for each and remembered (a driver call on every launch is half a microsecond of host time).
template <auto kKernel>
inline bool allow_smem(int bytes) {
    static std::atomic<uint64_t> devices{0};   // bit d: set on device d
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const uint64_t bit = dev < 64 ? (uint64_t)1 << dev : 0;
    if ((devices.load(std::memory_order_acquire) & bit) != 0) return true;
    if (cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return false;
    devices.fetch_or(bit, std::memory_order_release);
    return true;
}

// Launches a kernel that begins with grid_dep_wait() (fkda_common.cuh) behind whatever kernel is in front of it on the stream,
// of the same call, the call before or the caller's own: its launch and start overlap that kernel's end, and nothing of it
// touches memory before that end.  (One token of 32 heads, steps back to back through Python: 4.1 -> 2.9 to 3.4 us, by the host; a
// prompt of 100 tokens, 8 heads: 12.3 -> 11.2; 4 x 1 tokens of 32 heads: 6.2 -> 4.5.  With nothing in front there is nothing to gain.)
template <typename... KernelArgs, typename... Args>
inline bool launch_dependent(void (*kernel)(KernelArgs...), int64_t ctas, int threads, int smem, cudaStream_t stream, const Args&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess;
}

// Fills the kernel arguments common to both implementations (pointers, strides, gate scale,
// workspace carving).
void fill_args(const fkda_fwd_params& p, TwoPassArgs* a);
// The prefix kernel of a ragged batch: chunk (and state-export) prefix tables, the length order if asked for, and the path
// decision if a.short_flag is set; clears the header (the note on the records only if the call is going to write new ones
// or none) and `n_flags` range flags.
bool launch_tile_prefix(const TwoPassArgs& a, int32_t* seq_order, bool decode_enqueued, cudaStream_t stream, int n_flags = 0);
// First state-export slot of sequence n.
__device__ __forceinline__ int64_t cs_first_slot(const TwoPassArgs& a, int64_t n) {
    if (a.cu_seqlens != nullptr) return a.cs_prefix[n];
    const int64_t group = 16 * (int64_t)a.cs_every;
    return n * ((a.T + group - 1) / group);
}

}  // namespace fkda
