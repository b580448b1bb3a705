// The prepare stage as a kernel of its own: every warp turns (chunk, head) units into chunk records in the workspace (fkda_prep.cuh
// does the work).  Grid-stride: warp w of the grid takes units w, w + W, ... with the head index fastest, so that
// neighbouring warps read neighbouring 256-byte rows.  One record block of shared memory per warp; a finished record leaves by
// a bulk copy (kTc) or, for the CUDA-core recurrence, in that kernel's plain layout.
// Bound by the latency of a unit (7 us of dependent instructions and loads, two thirds of it its rows) at 12 warps per SM: 0.7 of the
// copy bandwidth on its own 27 KB per unit (16 384 units: 91 us, 96 before two rows shared their norms; on 52 SMs beside a walk
// 12 ns per unit, 4.3 of the whole GPU's; the 1 568 units of a 777-token prompt with 32 heads: 13.0 us against 14.7).
#pragma once

#include "fkda_prep.cuh"

namespace fkda {

// Where chunk `tile` of the (possibly ragged) batch lives: first token and number of valid rows.
// Returns false for a tile index past the last chunk (ragged upper bound).
__device__ __forceinline__ bool locate_tile(const TwoPassArgs& a, int64_t tile, int64_t* t0, int* len) {
    int64_t n, local_t, bos, seq_len;
    if (a.cu_seqlens != nullptr) {
        const int32_t* pre = a.tile_prefix;
        if (tile >= pre[a.N]) return false;
        int64_t lo = 0, hi = a.N;  // find n with pre[n] <= tile < pre[n+1]
        while (hi - lo > 1) {
            int64_t mid = (lo + hi) >> 1;
            if (pre[mid] <= tile) lo = mid; else hi = mid;
        }
        n = lo;
        local_t = tile - pre[n];
        bos = a.cu_seqlens[n];
        seq_len = a.cu_seqlens[n + 1] - bos;
    } else {
        const int64_t tps = (a.T + kChunk - 1) / kChunk;
        n = tile / tps;
        local_t = tile - n * tps;
        bos = n * a.T;
        seq_len = a.T;
    }
    *t0 = bos + local_t * kChunk;
    *len = (int)min((int64_t)kChunk, seq_len - local_t * kChunk);
    return true;
}

// Warps per CTA: 12 with 168 registers each; 15, as many as have room for a record block, with 128, for 13 to 15 units per SM, where
// that makes one round of units out of two (so its warps take one unit each, with no next one to ask for and no spills).  More rounds are not worth it, although there may be one less
// (us of the stage with 12 and with 15 warps, by units per SM: 12: 14.5 both; 13: 20.6, 16.9; 14: 20.8, 18.4; 15: 21.2, 18.5;
// 25: 30.0, 31.0; 28: 31.1, 32.6; 30: 32.3, 32.8; 37: 39.9, 43.6; 45: 41.2, 45.1).
constexpr int kPrepWarps = 12, kPrepWarpsMost = 15;

// The plain record of the CUDA-core recurrence (kWs* layout): kd, qd, kr row-major, INV and Mqk row-major.
__device__ __forceinline__ void prep_export_plain(uint8_t* ws, const uint8_t* rec_ptr, int lane) {
    const uint32_t rec = sm100::smem_u32(rec_ptr);
    const int c = lane & 15, hh = lane >> 4;
#pragma unroll 2
    for (int i = 0; i < 8; ++i) {
        const int r = 8 * hh + i;
        *reinterpret_cast<uint4*>(ws + kWsKd + r * 256 + c * 16) = prep_lds(rec + kTcB1 + tc_b1_off(r, c));
        *reinterpret_cast<uint4*>(ws + kWsQd + r * 256 + c * 16) = prep_lds(rec + kTcB1 + tc_b1_off(r + 16, c));
        *reinterpret_cast<uint4*>(ws + kWsKr + r * 256 + c * 16) = prep_lds(rec + kTcKr + tc_kr_off(r, c));
    }
    *reinterpret_cast<uint4*>(ws + kWsEt + lane * 16) = prep_lds(rec + kTcEt + lane * 16);
    const int i = lane >> 1, j = 8 * (lane & 1);   // a 16-byte piece of each 16 x 16 matrix
    *reinterpret_cast<uint4*>(ws + kWsInv + (i * kChunk + j) * 2) = prep_lds(rec + kTcInv + tc_sq_off(i, j));
    *reinterpret_cast<uint4*>(ws + kWsMqk + (i * kChunk + j) * 2) = prep_lds(rec + kTcMqk + tc_sq_off(i, j));
}

template <bool kTc, int kMaxWarps>
__global__ void __launch_bounds__(kMaxWarps * 32, 1) prepare_warp_kernel(const __grid_constant__ TwoPassArgs a) {
    // (otherwise the recurrence's CTAs would fill the first SMs that fall free two by two)
    if (a.early_rows) grid_dep_launch();
    grid_dep_wait();
    // the first launch of a fixed batch's forward clears the device status (the prefix kernel that of a ragged batch)
    if (a.cu_seqlens == nullptr && a.slab_c0 == 0 && blockIdx.x == 0 && threadIdx.x == 0) *a.status = 0;
    // (a ragged batch that the fused short-sequence kernel has served: nothing to do)
    if (a.short_flag != nullptr && *a.short_flag != 0) return;
    if (a.on_demand) {   // (these records get no note: CTAs that start later still have to find none)
        if (*a.records == a.records_tag) return;
    } else if (a.slab_c0 == 0 && blockIdx.x == 0 && threadIdx.x == 0) {
        *a.records = a.records_tag;
    }
    extern __shared__ uint8_t prep_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t* rec = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(prep_smem) + 127) & ~(uintptr_t)127) + warp * kTcRecord;
    // units = (chunk, head) pairs, head fastest; with a slab (fixed batches) only chunks [slab_c0, slab_c0 +
    // slab_chunks) of every sequence, enumerated densely
    const int64_t tps = (a.T + kChunk - 1) / kChunk;  // chunks per sequence of a fixed batch
    const int64_t n_units = (a.slab_chunks > 0 ? a.N * (int64_t)a.slab_chunks : a.total_tiles) * a.H;
    const int warps = blockDim.x >> 5;
    const int64_t stride = (int64_t)gridDim.x * warps;
    // units past the last chunk of a ragged batch (upper-bound tile count) all sit at the end of the range
    auto locate = [&](int64_t u, int64_t* tile, int64_t* t0, int* len, int* h) {
        if (u >= n_units) return false;
        int64_t t = u / a.H;
        *h = (int)(u - t * a.H);
        if (a.slab_chunks > 0) {
            const int64_t n = t / a.slab_chunks;
            t = n * tps + a.slab_c0 + (t - n * a.slab_chunks);
        }
        *tile = t;
        return locate_tile(a, t, t0, len);
    };
    int64_t u = (int64_t)blockIdx.x * warps + warp;
    int64_t tile = 0, tile_n = 0, t0 = 0, t0n = 0;
    int len = 0, h = 0, lenn = 0, hn = 0;
    bool valid = locate(u, &tile, &t0, &len, &h);
    PrepHead x;
    PrepSrc src;
    if (valid) {
        src = prep_src(a, t0, len, h, lane);
        prep_load(a, src, t0, len, h, lane, x);
    }
    constexpr bool kOneRound = kMaxWarps == kPrepWarpsMost;   // one unit per warp (see launch_prepare_warp)
    while (valid) {
        const bool next_valid = !kOneRound && locate(u + stride, &tile_n, &t0n, &lenn, &hn);
        uint8_t* ws = a.workspace + ((int64_t)h * a.total_tiles + tile) * (int64_t)(kTc ? kTcRecord : kWsRecord);
        prep_compute<false, true>(a, src, len, rec, lane, x,
                     [&]() {   // the previous record has left the block
                         if (kTc && lane == 0) sm100::bulk_wait_group_read<0>();
                         __syncwarp();
                         return true;
                     },
                     [&]() {   // the head of the next unit travels while the products and the inverse run
                         if (!kOneRound && next_valid) {
                             src = prep_src(a, t0n, lenn, hn, lane);
                             prep_load(a, src, t0n, lenn, hn, lane, x);
                         }
                     });
        if constexpr (kTc) {
            sm100::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                sm100::bulk_s2g(ws, rec, kTcRecord);
                sm100::bulk_commit_group();
            }
        } else {
            prep_export_plain(ws, rec, lane);
            __syncwarp();
        }
        u += stride;
        valid = next_valid;
        tile = tile_n; t0 = t0n; len = lenn; h = hn;
    }
    sm100::bulk_wait_group<0>();  // (lane 0) the last records have landed
}

// max_ctas > 0 caps the grid (a launch that shares the GPU with a concurrent recurrence kernel); dependent: behind another
// kernel of the same call
template <bool kTc>
inline int launch_prepare_warp(const TwoPassArgs& a, cudaStream_t stream, int max_ctas = 0, bool dependent = false) {
    const int sms = device_sm_count();
    const int64_t n_units = (a.slab_chunks > 0 ? a.N * (int64_t)a.slab_chunks : a.total_tiles) * a.H;
    // few units: spread over all SMs, with as many warps per CTA as that takes
    const int64_t max_grid = max_ctas > 0 && max_ctas < sms ? max_ctas : sms;
    const int64_t per = (n_units + max_grid - 1) / max_grid;
    const bool most = per > kPrepWarps && per <= kPrepWarpsMost;   // one round instead of two
    const int max_warps = most ? kPrepWarpsMost : kPrepWarps;
    if (!(most ? allow_smem<prepare_warp_kernel<kTc, kPrepWarpsMost>>(kPrepWarpsMost * kTcRecord + 128)
               : allow_smem<prepare_warp_kernel<kTc, kPrepWarps>>(kPrepWarps * kTcRecord + 128)))
        return FKDA_ERR_LAUNCH;
    const auto kernel = most ? prepare_warp_kernel<kTc, kPrepWarpsMost> : prepare_warp_kernel<kTc, kPrepWarps>;
    const int warps = (int)(per < 1 ? 1 : (per < max_warps ? per : max_warps));
    int64_t ctas = (n_units + warps - 1) / warps;
    if (ctas > max_grid) ctas = max_grid;
    if (ctas < 1) ctas = 1;
    if (dependent) return launch_dependent(kernel, ctas, warps * 32, warps * kTcRecord + 128, stream, a) ? FKDA_OK : FKDA_ERR_LAUNCH;
    kernel<<<(unsigned)ctas, warps * 32, warps * kTcRecord + 128, stream>>>(a);
    return FKDA_OK;
}

}  // namespace fkda
