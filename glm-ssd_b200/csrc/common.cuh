// Shared host/device helpers of the attention library.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/glmssd_attn.h"

#define GS_EXPORT extern "C" __attribute__((visibility("default")))

namespace gs {

// Last-error text, per host thread (gs_attn_last_error_string).
void set_error(const char *fmt, ...);

inline int fail_invalid(const char *what) {
    set_error("%s", what);
    return (int) cudaErrorInvalidValue;
}

#define GS_TRY(expr)                                                          \
    do {                                                                      \
        cudaError_t _e = (expr);                                              \
        if (_e != cudaSuccess) {                                              \
            gs::set_error("%s: %s", #expr, cudaGetErrorString(_e));           \
            return (int) _e;                                                  \
        }                                                                     \
    } while (0)

// ---- decode workspace layout -------------------------------------------------------------------
// [0, 32768)               status block: int32 status word (sticky, kernels only OR into it);
//                           int32 at byte 4: when non-zero, CTA 0 of the tcgen05 kernel writes clock64
//                           stamps of its first tiles as int64 from byte 256 on (a tuning aid, off by default)
//   [4096, 16384)           with the same switch every CTA of the tcgen05 kernel writes eight int64 %globaltimer
//                           stamps (entry, inputs visible, first tile landed, drain start/end, exit, SM id)
//   [16384, 32768)          and every CTA of the combine kernel eight stamps of its own
// [32768, ...)             per-sequence segment descriptors, then
//                           partial accumulators f32 [n_segments][rows_q][d_v]
// then                     partial (m, l)       f32 [n_segments][rows_q][2]
// A "segment" is the share of one sequence handled by one CTA (tcgen05 kernel: at most
// n_ctas + n_seq of them) or one (sequence, token, split) triple (CUDA-core kernel).
constexpr int kStatusBytes = 32768;
constexpr int kCtaProfOffsetBytes = 4096;       // [cta][8] int64
constexpr int kCombineProfOffsetBytes = 16384;  // [cta][8] int64, first 256 CTAs
constexpr int kProfOffsetBytes = 256;
constexpr int kProfSlots = 16;   // stamps per tile
constexpr int kProfTiles = 24;   // tiles recorded
constexpr int kMaxCtas = 160;       // persistent grid never exceeds this (B200 has 148 SMs)
constexpr int kSimtMaxSplits = 64;  // CUDA-core kernel: splits per (sequence, token)

inline int64_t decode_segments_bound(int n_seq, int T) {
    const int64_t umma = (int64_t) kMaxCtas + n_seq;
    const int64_t simt = (int64_t) n_seq * T * kSimtMaxSplits;
    return umma > simt ? umma : simt;
}

// Units (of unit_rows rows) one CTA of the tcgen05 decode kernel takes; the combine kernel recomputes the schedule with it.
// Several sequences: an equal share.  One sequence: whole 64-row tiles, since the last tile of a CTA costs what a full one
// does - 32768 rows are 128 runs of 4 tiles (18.5 us with two query tokens), not 147 of 3.5 (18.9 us) - and a record less to
// write and to merge for every CTA left out; for the same reason from 75 tiles on at least two tiles, which the two stages hold
// at once anyway (4096 rows: 64 runs 9.4 us, 128 half tiles 10.9 us; 8192 rows: 64 runs of two 10.2 us, 128 of one 11.1 us).
__host__ __device__ inline int decode_chunk(int total_units, int n_ctas, bool one_sequence, int unit_rows) {
    const int even = (total_units + n_ctas - 1) / n_ctas;
    if (!one_sequence) return even > 1 ? even : 1;
    const int shift = unit_rows == 16 ? 2 : 0, tiles = (total_units + (1 << shift) - 1) >> shift;
    int t = (tiles + n_ctas - 1) / n_ctas;
    if (t < 2) t = tiles > 74 ? 2 : 1;
    if (tiles <= 1 && n_ctas >= 4) return 1;  // a single tile: a unit each (64 rows 8.96 -> 8.5 us)
    return t << shift;
}
// CTAs that rule can use for any length up to max_rows (148 from 296 tiles on): no more need to be launched.
inline int decode_grid(int64_t max_rows, int sm_count) {
    const int64_t tiles = (max_rows + 63) / 64;
    const int64_t n = tiles <= 1 ? 4 : tiles <= 74 ? tiles : tiles <= 148 ? 74 : (tiles + 1) / 2;
    return (int) (n < 1 ? 1 : n < sm_count ? n : sm_count);
}

// Row addressing shared by the kernels: explicit list, paged or dense.
struct RowMap {
    const int32_t *list;   // explicit positions (legacy `sel` row) or nullptr
    const int32_t *pages;  // page ids of this sequence or nullptr
    int64_t base;          // dense: first row
    int page_rows;
    __device__ __forceinline__ int64_t operator()(int64_t i) const {
        if (list) return list[i];
        if (pages) return (int64_t) pages[i / page_rows] * page_rows + (i % page_rows);
        return base + i;
    }
};

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace gs
