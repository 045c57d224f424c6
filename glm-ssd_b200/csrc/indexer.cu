// DSA k-pool indexer: the kernels that produce the attended position lists (sel, cnt) the attention call
// consumes once the context is longer than top_k positions (crates/engine/src/forward.rs:864-895).  Same entry
// points and arguments as the reference (crates/cuda/kernels/ops.cu:619-791, Rust declarations
// crates/cuda/src/lib.rs:101-113):
//
//   gs_idx_pool    pooled indexer key of every pool of `kpool` positions that completes inside the chunk, plus
//                  the hand-over of the trailing incomplete pool's raw rows to the ring buffers - one launch
//                  (the reference needs two: the pool that straddles the chunk start reads the ring slots the
//                  hand-over then rewrites, so here the same thread does both for its column, in that order);
//   gs_idx_score   score[t][p] = sum_h w[t][h] * relu(scale * q[t][h] . P[p]) over the complete pools;
//   gs_idx_select  exact top-k of the scores (radix select on the order-preserving integer image, as the
//                  reference) and the position list built from it.
//
// One difference in gs_idx_select, on purpose: the reference fills the list in the order its threads reach an
// atomic counter, so the order of the pools inside `sel` - and, among pools whose score equals the k-th largest,
// which of them are taken - changes from run to run there.  Here the list is deterministic: pools in ascending
// index, ties to the lowest indices.  The set of selected pools is the reference's whenever the k-th largest
// score is unique; `cnt` is always the same.
#include <cuda_bf16.h>

#include "internal.cuh"
#include "sm100_prims.cuh"

namespace gs {
namespace {

// ---- pooling ------------------------------------------------------------------------------------------------
__device__ __forceinline__ const float *idx_row(const float *chunk, const float *ring, int64_t pos, int p0, int Dk, int kpool) {
    return pos >= p0 ? chunk + (pos - p0) * Dk : ring + (pos % kpool) * Dk;
}

// grid (column blocks, max(1, completing pools)); thread = one column of one pool.  Only the first completing pool
// (the one holding position p0) can reach into the rings; its threads also hand the trailing rows over afterwards.
// A few hundred bytes per thread: the time is the chain of dependent memory round trips.  KP > 0 (kpool as a constant)
// requests gates, keys and ape together, one round trip instead of three (a decode step, cold caches: 7.7 -> 3.0 us).
template <int KP>
__global__ void __launch_bounds__(128) k_idx_pool(const float *__restrict__ kc, const float *__restrict__ gc, float *rk, float *rg,
                                                  const float *__restrict__ ape, float *__restrict__ P, int p0, int T, int Dk, int kpool_arg) {
    const int kpool = KP > 0 ? KP : kpool_arg;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int end = p0 + T;
    const int jf = p0 / kpool, jl = end / kpool;
    const int64_t j = (int64_t) jf + blockIdx.y;
    sm100::griddep_wait();
    sm100::griddep_launch_dependents();
    if (c >= Dk) return;
    if (j < jl) {
        float mx = -INFINITY, sum = 0.f, acc = 0.f;
        if (KP > 0) {
            float g[KP > 0 ? KP : 1], k[KP > 0 ? KP : 1], a[KP > 0 ? KP : 1];
#pragma unroll
            for (int m = 0; m < KP; m++) {
                g[m] = idx_row(gc, rg, j * kpool + m, p0, Dk, kpool)[c];
                k[m] = idx_row(kc, rk, j * kpool + m, p0, Dk, kpool)[c];
                a[m] = ape[m * Dk + c];
            }
#pragma unroll
            for (int m = 0; m < KP; m++) mx = fmaxf(mx, g[m] + a[m]);
#pragma unroll
            for (int m = 0; m < KP; m++) {
                const float e = expf(g[m] + a[m] - mx);
                sum += e;
                acc = fmaf(e, k[m], acc);
            }
        } else {
#pragma unroll 4
            for (int m = 0; m < kpool; m++) mx = fmaxf(mx, idx_row(gc, rg, j * kpool + m, p0, Dk, kpool)[c] + ape[m * Dk + c]);
#pragma unroll 4
            for (int m = 0; m < kpool; m++) {
                const int64_t pos = j * kpool + m;
                const float e = expf(idx_row(gc, rg, pos, p0, Dk, kpool)[c] + ape[m * Dk + c] - mx);
                sum += e;
                acc = fmaf(e, idx_row(kc, rk, pos, p0, Dk, kpool)[c], acc);
            }
        }
        P[j * Dk + c] = acc / sum;
    }
    if (blockIdx.y == 0) {
        const int first = max(p0, jl * kpool);
        for (int64_t pos = first; pos < end; pos++) {
            rk[(pos % kpool) * Dk + c] = kc[(pos - p0) * Dk + c];
            rg[(pos % kpool) * Dk + c] = gc[(pos - p0) * Dk + c];
        }
    }
}

// ---- scores on the CUDA cores -------------------------------------------------------------------------------
// Decode and MTP-verify steps (a few queries), and the shapes the tensor form below does not take.  A warp works on 32
// pools x 32 heads at a time, a lane on 4 pools x 8 heads with four running sums each (the columns modulo 4, as two packed
// f32 pairs): per four columns 12 16-byte reads from shared memory feed 64 packed FMAs.  What bounds it is the 128 bytes a
// cycle that shared memory returns to the registers - a 16-byte read costs four cycles even when all lanes read the same
// word - so the register tile decides: 1536 cycles of reads for 32 pools x 32 heads x 128 columns.  The head terms of a pool
// then meet in shared memory and are added in ascending head order.  A block keeps its query and each of its warps walks
// tiles, the next tile's keys in flight while it works on one.
// (32 heads x 128 columns; 8192 pools, one query / 16384 pools, two queries: 7.5 / 13.4 us.  40 / 79 us with one 4-byte read per
// FMA, 8.2 / 22.7 us with a pool's key in a lane's registers and the query row read as broadcast 16-byte words.)
constexpr int SC_POOLS = 32, SC_HEADS = 32, SC_WARPS = 2, SC_C4 = 32;  // Dk <= 4 * SC_C4 = 128
constexpr int SC_ROW = SC_C4 * 4 + 4;                   // rows padded by 16 bytes: eight consecutive rows cover all banks
constexpr int score_smem(int Hq) {
    return (SC_WARPS * (2 * SC_POOLS * SC_ROW + SC_HEADS * SC_POOLS) + Hq * (SC_ROW + 1)) * (int) sizeof(float);
}
// The query rows of a launch sit in shared memory; more heads than fit are worked off in launches of this many, each going
// on with the sums the one before left in `score` (the heads are added in ascending order either way).
constexpr int SC_MAX_HEADS = 9 * SC_HEADS;
static_assert(score_smem(SC_MAX_HEADS) <= 232448, "shared memory of one CTA");
__device__ __forceinline__ void fma_f32x2(uint64_t &d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// q, w: this launch's Hq of the Hq_all heads of every query; GO_ON: after the heads in front of them
template <bool GO_ON>
__global__ void __launch_bounds__(SC_WARPS * 32) k_idx_score(const float *__restrict__ q, const float *__restrict__ w,
                                                             const float *__restrict__ P, float *__restrict__ score,
                                                             int64_t score_stride, int pos0, int kpool, int Hq, int Dk, float scale,
                                                             int Hq_all) {
    extern __shared__ __align__(16) float sc_smem[];
    const int t = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float *sq = sc_smem;                                                             // [Hq][SC_ROW]
    float *sk = sq + Hq * SC_ROW + warp * (2 * SC_POOLS * SC_ROW + SC_HEADS * SC_POOLS);  // this warp's [2][32][SC_ROW]
    float *sr = sk + 2 * SC_POOLS * SC_ROW;                                          // its relu terms [32 heads][32 pools]
    float *sw = sc_smem + Hq * SC_ROW + SC_WARPS * (2 * SC_POOLS * SC_ROW + SC_HEADS * SC_POOLS);  // [Hq]
    const int n_pool = (pos0 + t + 1) / kpool, n_tiles = (n_pool + SC_POOLS - 1) / SC_POOLS;
    const bool vec = (Dk & 3) == 0 && !((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(P)) & 15);
    const int n4 = (Dk + 3) >> 2;                  // columns up to a multiple of four: zeros
    sm100::griddep_wait();
    sm100::griddep_launch_dependents();
    auto load_rows = [&](float *dst, const float *src, int rows, int last, int i0, int n_thr) {  // rows past `last` repeat it
        if (vec) {
            for (int i = i0; i < rows * n4; i += n_thr) {
                const int r = i / n4, c = i - r * n4;
                sm100::cp_async16(dst + r * SC_ROW + c * 4, src + (int64_t) min(r, last) * Dk + c * 4);
            }
        } else {
            for (int i = i0; i < rows * n4 * 4; i += n_thr) {
                const int r = i / (n4 * 4), c = i - r * (n4 * 4);
                dst[r * SC_ROW + c] = c < Dk ? __ldcg(src + (int64_t) min(r, last) * Dk + c) : 0.f;
            }
        }
        sm100::cp_async_commit();
    };
    auto load_tile = [&](int tile, int buf) {      // pools past the end work on a valid row and drop the result
        load_rows(sk + buf * SC_POOLS * SC_ROW, P + (int64_t) tile * SC_POOLS * Dk, SC_POOLS, n_pool - 1 - tile * SC_POOLS, lane, 32);
    };
    const int step = gridDim.x * SC_WARPS;
    int tile = blockIdx.x * SC_WARPS + warp;
    load_rows(sq, q + (int64_t) t * Hq_all * Dk, Hq, Hq - 1, tid, SC_WARPS * 32);
    if (tile < n_tiles) load_tile(tile, 0);
    for (int i = tid; i < Hq; i += SC_WARPS * 32) sw[i] = w[(int64_t) t * Hq_all + i];
    sm100::cp_async_wait_all();
    __syncthreads();
    const int pg = lane >> 2, hg = lane & 3;       // pools pg + 8 j, heads hg + 4 i of a pass
    for (int buf = 0; tile < n_tiles; tile += step, buf ^= 1) {
        sm100::cp_async_wait_all();
        __syncwarp();
        if (tile + step < n_tiles) load_tile(tile + step, buf ^ 1);
        const float *kt = sk + buf * SC_POOLS * SC_ROW + pg * SC_ROW;
        float total = 0.f;
        if (GO_ON && tile * SC_POOLS + lane < n_pool) total = score[(int64_t) t * score_stride + tile * SC_POOLS + lane];
        for (int h0 = 0; h0 < Hq; h0 += SC_HEADS) {
            const int nh = min(SC_HEADS, Hq - h0);
            uint64_t acc[4][8][2];
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int i = 0; i < 8; i++) acc[j][i][0] = acc[j][i][1] = 0;
            const float *qh[8];  // heads past the last repeat it
#pragma unroll
            for (int i = 0; i < 8; i++) qh[i] = sq + (h0 + min(hg + 4 * i, nh - 1)) * SC_ROW;
#pragma unroll 2
            for (int c = 0; c < n4; c++) {
                ulonglong2 k[4];
#pragma unroll
                for (int j = 0; j < 4; j++) k[j] = *reinterpret_cast<const ulonglong2 *>(kt + j * 8 * SC_ROW + c * 4);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(qh[i] + c * 4);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        fma_f32x2(acc[j][i][0], v.x, k[j].x);
                        fma_f32x2(acc[j][i][1], v.y, k[j].y);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float2 a = *reinterpret_cast<const float2 *>(&acc[j][i][0]), b = *reinterpret_cast<const float2 *>(&acc[j][i][1]);
                    sr[(hg + 4 * i) * SC_POOLS + pg + 8 * j] = fmaxf(((a.x + a.y) + (b.x + b.y)) * scale, 0.f);
                }
            __syncwarp();
#pragma unroll 8
            for (int h = 0; h < nh; h++) total = fmaf(sw[h0 + h], sr[h * SC_POOLS + lane], total);
            __syncwarp();
        }
        const int p = tile * SC_POOLS + lane;
        if (p < n_pool) score[(int64_t) t * score_stride + p] = total;
    }
}

// Up to three heads (from 16 queries on, four): a key is used so little that staging it costs more than it saves.  Block = 64 pools x 4 column parts; thread
// (pool, part) holds columns part, part + 4, ... of its pool's key in registers and joins the parts by two shuffles: the same
// sums.  (One head x 128 columns, 64 queries x 8192 pools: 74 us this way, 230 with the register tiles; four heads
// x 64 columns 93 / 107 us, of one query 5.4 / 5.1.)
constexpr int SF_POOLS = 64, SF_PARTS = 4, SF_MAXI = 32, SF_HEADS = 4;  // Dk <= SF_PARTS * SF_MAXI
__global__ void __launch_bounds__(SF_POOLS * SF_PARTS) k_idx_score_few(const float *__restrict__ q, const float *__restrict__ w,
                                                                      const float *__restrict__ P, float *__restrict__ score,
                                                                      int64_t score_stride, int pos0, int kpool, int Hq, int Dk, float scale) {
    __shared__ float sq[SF_HEADS * SF_PARTS * SF_MAXI], sw[SF_HEADS];
    const int t = blockIdx.y, n_pool = (pos0 + t + 1) / kpool, p_base = blockIdx.x * SF_POOLS;
    sm100::griddep_wait();
    sm100::griddep_launch_dependents();
    if (p_base >= n_pool) return;
    const float *qt = q + (int64_t) t * Hq * Dk;
    for (int i = threadIdx.x; i < Hq * Dk; i += SF_POOLS * SF_PARTS) sq[i] = qt[i];
    if (threadIdx.x < Hq) sw[threadIdx.x] = w[(int64_t) t * Hq + threadIdx.x];
    const int part = threadIdx.x & (SF_PARTS - 1), p = p_base + threadIdx.x / SF_PARTS;
    const float *pk = P + (int64_t) min(p, n_pool - 1) * Dk;  // (pools past the end work on a valid row and drop the result)
    float key[SF_MAXI];
#pragma unroll
    for (int i = 0; i < SF_MAXI; i++) key[i] = i * SF_PARTS + part < Dk ? pk[i * SF_PARTS + part] : 0.f;
    __syncthreads();
    float total = 0.f;
    for (int h = 0; h < Hq; h++) {
        float d = 0.f;
#pragma unroll
        for (int i = 0; i < SF_MAXI; i++)
            if (i * SF_PARTS < Dk) d = fmaf(i * SF_PARTS + part < Dk ? sq[h * Dk + i * SF_PARTS + part] : 0.f, key[i], d);
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        total = fmaf(sw[h], fmaxf(d * scale, 0.f), total);
    }
    if (part == 0 && p < n_pool) score[(int64_t) t * score_stride + p] = total;
}

// ---- scores of a prefill block on the tensor cores ----------------------------------------------------------
// 2 T pools Hq Dk operations: 17 GFLOP for 256 queries x 8192 pools x 32 heads x 128 columns, 0.23 ms at the f32 peak of
// the CUDA cores.  The scores decide an exact top-k, so f32 precision has to stay: every f32 value is the sum of three
// bf16 values (8 significand bits each, x = x1 + x2 + x3 exactly), and of the nine products of two such sums the six
// with a weight above 2^-24 are formed on tcgen05: x1 y3, x3 y1, x2 y2, x1 y2, x2 y1, x1 y1.  The tensor core truncates at
// every accumulation, so the large products come last, and every block of 64 columns has an f32 accumulator of its own:
// four steps on a large sum instead of 48 (rms error against float64 of 256 x 8192 scores of rms 2.3: 3.2e-7 on the CUDA
// cores, 1.4e-6 with one accumulator, 2.7e-7 this way).
//   D[128 pools x 64] = P_tile[128 x Dk] . Q_unit[64 x Dk]^T   per unit; columns = the heads of 64 / Hq queries.
// Pools fill the 128 lanes, so that the sum over a query's heads runs inside one thread and the scores of 32 consecutive
// pools leave in one line.  A CTA walks consecutive units (pool tile major): the three parts of its pool tile stay in
// tensor memory (192 columns), the query rows stream through a shared-memory ring of 64-column blocks (3 x 8 KB each).
// Eight warps read the f32 query rows (bulk copies from L2), split them and write the swizzled operand blocks; two threads issue the
// 48 MMAs of a unit (M = 128, N = 64, K = 16, A in tensor memory: 33 cycles each); four warps load and split the pool
// tile, and read the finished accumulators (two sets in tensor memory) for scale, relu, weight and sum.
// Why A is in tensor memory: with both operands in shared memory (128 columns per unit, 65 cycles per MMA) the MMAs alone
// take 126 of the 128 bytes a cycle shared memory delivers, and the splitting warps' stores come on top.
// 256 queries x 8192 pools x 32 heads x 128 columns: 78 us (2892 on the CUDA cores before); the tensor pipe is active in two
// thirds of the cycles, the rest is the splitting of the query rows, which every pool tile repeats, and a start of 4 us.
constexpr int ST_M = 128, ST_N = 64;                  // pools and query-head columns of a unit
constexpr int ST_BLK = ST_N * 128;                    // bytes of one [64 rows][64 columns] bf16 block
constexpr int ST_PARTS = 3;
constexpr int ST_STAGE = ST_PARTS * ST_BLK;           // one 64-column block of the query rows, three parts
constexpr int ST_STAGES = 6;
constexpr int ST_RAW = ST_N * 128 * 4, ST_RAWS = 2;    // the query rows of a unit as they are, f32
// warps 0-7 pool tile and epilogue (two groups, units of even / odd number), 8-15 conversion (two groups, ring stages of
// even / odd number), 16 copies of the query rows, then one MMA-issuing warp per column block
constexpr int ST_CONV_WARP0 = 8, ST_LOAD_WARP = 16, ST_MMA_WARP0 = 17;
constexpr int st_threads(int kb) { return 32 * (ST_MMA_WARP0 + kb); }
constexpr int ST_A_COL = 4 * ST_N;                    // tensor memory: two pairs of accumulators, then the pool tile's parts

__device__ int32_t g_idx_status;                      // sticky: a bounded wait of the kernel below gave up

struct ScoreParams {
    const float *q, *w, *P;
    float *score;
    int64_t score_stride;
    int pos0, T, kpool, Hq, Dk;
    float scale;
    int n_pools;        // complete pools of the last query: rows of P that may be read
    int tok;            // queries per unit
    int n_tg;           // units per pool tile
    int n_units;
};

struct ScoreMisc {
    uint64_t raw_full[ST_RAWS], raw_empty[ST_RAWS], b_full[ST_STAGES], b_empty[ST_STAGES], d_full[2], d_empty[2], a_full;
    uint32_t tmem_base;
    int abort_flag;
    alignas(16) float w[2][ST_N];
};
constexpr int ST_SMEM = ST_RAWS * ST_RAW + ST_STAGES * ST_STAGE + (int) sizeof(ScoreMisc) + 1024;

// Two f32 values -> packed pairs of the three bf16 parts.
__device__ __forceinline__ void split3(float x, float y, uint32_t &w1, uint32_t &w2, uint32_t &w3) {
    const __nv_bfloat162 h1 = __floats2bfloat162_rn(x, y);
    const float2 f1 = __bfloat1622float2(h1);
    const float rx = x - f1.x, ry = y - f1.y;      // exact
    const __nv_bfloat162 h2 = __floats2bfloat162_rn(rx, ry);
    const float2 f2 = __bfloat1622float2(h2);
    const __nv_bfloat162 h3 = __floats2bfloat162_rn(rx - f2.x, ry - f2.y);
    w1 = *reinterpret_cast<const uint32_t *>(&h1);
    w2 = *reinterpret_cast<const uint32_t *>(&h2);
    w3 = *reinterpret_cast<const uint32_t *>(&h3);
}

// One score in f32 on this thread, with the sums of the CUDA-core form: for values the split cannot hold.  An infinite or
// near-maximal operand splits into infinity and x - infinity, every sum it enters is NaN, and relu makes that a 0 where an f32
// sum keeps the infinity.  (Out of line: nobody should come here.)
static __device__ __noinline__ float score_f32(const ScoreParams &S, int t, int p) {
    const float *k = S.P + (int64_t) p * S.Dk;
    float total = 0.f;
    for (int h = 0; h < S.Hq; h++) {
        const float *v = S.q + ((int64_t) t * S.Hq + h) * S.Dk;
        float a[4] = {0.f, 0.f, 0.f, 0.f};
        for (int c = 0; c < S.Dk; c += 4)  // (Dk is a multiple of four in this form)
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = fmaf(v[c + i], k[c + i], a[i]);
        total = fmaf(S.w[(int64_t) t * S.Hq + h], fmaxf(((a[0] + a[1]) + (a[2] + a[3])) * S.scale, 0.f), total);
    }
    return total;
}

// relu that passes a NaN on, so that it is seen in the total.
__device__ __forceinline__ float relu_nan(float x) {
    float r;
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(x));
    return r;
}

// KB: 64-column blocks of a row (Dk <= 64 * KB)
template <int KB>
__global__ void __launch_bounds__(st_threads(KB), 1) k_idx_score_umma(const ScoreParams S) {
    using namespace sm100;
    extern __shared__ uint8_t st_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(st_raw) + 1023) & ~(uintptr_t) 1023);
    uint8_t *raw_smem = smem + ST_STAGES * ST_STAGE;
    ScoreMisc &M = *reinterpret_cast<ScoreMisc *>(raw_smem + ST_RAWS * ST_RAW);
    volatile int *abort_flag = &M.abort_flag;
    int32_t *status = &g_idx_status;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < ST_STAGES; i++) {
            mbar_init(&M.b_full[i], 4);
            mbar_init(&M.b_empty[i], 1);
        }
        for (int i = 0; i < ST_RAWS; i++) {
            mbar_init(&M.raw_full[i], 1);
            mbar_init(&M.raw_empty[i], KB * 4);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&M.d_full[i], KB);
            mbar_init(&M.d_empty[i], 4);
        }
        mbar_init(&M.a_full, 8);
        M.abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == ST_MMA_WARP0) {
        tmem_alloc(&M.tmem_base, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = M.tmem_base;
    griddep_wait();
    griddep_launch_dependents();
    // consecutive units, the counts of two CTAs differ by at most one
    const int u0 = (int) ((int64_t) S.n_units * blockIdx.x / gridDim.x), u1 = (int) ((int64_t) S.n_units * (blockIdx.x + 1) / gridDim.x);

    if (warp >= ST_CONV_WARP0 && warp < ST_LOAD_WARP) {
        // ---- conversion of the query rows: f32 -> three swizzled bf16 blocks.  Group g takes the ring stages g, g + 2, ...
        // (two column blocks per row: always column block g).  Thread = (row mod 8, 16 bytes of f32), eight rows.
        const int g = (warp - ST_CONV_WARP0) >> 2, ct = (tid - ST_CONV_WARP0 * 32) & 127, c4 = ct & 15, r0 = ct >> 4;
        const uint32_t off0 = (uint32_t) (r0 * 128 + (((c4 >> 1) ^ (r0 & 7)) << 4) + (c4 & 1) * 8);  // rows 8 apart share r mod 8
        const int u_step = KB == 2 ? 1 : 2, n_u = u1 - u0;
        const int col = (KB == 2 ? g * 64 : 0) + c4 * 4;
        const bool col_ok = col < S.Dk;
        const uint32_t src0 = (uint32_t) (r0 * S.Dk + col) * 4, row_step = (uint32_t) S.Dk * 32;
        int st = g, tg = (u0 + (KB == 2 ? 0 : g)) % S.n_tg;
        uint32_t st_ph = 1;
        for (int i = KB == 2 ? 0 : g; i < n_u; i += u_step) {
            const int rb = i % ST_RAWS, n_rows = min(S.tok, S.T - tg * S.tok) * S.Hq;
            tg += u_step;
            while (tg >= S.n_tg) tg -= S.n_tg;
            if (!mbar_wait(&M.raw_full[rb], (i / ST_RAWS) & 1, abort_flag, status, 1)) break;
            const uint8_t *src = raw_smem + rb * ST_RAW + src0;
            float4 v[8];
#pragma unroll
            for (int k = 0; k < 8; k++)
                v[k] = col_ok && r0 + k * 8 < n_rows ? *reinterpret_cast<const float4 *>(src + k * row_step) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (!mbar_wait(&M.b_empty[st], st_ph, abort_flag, status, 1)) break;
            uint8_t *dst = smem + st * ST_STAGE + off0;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                uint2 p1, p2, p3;
                split3(v[k].x, v[k].y, p1.x, p2.x, p3.x);
                split3(v[k].z, v[k].w, p1.y, p2.y, p3.y);
                *reinterpret_cast<uint2 *>(dst + k * 8 * 128) = p1;
                *reinterpret_cast<uint2 *>(dst + k * 8 * 128 + ST_BLK) = p2;
                *reinterpret_cast<uint2 *>(dst + k * 8 * 128 + 2 * ST_BLK) = p3;
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&M.b_full[st]);
                mbar_arrive(&M.raw_empty[rb]);
            }
            st += 2;
            if (st >= ST_STAGES) {
                st -= ST_STAGES;
                st_ph ^= 1;
            }
        }
    } else if (warp == ST_LOAD_WARP) {
        // ---- the query rows of a unit are consecutive in memory: one bulk copy (loads by the converting threads took the
        // same time, but 64 registers more each for what has to be in flight)
        int tg = u0 % S.n_tg;
        for (int i = 0; i < u1 - u0; i++) {
            const int rb = i % ST_RAWS, n_rows = min(S.tok, S.T - tg * S.tok) * S.Hq;
            if (!mbar_wait(&M.raw_empty[rb], ((i / ST_RAWS) & 1) ^ 1, abort_flag, status, 1)) break;
            if (elect_one()) {
                const uint32_t bytes = (uint32_t) (n_rows * S.Dk) * 4;
                mbar_arrive_expect_tx(&M.raw_full[rb], bytes);
                bulk_load(raw_smem + rb * ST_RAW, S.q + (int64_t) tg * S.tok * S.Hq * S.Dk, bytes, &M.raw_full[rb]);
            }
            __syncwarp();
            if (++tg == S.n_tg) tg = 0;
        }
    } else if (warp >= ST_MMA_WARP0) {
        // ---- MMA issue: warp kb of these takes column block kb of every unit, with an accumulator of its own (one issuing
        // thread gets about 65 cycles per MMA here, two keep the pipe at its own rate)
        const int kb = warp - ST_MMA_WARP0;
        constexpr uint32_t idesc = make_idesc_bf16(ST_M, ST_N, 0, 0);
        const uint64_t d_kmaj = make_smem_desc(0, 16, 1024, kSwizzle128B);
        const uint32_t b_lo = smem_u32(smem) >> 4, as = tmem + ST_A_COL + kb * 32;
        int n_a = 0, un = 0, st = kb, left = 0, tg = u0 % S.n_tg;
        uint32_t st_ph = 0;
        bool ok = true;
        for (int u = u0; ok && u < u1; u++, un++) {
            if (left == 0) {  // a new pool tile
                left = S.n_tg - tg;
                tg = 0;
                ok = mbar_wait(&M.a_full, n_a & 1, abort_flag, status, 2);
                n_a++;
            }
            left--;
            bool lane_ok = mbar_wait_lane(&M.d_empty[un & 1], ((un >> 1) & 1) ^ 1, abort_flag, status, 2);
            lane_ok &= mbar_wait_lane(&M.b_full[st], st_ph, abort_flag, status, 2);
            ok = __all_sync(0xffffffffu, ok && lane_ok);
            if (!ok) break;
            const uint32_t d = tmem + (un & 1) * 2 * ST_N + kb * ST_N;
            const uint64_t bd = d_kmaj + (b_lo + st * (ST_STAGE >> 4));
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int pr = 0; pr < 6; pr++) {
                    // the small products first: (1,3) (3,1) (2,2) (1,2) (2,1) (1,1)
                    constexpr int pa[6] = {0, 2, 1, 0, 1, 0}, pb[6] = {2, 0, 1, 1, 0, 0};
#pragma unroll
                    for (int ks = 0; ks < 4; ks++)
                        umma_ts(d, as + pa[pr] * 64 + ks * 8, bd + (pb[pr] * (ST_BLK >> 4) + ks * 2), idesc, pr > 0 || ks > 0);
                }
                umma_commit(&M.b_empty[st]);
                umma_commit(&M.d_full[un & 1]);
            }
            __syncwarp();
            st += KB;
            if (st >= ST_STAGES) {
                st -= ST_STAGES;
                st_ph ^= 1;
            }
        }
    } else {
        // ---- pool tile and epilogue: thread = one pool.  Both groups walk all units: each loads half of every new pool
        // tile, group g finishes the units of number g, g + 2, ...
        const int g = warp >> 2, row = tid & 127;
        const uint32_t lane_base = (uint32_t) ((warp & 3) * 32) << 16;
        const int n_w = S.T * S.Hq, cpt = S.Hq >> 4;  // 16-column chunks per query
        int un = 0, pt = u0 / S.n_tg, tg = u0 - pt * S.n_tg;
        bool new_tile = true;
        auto weight = [&](int t_unit) {  // thread i < 64: the weight of column i of the unit
            const int wi = t_unit * S.tok * S.Hq + row;
            return row < ST_N && wi < n_w ? __ldcg(S.w + wi) : 0.f;
        };
        float w_next = weight((u0 + g) % S.n_tg);
        for (int u = u0; u < u1; u++, un++, tg++) {
            if (tg == S.n_tg) {
                tg = 0;
                pt++;
                new_tile = true;
            }
            const int p = pt * ST_M + row;
            if (new_tile) {
                new_tile = false;
                // the MMAs of the old tile are over when its last unit's accumulators are complete; if that does not come, they
                // may still be reading the old parts, which then stay (the waits for the new ones end with the abort flag)
                const bool over = un == 0 || mbar_wait(&M.d_full[(un - 1) & 1], ((un - 1) >> 1) & 1, abort_flag, status, 4);
                tc_fence_after();  // (group g has ordered itself behind its own units only)
                if (over) {
                    const float *src = S.P + (int64_t) p * S.Dk;
                    float4 x[KB][8];
#pragma unroll
                    for (int i = 0; i < KB; i++)
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            const int c = (g * KB + i) * 32 + j * 4;
                            x[i][j] = p < S.n_pools && c < S.Dk ? __ldcg(reinterpret_cast<const float4 *>(src + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
                        }
#pragma unroll
                    for (int i = 0; i < KB; i++) {
                        uint32_t p1[16], p2[16], p3[16];
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            split3(x[i][j].x, x[i][j].y, p1[2 * j], p2[2 * j], p3[2 * j]);
                            split3(x[i][j].z, x[i][j].w, p1[2 * j + 1], p2[2 * j + 1], p3[2 * j + 1]);
                        }
                        const uint32_t a = tmem + lane_base + ST_A_COL + (g * KB + i) * 16;
                        tmem_st16(a, p1);
                        tmem_st16(a + 64, p2);
                        tmem_st16(a + 128, p3);
                    }
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&M.a_full);
                }
            }
            if ((un & 1) != g) continue;
            const int t0 = tg * S.tok, n_tok = min(S.tok, S.T - t0);
            // the weights of this unit's queries (each group has a buffer of its own)
            if (group_any(1 + g, 128, *abort_flag != 0)) break;  // (one decision for the group; the old weights are read)
            if (row < ST_N) M.w[g][row] = w_next;
            w_next = weight(tg + 2 < S.n_tg ? tg + 2 : (tg + 2) % S.n_tg);
            named_bar_sync(1 + g, 128);
            const bool ok = mbar_wait(&M.d_full[g], (un >> 1) & 1, abort_flag, status, 4);
            tc_fence_after();
            // 16 columns of both accumulators at a time, the next 16 in flight while these are worked on
            const uint32_t d_addr = tmem + lane_base + g * 2 * ST_N;
            uint32_t r[2][16], e[2][16];
            tmem_ld16(d_addr, r[0]);
            if (KB == 2) tmem_ld16(d_addr + ST_N, e[0]);
            float total = 0.f;
            int k = 0, left = cpt, redo = 0;
#pragma unroll
            for (int c = 0; c < ST_N / 16; c++) {
                tmem_wait_ld();
                if (c + 1 < ST_N / 16) {
                    tmem_ld16(d_addr + (c + 1) * 16, r[(c + 1) & 1]);
                    if (KB == 2) tmem_ld16(d_addr + ST_N + (c + 1) * 16, e[(c + 1) & 1]);
                } else {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&M.d_empty[g]);
                }
                const float4 *w4 = reinterpret_cast<const float4 *>(&M.w[g][c * 16]);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float4 wv = w4[i];
                    auto term = [&](int j, float wj) {
                        float d = __uint_as_float(r[c & 1][4 * i + j]);
                        if (KB == 2) d += __uint_as_float(e[c & 1][4 * i + j]);
                        total = fmaf(wj, relu_nan(d * S.scale), total);
                    };
                    term(0, wv.x);
                    term(1, wv.y);
                    term(2, wv.z);
                    term(3, wv.w);
                }
                if (--left == 0) {  // the query's last chunk
                    if (ok && k < n_tok && p < (S.pos0 + t0 + k + 1) / S.kpool) {
                        S.score[(int64_t) (t0 + k) * S.score_stride + p] = total;
                        if (!(fabsf(total) <= 3.402823466e+38f)) redo |= 1 << k;
                    }
                    total = 0.f;
                    k++;
                    left = cpt;
                }
            }
            if (redo) {  // (behind the loop: a call inside it would spill the columns in flight)
                for (k = 0; k < n_tok; k++)
                    if ((redo >> k) & 1) S.score[(int64_t) (t0 + k) * S.score_stride + p] = score_f32(S, t0 + k, p);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && tid == 0) {  // MMAs that were issued may still be reading shared memory
        const long long c0 = clock64();
        while (clock64() - c0 < 2000000LL) {
        }
    }
    __syncthreads();
    if (warp == ST_MMA_WARP0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// ---- selection ----------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t f2ord(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// One block per query.  Selection on the order-preserving integer image: a histogram of the top 12 bits gives the bin the
// k-th largest value lies in; the values of that bin (about 2 % of them) go to a list, from which further digits of 10 bits
// are taken (from all values when it does not fit) until it is short enough for every value in it to count the larger and
// the equal ones.  Then one ordered pass writes the list of positions: ballots of "greater" and "equal" flags of 32
// consecutive pools each, one scan over the counts, and a thread per ballot (a warp when they are few) writes the pools it
// holds - the pools appear in ascending index and ties go to the lowest indices.
// Latency-bound (32 KB of scores at 32K positions): what counts is the number of passes and barriers and the chains within
// them.  The image is kept in shared memory when it fits, so memory is read once, eight loads in flight per thread; the
// first digit is wide because eight bits of a float are little more than its sign and exponent - nearly all values then
// share a few bins and the shared-memory atomics serialise, here a warp's values spread over 50 bins and more.
// (8192 pools, one query / 256 queries: 6.6 / 13.6 us; 17 / 36 us with four 8-bit passes over global memory and an ordered pass
// with three barriers per 1024 pools.)
constexpr int SEL_NT = 512, SEL_NW = SEL_NT / 32, SEL_BINS = 4096;
constexpr int SEL_CACHE = 36864;          // scores of a query kept in shared memory (144 KB)
constexpr int SEL_LIST = 2048;            // values of the k-th largest value's bin kept in a list
constexpr int SEL_RANK = 128;             // a list up to this long is ranked value by value (all against all), longer ones take a digit first
constexpr int SEL_SLAB = 4 * SEL_NT;      // groups of 32 pools the ordered pass takes at once
constexpr int SEL_WIDE = 64;              // with no more groups than this in a slab, a warp writes a group
struct SelSmem {
    union {
        alignas(16) uint32_t hist[SEL_BINS];
        uint2 flags[SEL_SLAB];            // ordered pass: ballots of "greater" and "equal"
    };
    alignas(16) uint32_t list[SEL_LIST];
    uint2 base[SEL_WIDE];                 // greater and equal values in front of a group
    uint32_t wsum[2][32];
    uint32_t digit, need, n_list;
};
static_assert(SEL_SLAB * 8 <= SEL_BINS * 4, "the ballots lie over the bins");

// Inclusive sum over the lanes of a warp.
__device__ __forceinline__ uint32_t warp_scan(uint32_t v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

// One digit: counts of the bins from the top, PER bins per thread; exactly one thread owns the bin in which the running
// count reaches `need` (need >= 1) and leaves the digit and what is still needed in S.
template <int PER>
__device__ __forceinline__ void select_digit(SelSmem &S, uint32_t need) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int BINS = PER * SEL_NT;
    uint32_t mine[PER], tot = 0;
    // thread i owns bins [BINS - PER (i + 1), BINS - PER i), taken from the top
#pragma unroll
    for (int i = 0; i < PER; i += 2) {
        const uint2 v = *reinterpret_cast<const uint2 *>(&S.hist[BINS - PER * (tid + 1) + PER - 2 - i]);
        mine[i] = v.y;
        mine[i + 1] = v.x;
        tot += v.x + v.y;
    }
    const uint32_t incl = warp_scan(tot, lane);
    if (lane == 31) S.wsum[0][warp] = incl;
    __syncthreads();
    const uint32_t ws = warp_scan(lane < SEL_NW ? S.wsum[0][lane] : 0u, lane);
    const uint32_t prev = __shfl_sync(0xffffffffu, ws, warp > 0 ? warp - 1 : 0);
    uint32_t above = incl - tot + (warp > 0 ? prev : 0u);  // values in higher bins
    if (above < need && above + tot >= need) {
#pragma unroll
        for (int i = 0; i < PER; i++) {
            if (above < need && above + mine[i] >= need) {
                S.digit = (uint32_t) (BINS - PER * tid - 1 - i);
                S.need = need - above;
            }
            above += mine[i];
        }
    }
    __syncthreads();
}

template <bool CACHED>
__global__ void __launch_bounds__(SEL_NT) k_idx_select(const float *__restrict__ score, int64_t score_stride, int pos0, int kpool,
                                                       int top_k, int *__restrict__ sel, int sel_stride, int *__restrict__ cnt) {
    __shared__ SelSmem S;
    extern __shared__ uint32_t sel_img[];
    const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int pos = pos0 + t;
    const int n_pool = (pos + 1) / kpool;
    int *out = sel + (int64_t) t * sel_stride;
    for (int i = tid; i < SEL_BINS / 4; i += SEL_NT) reinterpret_cast<uint4 *>(S.hist)[i] = make_uint4(0, 0, 0, 0);
    if (tid == 0) S.n_list = 0;
    __syncthreads();
    sm100::griddep_wait();
    sm100::griddep_launch_dependents();
    if (n_pool <= top_k) {  // everything is attended (ops.cu:728-731)
        for (int i = tid; i <= pos; i += SEL_NT) out[i] = i;
        if (tid == 0) cnt[t] = pos + 1;
        return;
    }
    const float *sc = score + (int64_t) t * score_stride;
    // f(value image, valid) for every pool of this thread, eight at a time
    auto for_all = [&](auto f) {
        for (int p0 = tid; p0 < n_pool; p0 += 8 * SEL_NT) {
            uint32_t u[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int p = min(p0 + k * SEL_NT, n_pool - 1);
                u[k] = CACHED ? sel_img[p] : f2ord(__ldcg(sc + p));
            }
#pragma unroll
            for (int k = 0; k < 8; k++) f(u[k], p0 + k * SEL_NT < n_pool);
        }
    };
    uint32_t U = 0xffffffffu, need = 0;  // top_k = 0: nothing exceeds the threshold, nothing equal to it is taken
    if (top_k > 0) {
        for (int p0 = tid; p0 < n_pool; p0 += 8 * SEL_NT) {
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = __ldcg(sc + min(p0 + k * SEL_NT, n_pool - 1));
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int p = p0 + k * SEL_NT;
                const uint32_t u = f2ord(v[k]);
                if (p < n_pool) {
                    if (CACHED) sel_img[p] = u;
                    atomicAdd(&S.hist[u >> 20], 1u);
                }
            }
        }
        __syncthreads();
        select_digit<SEL_BINS / SEL_NT>(S, (uint32_t) top_k);
        const uint32_t top = S.digit;
        U = top << 20;
        need = S.need;
        auto push = [&](uint32_t u) {
            const uint32_t i = atomicAdd(&S.n_list, 1u);
            if (i < SEL_LIST) S.list[i] = u;
        };
        for_all([&](uint32_t u, bool valid) {
            if (valid && u >> 20 == top) push(u);
        });
        __syncthreads();
        int n = (int) S.n_list;
        for (int shift = 20;;) {
            if (n <= SEL_RANK) {
                // thread i ranks value i: the k-th largest has fewer than `need` larger ones and at least `need` not smaller
                if (tid < 8) S.list[n + tid] = 0;  // (the loop takes eight at a time: the smallest image, above nothing)
                __syncthreads();
                if (warp * 32 < n) {
                    const uint32_t mine = tid < n ? S.list[tid] : 0u;
                    uint32_t gt = 0, ge = 0;
                    for (int j = 0; j < n; j += 8) {
                        const uint4 a = *reinterpret_cast<const uint4 *>(&S.list[j]), b = *reinterpret_cast<const uint4 *>(&S.list[j + 4]);
                        const uint32_t v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            gt += v[i] > mine;
                            ge += v[i] >= mine;
                        }
                    }
                    if (tid < n && gt < need && ge >= need) {  // (every thread that holds this value stores the same)
                        S.digit = mine;
                        S.need = need - gt;
                    }
                }
                __syncthreads();
                U = S.digit;
                need = S.need;
                break;
            }
            // ten more bits of it
            const uint32_t known = U >> shift;
            const int sh = shift - 10;
            *reinterpret_cast<uint2 *>(&S.hist[tid * 2]) = make_uint2(0, 0);
            uint32_t mine[SEL_LIST / SEL_NT];
            const bool listed = n <= SEL_LIST;
#pragma unroll
            for (int k = 0; k < SEL_LIST / SEL_NT; k++) mine[k] = S.list[tid + k * SEL_NT];
            __syncthreads();
            if (tid == 0) S.n_list = 0;
            if (listed) {
#pragma unroll
                for (int k = 0; k < SEL_LIST / SEL_NT; k++)
                    if (tid + k * SEL_NT < n) atomicAdd(&S.hist[(mine[k] >> sh) & 1023], 1u);
            } else {
                for_all([&](uint32_t u, bool valid) {
                    if (valid && u >> shift == known) atomicAdd(&S.hist[(u >> sh) & 1023], 1u);
                });
            }
            __syncthreads();
            select_digit<2>(S, need);
            U |= S.digit << sh;
            need = S.need;
            shift = sh;
            if (shift == 0) break;
            if (listed) {
#pragma unroll
                for (int k = 0; k < SEL_LIST / SEL_NT; k++)
                    if (tid + k * SEL_NT < n && mine[k] >> shift == U >> shift) push(mine[k]);
            } else {
                for_all([&](uint32_t u, bool valid) {
                    if (valid && u >> shift == U >> shift) push(u);
                });
            }
            __syncthreads();
            n = (int) S.n_list;
        }
    }
    const uint32_t need_eq = need;  // take every value above U and the first need_eq values equal to it
    const bool vec4 = kpool == 4 && !(reinterpret_cast<uintptr_t>(out) & 15);
    uint32_t run_gt = 0, run_eq = 0;            // greater and equal values in front of the groups at hand
    for (int slab = 0; slab < n_pool; slab += SEL_SLAB * 32) {
        const int n = min(n_pool - slab, SEL_SLAB * 32), groups = (n + 31) >> 5;
        __syncthreads();
        for (int g0 = warp; g0 < groups; g0 += 8 * SEL_NW) {
            uint32_t u[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int p = slab + min((g0 + k * SEL_NW) * 32 + lane, n - 1);
                u[k] = CACHED ? sel_img[p] : f2ord(__ldcg(sc + p));
            }
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int g = g0 + k * SEL_NW;
                const bool valid = g * 32 + lane < n;
                const uint32_t b_gt = __ballot_sync(0xffffffffu, valid && u[k] > U), b_eq = __ballot_sync(0xffffffffu, valid && u[k] == U);
                if (lane == 0 && g < groups) S.flags[g] = make_uint2(b_gt, b_eq);
            }
        }
        __syncthreads();
        for (int gb = 0; gb < groups; gb += SEL_NT) {  // a thread per group
            uint2 f = gb + tid < groups ? S.flags[gb + tid] : make_uint2(0u, 0u);
            const uint32_t ig = warp_scan(__popc(f.x), lane), ie = warp_scan(__popc(f.y), lane);
            if (lane == 31) {
                S.wsum[0][warp] = ig;
                S.wsum[1][warp] = ie;
            }
            __syncthreads();
            const uint32_t wg = warp_scan(lane < SEL_NW ? S.wsum[0][lane] : 0u, lane), we = warp_scan(lane < SEL_NW ? S.wsum[1][lane] : 0u, lane);
            const uint32_t pg = __shfl_sync(0xffffffffu, wg, warp > 0 ? warp - 1 : 0), pe = __shfl_sync(0xffffffffu, we, warp > 0 ? warp - 1 : 0);
            uint32_t gt = run_gt + (warp > 0 ? pg : 0u) + ig - __popc(f.x), eq = run_eq + (warp > 0 ? pe : 0u) + ie - __popc(f.y);
            if (groups <= SEL_WIDE) {
                // few groups: every thread would write the pools of its group one by one (512 of 600: 27 each); a warp takes a
                // group instead, a lane per pool
                if (tid < SEL_WIDE) S.base[tid] = make_uint2(gt, eq);
                __syncthreads();
                for (int g = warp; g < groups; g += SEL_NW) {
                    const uint2 m = S.flags[g], b = S.base[g];
                    const uint32_t below = (1u << lane) - 1;
                    const bool is_gt = (m.x >> lane) & 1, is_eq = (m.y >> lane) & 1;
                    const uint32_t e = b.y + __popc(m.y & below);
                    if (is_gt || (is_eq && e < need_eq)) {
                        const int64_t slot = (int64_t) (b.x + __popc(m.x & below) + min(e, need_eq)) * kpool;
                        const int first = (slab + g * 32 + lane) * kpool;
                        if (vec4) *reinterpret_cast<int4 *>(out + slot) = make_int4(first, first + 1, first + 2, first + 3);
                        else for (int i = 0; i < kpool; i++) out[slot + i] = first + i;
                    }
                }
            } else for (uint32_t m = f.x | f.y; m; m &= m - 1) {
                const int b = __ffs(m) - 1;
                const bool is_gt = (f.x >> b) & 1;
                if (is_gt || eq < need_eq) {
                    const int64_t slot = (int64_t) (gt + min(eq, need_eq)) * kpool;  // taken pools in front of this one
                    const int first = (slab + (gb + tid) * 32 + b) * kpool;
                    if (vec4) *reinterpret_cast<int4 *>(out + slot) = make_int4(first, first + 1, first + 2, first + 3);
                    else for (int i = 0; i < kpool; i++) out[slot + i] = first + i;
                }
                gt += is_gt;
                eq += !is_gt;
            }
            run_gt += __shfl_sync(0xffffffffu, wg, 31);
            run_eq += __shfl_sync(0xffffffffu, we, 31);
            __syncthreads();  // wsum is written again
        }
    }
    const int base = top_k * kpool, tail0 = n_pool * kpool;
    for (int i = tid; tail0 + i <= pos; i += SEL_NT) out[base + i] = tail0 + i;
    if (tid == 0) cnt[t] = base + (pos + 1 - tail0);
}

template <int KB>
int launch_score_umma(const ScoreParams &S, int sm_count, cudaStream_t st) {
    // attributes are set on every call: a cached flag would go stale across a device reset
    GS_TRY(cudaFuncSetAttribute(k_idx_score_umma<KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_SMEM));
    return launch_pdl(k_idx_score_umma<KB>, dim3(S.n_units < sm_count ? S.n_units : sm_count), st_threads(KB), ST_SMEM, st, S);
}

}  // namespace

int read_idx_status(int32_t *out) {
    GS_TRY(cudaMemcpyFromSymbol(out, g_idx_status, sizeof(int32_t)));
    return 0;
}

}  // namespace gs

using namespace gs;

GS_EXPORT int gs_idx_pool(const float *kc, const float *gc, float *rk, float *rg, const float *ape, float *P, int p0, int T,
                          int Dk, int kpool, void *stream) {
    if (T <= 0) return 0;
    if (p0 < 0 || Dk <= 0 || kpool <= 0) return fail_invalid("gs_idx_pool: need p0 >= 0, Dk > 0, kpool > 0");
    if (!kc || !gc || !rk || !rg || !ape || !P) return fail_invalid("gs_idx_pool: null pointer");
    const int jf = p0 / kpool, jl = (p0 + T) / kpool;
    const int n_pools = jl - jf;
    if (n_pools > 65535) return fail_invalid("gs_idx_pool: more than 65535 pools complete in one call");
    dim3 grid((Dk + 127) / 128, n_pools > 0 ? n_pools : 1);
    auto kernel = kpool == 4 ? k_idx_pool<4> : k_idx_pool<0>;
    return launch_pdl(kernel, grid, 128, 0, (cudaStream_t) stream, kc, gc, rk, rg, ape, P, p0, T, Dk, kpool);
}

GS_EXPORT int gs_idx_score(const float *q, const float *w, const float *P, float *score, int64_t score_stride, int pos0, int T,
                           int kpool, int Hq, int Dk, float scale, void *stream) {
    if (kpool <= 0) return fail_invalid("gs_idx_score: kpool <= 0");
    const int max_pool = (pos0 + T) / kpool;
    if (max_pool <= 0 || T <= 0) return 0;  // ops.cu:703
    if (Dk > 128 || Dk <= 0) return fail_invalid("gs_idx_score: Dk must be 1..128");  // ops.cu:704
    if (Hq <= 0 || (int64_t) Hq * (Dk + 1) * 4 > 48 * 1024) return fail_invalid("gs_idx_score: Hq * Dk beyond 12288");
    if (T > 65535) return fail_invalid("gs_idx_score: T > 65535");
    if (!q || !w || !P || !score) return fail_invalid("gs_idx_score: null pointer");
    int sms = 0, dev = 0;
    GS_TRY(cudaGetDevice(&dev));
    GS_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // The tensor form costs about 8 us plus 0.3 us a query, the CUDA-core form about 3 us a query (8192 pools, 32 heads,
    // 128 columns): from 5 queries on the tensor form.  It reads whole float4s and sums 16 heads at a time.
    if (T >= 5 && Hq % 16 == 0 && Hq <= ST_N && Dk % 4 == 0 && !((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(P)) & 15)) {
        ScoreParams S{};
        S.q = q;
        S.w = w;
        S.P = P;
        S.score = score;
        S.score_stride = score_stride;
        S.pos0 = pos0;
        S.T = T;
        S.kpool = kpool;
        S.Hq = Hq;
        S.Dk = Dk;
        S.scale = scale;
        S.n_pools = max_pool;
        S.tok = ST_N / Hq;
        S.n_tg = (T + S.tok - 1) / S.tok;
        const int64_t units = (int64_t) ((max_pool + ST_M - 1) / ST_M) * S.n_tg;
        if (units < (1ll << 31)) {
            S.n_units = (int) units;
            return Dk <= 64 ? launch_score_umma<1>(S, sms, (cudaStream_t) stream) : launch_score_umma<2>(S, sms, (cudaStream_t) stream);
        }
    }
    if (Hq < SF_HEADS || (Hq == SF_HEADS && T >= 16))
        return launch_pdl(k_idx_score_few, dim3((max_pool + SF_POOLS - 1) / SF_POOLS, T), SF_POOLS * SF_PARTS, 0, (cudaStream_t) stream, q, w, P, score,
                          score_stride, pos0, kpool, Hq, Dk, scale);
    // two blocks fit an SM: no more than they hold at once (one block over and a second, nearly empty round doubles the time:
    // 16 queries x 8192 pools x 8 heads 73 us with 304 blocks, 39 with 288)
    const int tiles = (max_pool + SC_POOLS - 1) / SC_POOLS, blocks = (tiles + SC_WARPS - 1) / SC_WARPS, want = 2 * sms > T ? 2 * sms / T : 1;
    const dim3 grid(blocks < want ? blocks : want, T);
    // attributes are set on every call: a cached flag would go stale across a device reset; always to the same value, since
    // another thread may be between its own setting and its launch
    for (int h0 = 0; h0 < Hq; h0 += SC_MAX_HEADS) {
        const int nh = Hq - h0 < SC_MAX_HEADS ? Hq - h0 : SC_MAX_HEADS;
        auto kernel = h0 > 0 ? k_idx_score<true> : k_idx_score<false>;
        GS_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, score_smem(SC_MAX_HEADS)));
        GS_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        if (int e = launch_pdl(kernel, grid, SC_WARPS * 32, score_smem(nh), (cudaStream_t) stream, q + (int64_t) h0 * Dk, w + h0, P, score,
                               score_stride, pos0, kpool, nh, Dk, scale, Hq))
            return e;
    }
    return 0;
}

GS_EXPORT int gs_idx_select(const float *score, int64_t score_stride, int pos0, int T, int kpool, int top_k, int *sel,
                            int sel_stride, int *cnt, void *stream) {
    if (T <= 0) return 0;  // ops.cu:788
    if (kpool <= 0 || top_k < 0 || pos0 < 0) return fail_invalid("gs_idx_select: need kpool > 0, top_k >= 0, pos0 >= 0");
    if (!sel || !cnt) return fail_invalid("gs_idx_select: null pointer");
    const int most = (pos0 + T) / kpool;  // scores of the last query
    const bool cached = most > top_k && most <= SEL_CACHE;
    if (!cached)
        return launch_pdl(k_idx_select<false>, dim3(T), SEL_NT, 0, (cudaStream_t) stream, score, score_stride, pos0, kpool, top_k, sel, sel_stride, cnt);
    GS_TRY(cudaFuncSetAttribute(k_idx_select<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SEL_CACHE * 4));
    GS_TRY(cudaFuncSetAttribute(k_idx_select<true>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    return launch_pdl(k_idx_select<true>, dim3(T), SEL_NT, (size_t) most * 4, (cudaStream_t) stream, score, score_stride, pos0, kpool, top_k,
                      sel, sel_stride, cnt);
}
