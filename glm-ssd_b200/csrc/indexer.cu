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
    sm100::griddep_launch_dependents();
    const int kpool = KP > 0 ? KP : kpool_arg;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int end = p0 + T;
    const int jf = p0 / kpool, jl = end / kpool;
    const int64_t j = (int64_t) jf + blockIdx.y;
    sm100::griddep_wait();
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
            for (int m = 0; m < kpool; m++) mx = fmaxf(mx, idx_row(gc, rg, j * kpool + m, p0, Dk, kpool)[c] + ape[m * Dk + c]);
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

// ---- scores -------------------------------------------------------------------------------------------------
// Block = 64 pools x 4 column parts (thread (pool, part) owns columns part, part + 4, part + 8, ... of its pool's key
// in registers); the query's heads sit in shared memory and are read as broadcasts.  Per (pool, head): 32 FMAs per
// thread and two shuffles to join the four parts.
constexpr int SC_POOLS = 64, SC_PARTS = 4, SC_MAXI = 32;  // Dk <= SC_PARTS * SC_MAXI = 128
__global__ void __launch_bounds__(SC_POOLS *SC_PARTS) k_idx_score(const float *__restrict__ q, const float *__restrict__ w,
                                                                  const float *__restrict__ P, float *__restrict__ score,
                                                                  int64_t score_stride, int pos0, int kpool, int Hq, int Dk, float scale) {
    const int t = blockIdx.y;
    const int n_pool = (pos0 + t + 1) / kpool;
    const int p_base = blockIdx.x * SC_POOLS;
    if (p_base >= n_pool) return;
    extern __shared__ float sq[];  // [Hq][Dk] then w [Hq]
    float *sw = sq + Hq * Dk;
    const float *qt = q + (int64_t) t * Hq * Dk;
    for (int i = threadIdx.x; i < Hq * Dk; i += blockDim.x) sq[i] = qt[i];
    for (int i = threadIdx.x; i < Hq; i += blockDim.x) sw[i] = w[(int64_t) t * Hq + i];
    __syncthreads();
    const int part = threadIdx.x & (SC_PARTS - 1);
    const int p = p_base + (threadIdx.x >> 2);
    const int pc = min(p, n_pool - 1);  // lanes past the end work on a valid row and drop the result
    float kreg[SC_MAXI];
    const float *pk = P + (int64_t) pc * Dk;
#pragma unroll
    for (int i = 0; i < SC_MAXI; i++) kreg[i] = (i * SC_PARTS + part) < Dk ? pk[i * SC_PARTS + part] : 0.f;
    float total = 0.f;
    for (int h = 0; h < Hq; h++) {
        const float *qh = sq + h * Dk;
        float d = 0.f;
#pragma unroll
        for (int i = 0; i < SC_MAXI; i++)
            if (i * SC_PARTS < Dk) d = fmaf((i * SC_PARTS + part) < Dk ? qh[i * SC_PARTS + part] : 0.f, kreg[i], d);
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        total = fmaf(sw[h], fmaxf(d * scale, 0.f), total);
    }
    if (part == 0 && p < n_pool) score[(int64_t) t * score_stride + p] = total;
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
// consecutive pools each, one scan over the counts, and a thread per ballot writes the pools it holds - the pools appear in
// ascending index and ties go to the lowest indices.
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
struct SelSmem {
    union {
        alignas(16) uint32_t hist[SEL_BINS];
        uint2 flags[SEL_SLAB];            // ordered pass: ballots of "greater" and "equal"
    };
    alignas(16) uint32_t list[SEL_LIST];
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
    sm100::griddep_launch_dependents();
    sm100::griddep_wait();
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
            for (uint32_t m = f.x | f.y; m; m &= m - 1) {
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

// The kernels of the indexer follow one another in a stream (pool, score, select, then the attention): each may be
// scheduled while the one in front still runs and waits for its results inside.
template <typename... KArgs, typename... Args>
int launch_pdl(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GS_TRY(cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...));
    return 0;
}

}  // namespace

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
    dim3 grid((max_pool + SC_POOLS - 1) / SC_POOLS, T);
    k_idx_score<<<grid, SC_POOLS * SC_PARTS, (size_t) Hq * (Dk + 1) * sizeof(float), (cudaStream_t) stream>>>(
        q, w, P, score, score_stride, pos0, kpool, Hq, Dk, scale);
    GS_TRY(cudaGetLastError());
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
