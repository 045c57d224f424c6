// Test of the bounded wait: the lanes of a warp wait on different barriers, one of which nothing completes.  The wait runs
// out after its limit (about a second) and has to give one answer to the whole warp.
#include <stdint.h>

#include "../glm-ssd_b200/csrc/sm100_prims.cuh"

using namespace gs::sm100;

__global__ void k_wait_check(int32_t *status, int32_t *out) {
    __shared__ __align__(8) uint64_t done, never;
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
        mbar_init(&done, 1);
        mbar_init(&never, 1);
        fence_barrier_init();
        abort_flag = 0;
        mbar_arrive(&done);
    }
    __syncthreads();
    // warp 0: half of the lanes on the barrier that never completes; warp 1: all lanes on the completed one
    out[tid] = mbar_wait(warp == 0 && (tid & 1) ? &never : &done, 0, &abort_flag, status, 32);
    __syncthreads();
    // the vote of a group: every thread gets the same answer, whoever saw the flag
    out[64 + tid] = group_any(1, 64, tid == 5 && *(volatile int *) &abort_flag != 0);
}

extern "C" __attribute__((visibility("default"))) int wait_check(int32_t *status, int32_t *out, void *stream) {
    k_wait_check<<<1, 64, 0, (cudaStream_t) stream>>>(status, out);
    return (int) cudaGetLastError();
}
