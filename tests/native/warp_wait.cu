/* A warp's bounded wait (warp_all of mbar_wait, cb_tma.cuh) whose lanes have different
 * limits: half of them give up long before the barrier's phase completes, the
 * others would see it complete. Compiled and run by test_warp_wait_gpu.py. */
#include "cb_tma.cuh"

namespace cb {

constexpr long long SOON = 0, COMPLETES = 4000000, LATE = 400000000;   /* cycles */

static __global__ void k_warp_wait(int *out) {
    __shared__ uint64_t bar;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x >= 32) {
        /* the second warp completes the phase after COMPLETES cycles */
        const long long t0 = clock64();
        while (clock64() - t0 < COMPLETES) __nanosleep(1000);
        if (lane == 0) mbar_arrive(&bar);
    } else {
        out[lane] = warp_all(mbar_wait(&bar, 0, lane < 16 ? SOON : LATE)) ? 1 : 0;
    }
    __syncthreads();
    if (threadIdx.x < 32) out[32 + lane] = warp_all(mbar_wait(&bar, 0, LATE)) ? 1 : 0;
}

}  // namespace cb

extern "C" int run_warp_wait(int *host) {
    int *dev = nullptr;
    cudaError_t e = cudaMalloc(&dev, 64 * sizeof(int));
    if (e == cudaSuccess) {
        cb::k_warp_wait<<<1, 64>>>(dev);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(host, dev, 64 * sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(dev);
    return (int)e;
}
