// A wait of k_level_bands (rgbd-flow_b200/csrc/level_bands.cuh) that runs out in a thread other than the block's
// first: no row arrives at the block's barrier, the wait ends after its tries, and the status word says so.
#include "../../rgbd-flow_b200/csrc/level_bands.cuh"

#include <cstdio>

using namespace rgbdflow;

__global__ void k_probe(int waiter, int polls, int* status, int* gave_up)
{
    __shared__ __align__(8) unsigned long long s_mbar;
    const unsigned mbar = (unsigned)__cvta_generic_to_shared(&s_mbar);
    if (threadIdx.x == 0) mbar_init(mbar);
    __syncthreads();
    bool lost = false;
    if ((int)threadIdx.x == waiter) {
        mbar_expect(mbar, 12);  // nobody sends
        lost = !mbar_wait(mbar, 0, polls);
        *gave_up = lost;
    }
    report_lost(lost, status);
}

int main()
{
    int* d = nullptr;
    if (cudaMalloc(&d, 2 * sizeof(int)) != cudaSuccess) return 1;
    for (int waiter : {0, 31, 40, 95}) {
        cudaMemset(d, 0, 2 * sizeof(int));
        k_probe<<<1, 96>>>(waiter, 1000, d, d + 1);
        int h[2] = {};
        if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
        if (h[0] != 1 || h[1] != 1) {
            std::printf("thread %d: gave up %d, status %d\n", waiter, h[1], h[0]);
            return 1;
        }
    }
    cudaMemset(d, 0, 2 * sizeof(int));
    k_probe<<<1, 96>>>(-1, 1000, d, d + 1);  // nobody waits: nothing to report
    int h[2] = {};
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess || h[0] || h[1]) return 1;
    std::printf("ok lost waits\n");
    return 0;
}
