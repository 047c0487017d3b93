// The time after which a wait of k_level_bands (rgbd-flow_b200/csrc/level_bands.cuh) gives up: its tries block, so the
// number of tries does not tell.  One block waits for a row that nobody sends, once.
#include "../../rgbd-flow_b200/csrc/level_bands.cuh"

#include <cstdio>

using namespace rgbdflow;

__global__ void k_probe(int polls, unsigned long long* ns, int* gave_up)
{
    __shared__ __align__(8) unsigned long long s_mbar;
    const unsigned mbar = (unsigned)__cvta_generic_to_shared(&s_mbar);
    if (threadIdx.x == 0) mbar_init(mbar);
    __syncthreads();
    unsigned long long a, b;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(a));
    const bool got = mbar_wait(mbar, 0, polls);
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(b));
    if (threadIdx.x == 0) {
        *ns = b - a;
        *gave_up = !got;
    }
}

int main()
{
    unsigned long long* ns = nullptr;
    int* gave_up = nullptr;
    if (cudaMallocManaged(&ns, sizeof(*ns)) != cudaSuccess || cudaMallocManaged(&gave_up, sizeof(int)) != cudaSuccess) return 1;
    // a hundredth of the tries, so that a limit that was far too long would not be waited out
    k_probe<<<1, 32>>>(kBandPolls / 100, ns, gave_up);
    if (cudaDeviceSynchronize() != cudaSuccess || !*gave_up) return 1;
    const double s = 100 * *ns * 1e-9;
    std::printf("a wait gives up after %.2f s\n", s);
    return s > 0.2 && s < 2 ? 0 : 1;
}
