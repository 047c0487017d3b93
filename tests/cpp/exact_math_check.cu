// exact_math.cuh against the FP32 operators on a GPU: every mantissa with exponents of both parities, at and beyond
// both ends of the range, infinities and NaN.  Prints the number of results that differ in a bit.
#include <cstdio>

#include "../../rgbd-flow_b200/csrc/exact_math.cuh"

using namespace rgbdflow;

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }
__global__ void k_mantissas(unsigned long long* bad)
{
    const int exps[] = {1, 30, 64, 65, 66, 100, 126, 127, 128, 141, 189, 190, 254, 255};
    unsigned long long n = 0;
    for (unsigned m = blockIdx.x * blockDim.x + threadIdx.x; m < 1u << 23; m += gridDim.x * blockDim.x)
        for (int e : exps) {
            const float x = __uint_as_float((unsigned)e << 23 | m);
            for (int neg = 0; neg < 2; neg++) {
                const float v = neg ? -x : x;
                if (e > 4) n += !same(div_small<12>(v), v / 12.0f) + !same(div_small<5>(v), v / 5.0f);
                float r[2] = {v, 1.0f}, s[2] = {v, 1.0f};
                inv_sqrt<float, 2>(r, r);
                inverse<float, 2>(s);
                n += !same(r[0], 1.0f / sqrtf(v)) + !same(s[0], 1.0f / v) + !same(r[1], 1.0f) + !same(s[1], 1.0f);
            }
        }
    if (n) atomicAdd(bad, n);
}

int main()
{
    unsigned long long* bad = nullptr;
    if (cudaMallocManaged(&bad, sizeof(*bad)) != cudaSuccess) return 2;
    *bad = 0;
    k_mantissas<<<1024, 256>>>(bad);
    const cudaError_t e = cudaDeviceSynchronize();
    std::printf("%s different %llu\n", cudaGetErrorString(e), *bad);
    return e == cudaSuccess && *bad == 0 ? 0 : 1;
}
