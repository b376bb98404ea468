// Compares the pair terms' square root and exponential with CUDA's functions
// over every FP32 value of the ranges their comments name.  Prints, per
// function, the number of values and of differences.
#include "../../sca2012_b200/csrc/sph_kernels.cuh"
#include <cstdio>
#include <cstring>

__global__ void compare(uint32_t first, uint32_t count, int which, unsigned long long *diff)
{
    unsigned long long bad = 0;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < count; k += (uint64_t)gridDim.x * blockDim.x) {
        const float x = __uint_as_float(first + (uint32_t)k);
        float got, want;
        if (which == 0) {
            got = sph::sqrt_of(x, sph::rsqrt_normal(x));
            want = __fsqrt_rn(x);
        } else {
            got = sph::ex2_normal(-x);
            want = exp2f(-x);
        }
        bad += __float_as_uint(got) != __float_as_uint(want);
    }
    if (bad) atomicAdd(diff, bad);
}

static uint32_t bits(float x)
{
    uint32_t u;
    memcpy(&u, &x, 4);
    return u;
}

int main()
{
    unsigned long long *diff;
    if (cudaMalloc(&diff, sizeof(*diff)) != cudaSuccess) return 1;
    const float lo[2] = {2.7e-20f, 0.0f}, hi[2] = {4e37f, 126.0f};   // 2^-x down to 2^-126
    for (int which = 0; which < 2; ++which) {
        const uint32_t first = bits(lo[which]), count = bits(hi[which]) - first + 1u;
        unsigned long long n = 0;
        cudaMemset(diff, 0, sizeof(*diff));
        compare<<<148 * 8, 256>>>(first, count, which, diff);
        if (cudaMemcpy(&n, diff, sizeof(n), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
        printf("%s %u %llu\n", which == 0 ? "sqrt" : "exp2", count, n);
    }
    cudaFree(diff);
    return 0;
}
