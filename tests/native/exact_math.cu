// exact_math.cu - the roots, reciprocals and quotients of device.cuh against CUDA's correctly
// rounded operators, on the GPU: counts of differing results. Test infrastructure only.
#include <cstdio>
#include <cstdint>
#include <cuda_runtime.h>
#include "device.cuh"
using namespace vxr::dev;

__device__ __forceinline__ void note(unsigned long long* bad, bool differs) {
    if (differs) atomicAdd(bad, 1ull);
}
// every mantissa of every binade of [2^-100, 2^100): sqrtf(x), 1 / x
__global__ void one_operand(unsigned long long* bad) {
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;   // 2^23 threads
    for (int e = 127 - 100; e < 127 + 100; e++) {
        const float x = __uint_as_float(((uint32_t)e << 23) | m);
        note(bad + 0, __float_as_uint(sqrt_rn(x)) != __float_as_uint(__fsqrt_rn(x)));
        note(bad + 1, __float_as_uint(rcp_rn(x)) != __float_as_uint(__fdiv_rn(1.0f, x)));
    }
}
// quotients: the 64 largest and smallest mantissas of b with every mantissa of a, and random
// pairs, quotient and reciprocal together
__global__ void quotients(unsigned long long* bad, uint32_t seed, int random) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;   // 2^23 threads
    uint32_t r = wang_hash(t ^ wang_hash(seed));
    for (int i = 0; i < 128; i++) {
        uint32_t mb = i < 64 ? 0x7FFFFFu - (uint32_t)i : (uint32_t)(i - 64), ma = t;
        int ea = 127, eb = 127;
        if (random) {
            mb = xs32(r) & 0x7FFFFFu;
            ma = xs32(r) & 0x7FFFFFu;
            ea = 127 - 50 + (int)(xs32(r) % 100u);
            eb = 127 - 30 + (int)(xs32(r) % 60u);
        }
        const float a = __uint_as_float(((uint32_t)ea << 23) | ma), b = __uint_as_float(((uint32_t)eb << 23) | mb);
        const uint32_t want = __float_as_uint(__fdiv_rn(a, b));
        note(bad + 2, __float_as_uint(quotient_rn(a, b, rcp_rn(b))) != want);
        note(bad + 3, __float_as_uint(quotient_rn(0.0f, b, rcp_rn(b))) != 0u);
    }
}

int main() {
    unsigned long long* bad;
    unsigned long long h[4];
    if (cudaMalloc(&bad, sizeof(h)) != cudaSuccess) return 2;
    cudaMemset(bad, 0, sizeof(h));
    one_operand<<<(1 << 23) / 256, 256>>>(bad);
    quotients<<<(1 << 23) / 256, 256>>>(bad, 1, 0);
    for (uint32_t s = 0; s < 8; s++) quotients<<<(1 << 23) / 256, 256>>>(bad, 100 + s, 1);
    if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    for (unsigned long long v : h) printf("%llu ", v);
    printf("\n");
    return 0;
}
