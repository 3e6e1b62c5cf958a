// debug_approx.cu -- the short root, quotient and reciprocal of approx.cuh
// against the IEEE operations.
#include <cuda_runtime.h>

#include "approx.cuh"
#include "engine.h"

namespace ldsc {

namespace {

// splitmix64's finaliser: arguments spread over all mantissas and exponents
__device__ __forceinline__ uint64_t mix(uint64_t z) {
    z = (z + 0x9E3779B97F4A7C15ull) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ uint64_t places(int64_t a, int64_t b) { return (uint64_t)(a > b ? a - b : b - a); }

__global__ void __launch_bounds__(256) k_debug_approx(int which, uint64_t first, uint64_t count,
                                                      unsigned long long* __restrict__ out) {
    unsigned long long differ = 0, most = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t x = first + i;
        uint64_t d;
        if (which == 0) {
            const float v = __uint_as_float((uint32_t)x);
            d = places(__float_as_int(sqrt_nr(v)), __float_as_int(__fsqrt_rn(v)));
        } else if (which == 1) {
            const uint64_t h = mix(x), g = mix(h);
            const float a = __uint_as_float((uint32_t)(h >> 63) << 31 | (107u + (uint32_t)(h >> 32) % 60u) << 23 |
                                            (uint32_t)(h & 0x7FFFFFu));
            const float b = __uint_as_float((129u + (uint32_t)(g >> 32) % 28u) << 23 | (uint32_t)(g & 0x7FFFFFu));
            d = places(__float_as_int(div_nr(a, b)), __float_as_int(__fdiv_rn(a, b)));
        } else {
            const uint64_t h = mix(x), g = mix(h);
            const double v = __longlong_as_double((long long)((2 + g % 2042) << 52 | (h & 0xFFFFFFFFFFFFFull)));
            d = recip_plain(v) ? places(__double_as_longlong(recip_halley(v)), __double_as_longlong(__drcp_rn(v))) : ~0ull;
        }
        differ += d != 0;
        most = d > most ? d : most;
    }
    if (differ) atomicAdd(out, differ);
    if (most) atomicMax(out + 1, most);
}

}  // namespace

cudaError_t launch_debug_approx(int which, uint64_t first, uint64_t count, unsigned long long* out, cudaStream_t stream) {
    if (count == 0) return cudaSuccess;
    k_debug_approx<<<148 * 8, 256, 0, stream>>>(which, first, count, out);
    return cudaGetLastError();
}

}  // namespace ldsc
