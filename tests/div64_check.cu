// Checks mk_div64 (mcsart_b200/csrc/common.cuh) and the FP64 projector's overlap
// weights (split_weight, projector.cuh) bit for bit against the compiler's
// division.  Operands: footprints of 2^-20 to 2^6 voxels at coordinates up to
// 2^16, and significands at random with exponents -40 .. 40.  Prints two counts.
#include <cstdio>

#include "projector.cuh"

using namespace mcsart;

__device__ __forceinline__ unsigned long long next(unsigned long long &h) {
    h ^= h << 13; h ^= h >> 7; h ^= h << 17;
    return h;
}
__device__ __forceinline__ double unit(unsigned long long &h) { return (next(h) >> 11) * 0x1p-53; }
__device__ __forceinline__ bool same(double a, double b) {
    return __double_as_longlong(a) == __double_as_longlong(b);
}

__global__ void check(unsigned long long *bad, int n) {
    unsigned long long h = (blockIdx.x * 1024ull + threadIdx.x + 1) * 0x9E3779B97F4A7C15ull;
    for (int i = 0; i < n; i++) {
        const double b = __hiloint2double((int)(next(h) & 0xfffff) | (1023 - 40 + (int)(next(h) % 81)) << 20,
                                          (int)next(h));
        const double a = __hiloint2double((int)(next(h) & 0xfffff) | (1023 - 40 + (int)(next(h) % 81)) << 20,
                                          (int)next(h)) * (next(h) & 1 ? 1.0 : -1.0);
        if (!same(mk_div64(a, b, 1.0 / b), a / b)) atomicAdd(&bad[0], 1ull);
        const double lo = (unit(h) - 0.25) * exp2(unit(h) * 16.0), hi = lo + exp2(unit(h) * 26.0 - 20.0);
        const double z = floor(lo) + (double)(next(h) % 3);
        if (z > hi) continue;
        const double width = hi - lo;
        if (!same(split_weight(z, lo, hi, 1.0 / width), overlap(z, lo, hi) / width))
            atomicAdd(&bad[1], 1ull);
    }
}

int main() {
    unsigned long long *bad, out[2];
    if (cudaMalloc(&bad, sizeof(out)) != cudaSuccess) return 1;
    cudaMemset(bad, 0, sizeof(out));
    check<<<4096, 256>>>(bad, 1000);
    if (cudaMemcpy(out, bad, sizeof(out), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    printf("%llu %llu\n", out[0], out[1]);
    return 0;
}
