// Two::inverse_mid (csrc/llb_model.cuh) against the division: every 32-bit
// pattern the guard Two::mid lets through, in both halves of the pair, and the
// guard itself for every pattern.  Prints the patterns let through, the
// reciprocals that differ and the patterns the guard judges wrongly.
#include <cstdio>

#include "llb_model.cuh"

using llb::Two;

__global__ void compare(unsigned long long* out) {
    unsigned long long mids = 0, differ = 0, guard = 0;
    const unsigned long long n = 1ull << 32, step = static_cast<unsigned long long>(gridDim.x) * blockDim.x;
    for (unsigned long long p = static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += step) {
        const float x = __uint_as_float(static_cast<unsigned>(p));
        const bool in = x > 0x1p-120f && x < 0x1p120f;  // false for NaN
        guard += Two::mid(Two::pack(x, 1.0f)) != in;
        guard += Two::mid(Two::pack(1.0f, x)) != in;
        if (!in) continue;
        ++mids;
        const float2 a = Two::unpack(Two::inverse_mid(Two::pack(x, 1.5f)));
        const float2 b = Two::unpack(Two::inverse_mid(Two::pack(1.5f, x)));
        const unsigned want = __float_as_uint(1.0f / x), third = __float_as_uint(1.0f / 1.5f);
        differ += __float_as_uint(a.x) != want || __float_as_uint(b.y) != want || __float_as_uint(a.y) != third ||
                  __float_as_uint(b.x) != third;
    }
    atomicAdd(out, mids);
    atomicAdd(out + 1, differ);
    atomicAdd(out + 2, guard);
}

int main() {
    unsigned long long *d = nullptr, h[3] = {0, 0, 0};
    if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return 1;
    compare<<<148 * 8, 256>>>(d);
    if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    std::printf("%llu %llu %llu\n", h[0], h[1], h[2]);
    return 0;
}
