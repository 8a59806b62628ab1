// Compares mfcfd_ieee.cuh with the operators on the GPU.  FP64: random
// arguments over the range ieee_ok admits, and arguments next to rounding
// boundaries (quotients and roots whose exact value lies close to a midpoint
// of two doubles, significands next to a power of two).  FP32: every
// significand for the reciprocal and (both parities of the exponent) the root,
// random pairs for the quotient.  Prints the number of arguments and of
// results whose bits differ.
#include <cstdio>
#include <cstdint>
#include <cstdlib>

#include <cuda_runtime.h>

#include "../3d-mfcfd_b200/csrc/mfcfd_ieee.cuh"

using namespace mfcfd;

__device__ uint64_t mix(uint64_t x) {
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

// a significand: random, or a few units from 1, from 2 or from a short one
__device__ uint64_t significand(uint64_t r) {
    const uint64_t m = r >> 12, one = (1ull << 52) - 1;
    switch (r & 7) {
    case 0: return m & 0xff;
    case 1: return (one - (m & 0xff)) & one;
    case 2: return (m & (one << 26)) & one;
    case 3: return (r >> 3 & 1) ? one : ((m & (one << 26)) + (m & 7)) & one;
    default: return m;
    }
}

__device__ double number(uint64_t r, int range) {
    const int e = 1023 - range + (int)(mix(r ^ 77) % (uint64_t)(2 * range));
    return __longlong_as_double((long long)(((uint64_t)e << 52) | significand(r)));
}

__global__ void check(uint64_t seed, int rounds, unsigned long long *bad) {
    const uint64_t id = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    unsigned long long wrong[3] = {0, 0, 0}, seen = 0;
    for (int k = 0; k < rounds; ++k) {
        const uint64_t r = mix(seed + id * 1000003ull + (uint64_t)k);
        const double b = number(r, 300);
        double a = number(mix(r), 390);
        // every other numerator puts the quotient next to a midpoint
        if (k & 1) {
            const double q = number(mix(r ^ 5), 60);
            const double ulp = __longlong_as_double(__double_as_longlong(q) + 1) - q;
            a = __fma_rn(q, b, 0.5 * ulp * b);
            if ((k & 6) == 2) a = __longlong_as_double(__double_as_longlong(a) ^ 1);
        }
        if ((r >> 40 & 1)) a = -a;
        if (!ieee_ok(b)) continue;
        ++seen;
        const double y = rcp_rn(b);
        if (__double_as_longlong(y) != __double_as_longlong(1.0 / b)) ++wrong[0];
        if (ieee_num_ok(a) && __double_as_longlong(quot_rn(a, b, y)) != __double_as_longlong(a / b)) ++wrong[1];
        const double zero = (r >> 41 & 1) ? 0.0 : -0.0;
        if (__double_as_longlong(quot_rn(zero, b, y)) != __double_as_longlong(zero / b)) ++wrong[1];
        // roots: random, and squares of midpoints
        double x = b;
        if (k & 1) {
            const double g = number(mix(r ^ 9), 140);
            const double ulp = __longlong_as_double(__double_as_longlong(g) + 1) - g;
            x = __fma_rn(g, g, g * ulp);
            x = __longlong_as_double(__double_as_longlong(x) + (int)(r >> 50 & 3) - 1);
        }
        if (ieee_ok(x) && __double_as_longlong(sqrt_rn(x)) != __double_as_longlong(sqrt(x))) ++wrong[2];
    }
    for (int w = 0; w < 3; ++w)
        if (wrong[w]) atomicAdd(bad + w, wrong[w]);
    atomicAdd(bad + 3, seen);
}

__global__ void check_f32(uint64_t seed, int rounds, unsigned long long *bad) {
    const uint64_t id = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, all = gridDim.x * (uint64_t)blockDim.x;
    unsigned long long wrong[3] = {0, 0, 0}, seen = 0;
    auto differ = [](float a, float b) { return __float_as_int(a) != __float_as_int(b); };
    for (uint64_t m = id; m < (1ull << 24); m += all) {
        // all significands in two neighbouring binades, at a random exponent
        const int e = 68 + 2 * (int)(mix(seed ^ m) % 59);
        const float b = __int_as_float((int)((uint32_t)(e << 23) + (uint32_t)m));
        if (!ieee_ok(b)) continue;
        ++seen;
        const float y = rcp_rn(b);
        if (differ(y, 1.0f / b)) ++wrong[0];
        if (differ(sqrt_rn(b), sqrtf(b))) ++wrong[2];
        for (int k = 0; k < rounds; ++k) {
            const uint64_t r = mix(seed + 64 * m + (uint64_t)k);
            float a = __int_as_float((int)(((uint32_t)(67 + r % 119) << 23) | (uint32_t)(r >> 40 & 0x7fffff)));
            if (k & 1) {                  // next to a midpoint
                const float q = __int_as_float((int)((127u << 23) | (uint32_t)(r >> 40 & 0x7fffff)));
                a = __fmaf_rn(q, b, 0x1p-24f * b);
                if (!ieee_ok(a)) continue;
            }
            if (differ(quot_nz(a, b, y), a / b)) ++wrong[1];
        }
    }
    for (int w = 0; w < 3; ++w)
        if (wrong[w]) atomicAdd(bad + w, wrong[w]);
    atomicAdd(bad + 3, seen);
}

int main(int argc, char **argv) {
    const int rounds = argc > 1 ? std::atoi(argv[1]) : 256;
    unsigned long long *bad = nullptr, h[4] = {0, 0, 0, 0};
    if (cudaMalloc(&bad, sizeof h) != cudaSuccess || cudaMemset(bad, 0, sizeof h) != cudaSuccess) return 2;
    check<<<148 * 8, 256>>>(20240607ull, rounds, bad);
    if (cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("arguments %llu wrong: reciprocal %llu quotient %llu root %llu\n", h[3], h[0], h[1], h[2]);
    unsigned long long f[4] = {0, 0, 0, 0};
    if (cudaMemset(bad, 0, sizeof h) != cudaSuccess) return 2;
    check_f32<<<148 * 8, 256>>>(20240608ull, 16, bad);
    if (cudaMemcpy(f, bad, sizeof f, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("FP32 arguments %llu wrong: reciprocal %llu quotient %llu root %llu\n", f[3], f[0], f[1], f[2]);
    cudaFree(bad);
    if (f[0] || f[1] || f[2] || !f[3]) return 1;
    return h[0] || h[1] || h[2] || !h[3] ? 1 : 0;
}
