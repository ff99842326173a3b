// Device check of the parts of sgl::normalize_fast
// (swegl_gb300/csrc/sgl_device.cuh) against square root, reciprocal and
// division:
//  - root_and_reciprocal's l for every float s from 2^-100 to 2^100, and its y
//    for the same s; an s whose y is not the rounded reciprocal is kept;
//  - quotient for each kept s with every numerator of l's octave and the one
//    below (a component is at most the length);
//  - quotient for every significand of l, with y the rounded reciprocal, by
//    `per` numerators: seeded ones, or all 2^23 of them when per is 2^23 (51 s,
//    in launches of 2^15 significands).
// Usage: normalize_roots_gpu PER.  Prints "<roots that differ> <reciprocals
// kept> <quotients of those that differ> <pairs> <quotients that differ>".
#include <cstdio>
#include <cstdlib>

#include "sgl_device.cuh"

using namespace sgl;

constexpr uint32_t kLo = (127u - 100u) << 23, kHi = (127u + 100u) << 23;
constexpr int kMaxKept = 1 << 16;
__device__ unsigned long long g_roots, g_kept, g_kept_bad, g_bad;
__device__ float g_list[kMaxKept];

__global__ void roots()
{
    for (uint32_t u = kLo + blockIdx.x * blockDim.x + threadIdx.x; u <= kHi; u += gridDim.x * blockDim.x) {
        const float s = __uint_as_float(u);
        float l, y;
        root_and_reciprocal(s, l, y);
        if (l != __fsqrt_rn(s))
            atomicAdd(&g_roots, 1ull);
        if (y != __frcp_rn(l)) {
            const unsigned long long k = atomicAdd(&g_kept, 1ull);
            if (k < kMaxKept)
                g_list[k] = s;
        }
    }
}

__global__ void kept_quotients(int n)
{
    for (int k = blockIdx.x; k < n; k += gridDim.x) {
        float l, y;
        root_and_reciprocal(g_list[k], l, y);
        const uint32_t top = __float_as_uint(l) & 0xFF800000u;
        unsigned bad = 0;
        for (uint32_t m = threadIdx.x; m < 1u << 24; m += blockDim.x) {
            const float x = __uint_as_float(top - (1u << 23) + m);
            bad += quotient(x, l, y) != __fdiv_rn(x, l);
        }
        if (bad)
            atomicAdd(&g_kept_bad, (unsigned long long)bad);
    }
}

__global__ void quotients(uint32_t first, uint32_t per)
{
    const uint32_t m = first + blockIdx.x;
    const float l = __uint_as_float(0x3F800000u | m), y = __frcp_rn(l);
    unsigned bad = 0;
    for (uint32_t k = threadIdx.x; k < per; k += blockDim.x) {
        const uint32_t n = per == 1u << 23 ? k : ((m * 0x9E3779B9u + k) * 0x85EBCA6Bu) >> 9;
        const float x = __uint_as_float(0x3F800000u | n);
        bad += quotient(x, l, y) != __fdiv_rn(x, l);
    }
    if (bad)
        atomicAdd(&g_bad, (unsigned long long)bad);
}

int main(int argc, char **argv)
{
    const uint32_t per = argc > 1 ? (uint32_t)strtoul(argv[1], nullptr, 10) : 1024u;
    roots<<<1216, 256>>>();
    unsigned long long wrong = 0, kept = 0, kept_bad = 0, bad = 0;
    if (cudaMemcpyFromSymbol(&wrong, g_roots, sizeof wrong) != cudaSuccess ||
        cudaMemcpyFromSymbol(&kept, g_kept, sizeof kept) != cudaSuccess || kept > kMaxKept)
        return 1;
    kept_quotients<<<1216, 256>>>((int)kept);
    const uint32_t step = 1u << 15;
    for (uint32_t m = 0; m < 1u << 23; m += step) {
        quotients<<<step, 256>>>(m, per);
        if (cudaDeviceSynchronize() != cudaSuccess)
            return 1;
    }
    if (cudaMemcpyFromSymbol(&kept_bad, g_kept_bad, sizeof kept_bad) != cudaSuccess ||
        cudaMemcpyFromSymbol(&bad, g_bad, sizeof bad) != cudaSuccess)
        return 1;
    printf("%llu %llu %llu %llu %llu\n", wrong, kept, kept_bad, (unsigned long long)per << 23, bad);
    return 0;
}
