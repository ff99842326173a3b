// Device check of sgl::normalize_fast (swegl_gb300/csrc/sgl_device.cuh), which
// normalises with one reciprocal square root, against sgl::normalize3 (square
// root, then three divisions): equal bits on `n` seeded vectors of ordinary,
// tiny, huge, zero, subnormal, infinite and NaN components, and lengths at the
// end of an octave.  Prints
// "<vectors> <differing>".
#include <cstdio>
#include <cstdlib>

#include "sgl_device.cuh"

using namespace sgl;

__device__ unsigned long long g_bad;

__device__ uint32_t mix(uint64_t x)
{
    x = (x + 0x9E3779B97F4A7C15ull) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return (uint32_t)(x >> 32);
}

// component k of vector i: any bits, bits near one, near a unit vector's, a zero, or an exponent at the guard's ends
__device__ float component(uint64_t i, int k)
{
    const uint32_t r = mix(4 * i + k), how = mix(i ^ 0x5555) % 8;
    if (how == 0)
        return __uint_as_float(r);
    if (how == 1 && r % 3 == 0)
        return r & 4 ? 0.0f : -0.0f;
    const uint32_t span = how < 5 ? 4 : 70, e = 127 + (int)(r >> 8) % (int)(2 * span) - (int)span;
    return __uint_as_float((r & 0x807FFFFFu) | (e << 23));
}

__global__ void check(uint64_t n)
{
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        V3 v = mk3(component(i, 0), component(i, 1), component(i, 2));
        if (mix(i ^ 0x5555) % 8 == 2) { // a power of two, and a length at or just below the next: all ones
            v.x = __uint_as_float((117u + mix(i) % 20u) << 23);
            v.z = v.x * (0.5f + (float)(mix(i ^ 0x77) >> 9) * 0x1p-24f);
            v.y = sqrtf(4.0f * v.x * v.x - v.x * v.x - v.z * v.z);
        }
        const V3 a = normalize_fast(v), z = normalize_fast<true>(v), b = normalize3(v);
        auto same = [](float x, float y) { return __float_as_uint(x) == __float_as_uint(y) || (x != x && y != y); };
        if (!same(a.x, b.x) || !same(a.y, b.y) || !same(a.z, b.z) || !same(z.x, b.x) || !same(z.y, b.y) || !same(z.z, b.z))
            atomicAdd(&g_bad, 1ull);
    }
}

int main(int argc, char **argv)
{
    const uint64_t n = argc > 1 ? strtoull(argv[1], nullptr, 10) : 1000000;
    check<<<1216, 256>>>(n);
    unsigned long long bad = ~0ull;
    if (cudaMemcpyFromSymbol(&bad, g_bad, sizeof bad) != cudaSuccess)
        return 1;
    printf("%llu %llu\n", (unsigned long long)n, bad);
    return 0;
}
