// Check of sgl::light_sum's skip of specular powers that cannot change the sum
// (swegl_gb300/csrc/sgl_shade.cuh) against a restatement of the reference's
// loop (src/render/pixel_shaders.cpp:159-205) that always takes the power: the
// two agree bit for bit.  One light per case, and the camera placed where the
// specular base s has p log2(s) within a few powers of two of the threshold.
// Exponents: 0..1024 (what a scene's materials may hold), and a default
// material's, which is not bounded: larger ones and negative ones.
// `light_skip host N` runs here, `light_skip device N` on the GPU, whose
// logarithm is the approximate one.  Prints "<cases> <differing> <cases below
// the threshold with an exponent of 1..1024> <... with another>".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "sgl_device.cuh"
#include "sgl_internal.h"
#include "sgl_shade.cuh"

using namespace sgl;

struct Counts {
    unsigned long long diff, inside, beyond;
};

__host__ __device__ static uint32_t mix(uint64_t x)
{
    x = (x + 0x9E3779B97F4A7C15ull) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return (uint32_t)(x >> 32);
}
struct Draws {
    uint64_t i;
    uint32_t k;
    __host__ __device__ uint32_t bits() { return mix(64 * i + k++); }
    __host__ __device__ float sym() { return (float)(int32_t)bits() * 0x1p-31f; } // -1..1
    __host__ __device__ V3 unit()
    {
        const V3 v = mk3(sym(), sym(), sym());
        return v.x * v.x + v.y * v.y + v.z * v.z < 1e-4f ? mk3(0.0f, 0.0f, 1.0f) : normalize3(v);
    }
};

// What the reference adds for one light in front of the surface: `specular`,
// its base, and `weight`, the diffuse term times the squared distance.
__host__ __device__ static float plain_light(const LightsDev &L, V3 center, V3 normal, V3 camvec, int shininess,
                                             float &base, float &weight)
{
    base = weight = 0.0f;
    float face_sun = -dot3(normal, mk3(L.sun[0], L.sun[1], L.sun[2]));
    face_sun = face_sun < 0.0f ? 0.0f : face_sun * L.sun_intensity;
    float dyn = 0.0f;
    V3 ld = sub3(center, mk3(L.pl[0].x, L.pl[0].y, L.pl[0].z));
    const float d2 = ld.x * ld.x + ld.y * ld.y + ld.z * ld.z;
    float diffuse = L.pl[0].w / d2;
    ld = normalize3(ld);
    const float alignment = -dot3(normal, ld);
    if (!(diffuse < 0.05f) && !(alignment < 0.0f)) {
        diffuse = diffuse * alignment;
        const V3 reflection = add3(ld, mul3(normal, alignment * 2.0f));
        float specular = dot3(reflection, camvec);
        if (specular > 0.0f) {
            base = specular;
            weight = diffuse * d2;
            specular = spec_pow(specular, shininess);
            specular = specular * (float)shininess / 2.0f;
            dyn = dyn + (diffuse + specular / d2);
        } else {
            dyn = dyn + diffuse;
        }
    }
    return L.ambient + face_sun + dyn;
}

__host__ __device__ static void check(uint64_t i, Counts &n)
{
    Draws d{i, 0u};
    LightsDev L{};
    L.ambient = 0.0f; // (the sum's last bits are the light's)
    L.sun[2] = 1.0f;
    L.n = 1;
    const V3 center = mul3(d.unit(), 20.0f), normal = d.unit();
    V3 to = d.unit(); // towards the light, in front of the surface
    if (dot3(to, normal) < 0.0f)
        to = neg3(to);
    to = mul3(to, 0.25f + 8.0f * fabsf(d.sym()));
    const V3 light = add3(center, to);
    L.pl[0] = make_float4(light.x, light.y, light.z, 50.0f);
    const uint32_t r = d.bits();
    int p;
    switch (i % 8) {
    case 0: p = (int)(r % 1025u); break;
    case 1: p = 1024 - (int)(r % 4u); break;
    case 2: p = 1 + (int)(r % 128u); break;
    case 3: p = 1025 + (int)(r % 4096u); break;
    case 4: p = (int)(r >> (1 + (r & 15u))); break; // up to 2^31 - 1
    case 5: p = 100000; break;
    case 6: p = -(int)(r >> (1 + (r & 31u) % 31u)); break;
    default: p = 1 + (int)(r % 1024u); break;
    }
    // the reflected direction, and a camera direction whose dot product with
    // it is s, for a power p log2(s) around log2(weight) - 36
    const V3 ld = normalize3(sub3(center, light));
    const float a = -dot3(normal, ld);
    const V3 refl = normalize3(add3(ld, mul3(normal, a * 2.0f)));
    const float want = log2f(50.0f * fmaxf(a, 1e-6f)) - 36.0f + 24.0f * d.sym();
    float s = exp2f(want / (float)(p > 0 ? p : 1));
    s = s < 1.0f ? s : 1.0f;
    V3 t = d.unit();
    t = normalize3(sub3(t, mul3(refl, dot3(t, refl))));
    const V3 camvec = add3(mul3(refl, s), mul3(t, sqrtf(fmaxf(0.0f, 1.0f - s * s))));
    float base, weight;
    const float plain = plain_light(L, center, normal, camvec, p, base, weight);
    const float got = light_sum(L, center, normal, camvec, p);
    if (!(got == plain || (got != got && plain != plain)))
        n.diff++;
    if (base > 0.0f && (float)p * log2_approx(base) < log2_approx(weight) - 36.0f) {
        if (p >= 1 && p <= 1024)
            n.inside++;
        else
            n.beyond++;
    }
}

__device__ Counts g_counts;
__global__ void k_check(uint64_t n)
{
    Counts c{};
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        check(i, c);
    atomicAdd(&g_counts.diff, c.diff);
    atomicAdd(&g_counts.inside, c.inside);
    atomicAdd(&g_counts.beyond, c.beyond);
}

int main(int argc, char **argv)
{
    const uint64_t n = argc > 2 ? strtoull(argv[2], nullptr, 10) : 1000000;
    Counts c{};
    if (argc > 1 && !strcmp(argv[1], "device")) {
        k_check<<<1216, 256>>>(n);
        if (cudaMemcpyFromSymbol(&c, g_counts, sizeof c) != cudaSuccess)
            return 1;
    } else {
        for (uint64_t i = 0; i < n; i++)
            check(i, c);
    }
    printf("%llu %llu %llu %llu\n", (unsigned long long)n, c.diff, c.inside, c.beyond);
    return 0;
}
