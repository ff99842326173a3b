// Host check of the posed primitives' boxes (sgl_cull.h, pose_box): seeded
// vertex sets, their box from cull_box, and node matrices (rotations, scales
// from 1e-4 to 1e4, mirrors, shears, translations up to 1e6, single zero rows);
// every vertex transformed as the pose pass does (transform3) lies in the box
// made from the untransformed one.  Prints "<boxes> <vertices> <outside>
// <outside without the rounding margin> <boxes that are not finite and not
// marked so>".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "sgl_cull.h"
#include "sgl_device.cuh"

using namespace sgl;

int main(int argc, char **argv)
{
    const long n = argc > 1 ? std::atol(argv[1]) : 100000;
    std::mt19937_64 gen(1234567);
    std::uniform_real_distribution<double> uni(-1.0, 1.0);
    auto exp10u = [&](double lo, double hi) { return std::pow(10.0, lo + (hi - lo) * 0.5 * (uni(gen) + 1.0)); };
    long vertices = 0, outside = 0, bare = 0, unmarked = 0;
    for (long k = 0; k < n; k++) {
        float M[16] = {};
        const int kind = (int)(gen() % 6);
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++)
                M[4 * i + j] = (float)uni(gen);
        if (kind == 1) { // an axis permutation with signs, as a quarter turn
            for (int i = 0; i < 3; i++)
                for (int j = 0; j < 3; j++)
                    M[4 * i + j] = j == (i + 1) % 3 ? (gen() & 1 ? 1.0f : -1.0f) : 0.0f;
        } else if (kind == 2) {
            const float s = (float)exp10u(-4, 4);
            for (int i = 0; i < 3; i++)
                for (int j = 0; j < 3; j++)
                    M[4 * i + j] *= s;
        } else if (kind == 3) {
            M[4] = M[5] = M[6] = 0.0f;
        }
        const double shift = kind == 4 ? 0.0 : exp10u(-3, 6);
        for (int i = 0; i < 3; i++)
            M[4 * i + 3] = (float)(shift * uni(gen));
        const int count = 1 + (int)(gen() % 66);
        const double size = exp10u(-4, 3), far = kind == 5 ? exp10u(0, 6) : 0.0;
        V3 p[66], at = mk3((float)(far * uni(gen)), (float)(far * uni(gen)), (float)(far * uni(gen)));
        float3 lo = make_float3(INFINITY, INFINITY, INFINITY), hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
        const bool wild = k % 64 == 63; // a coordinate that is infinite, or so large that its products are
        for (int v = 0; v < count; v++) {
            p[v] = mk3(at.x + (float)(size * uni(gen)), at.y + (float)(size * uni(gen)), at.z + (float)(size * uni(gen)));
            if (wild && v == 0)
                p[v].y = k % 128 == 63 ? INFINITY : 3e38f;
            lo = make_float3(fminf(lo.x, p[v].x), fminf(lo.y, p[v].y), fminf(lo.z, p[v].z));
            hi = make_float3(fmaxf(hi.x, p[v].x), fmaxf(hi.y, p[v].y), fmaxf(hi.z, p[v].z));
        }
        float4 bc, bh, pc, ph;
        cull_box(lo, hi, bc, bh);
        pose_box(M, bc, bh, pc, ph);
        if (std::isnan(pc.x))
            continue; // never skipped
        if (wild)
            unmarked++;
        const double c[3] = {pc.x, pc.y, pc.z}, h[3] = {ph.x, ph.y, ph.z};
        for (int v = 0; v < count; v++) {
            const V3 w = transform3(p[v], M);
            const double d[3] = {std::fabs(w.x - c[0]), std::fabs(w.y - c[1]), std::fabs(w.z - c[2])};
            bool out = false, tight = false;
            for (int i = 0; i < 3; i++) {
                const float *m = M + 4 * i;
                const double reach = std::fabs(m[0]) * (double)bh.x + std::fabs(m[1]) * (double)bh.y +
                                     std::fabs(m[2]) * (double)bh.z;
                out |= !(d[i] <= h[i]);
                tight |= !(d[i] <= reach);
            }
            vertices++;
            outside += out;
            bare += tight;
        }
    }
    std::printf("%ld %ld %ld %ld %ld\n", n, vertices, outside, bare, unmarked);
    return 0;
}
