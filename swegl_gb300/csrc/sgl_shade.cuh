// sgl_shade.cuh — the pixel shaders of the swegl render path on the device:
// pixel_shader_lights_phong, pixel_shader_lights_flat, pixel_shader_texture
// (nearest), pixel_shader_texture_bilinear, the material colour of
// pixel_shader_t, and their pixel_shader_light_and_texture<L, T>
// combinations (swegl/render/pixel_shaders.hpp:15-179,
// src/render/pixel_shaders.cpp:14-384), with the reference's single-precision
// operation order.
#pragma once

#include "sgl_device.cuh"
#include "sgl_internal.h"

namespace sgl {

// What the pixel shaders read at one fragment: the state that
// pixel_shader_light_and_texture<lights_phong, texture_bilinear>
// (swegl/render/pixel_shaders.hpp:76-97,125-150,121-179) carries along a span,
// evaluated at the fragment (sh_fragment), and what bind_material binds.
struct Shader {
    V3 center, n; // position, and normal before its normalisation
    V2 t;         // texture coordinates in texels
    const uint32_t *tex;
    uint32_t color;
    int tw, th, shininess;
    int flat_light; // pixel_shader_lights_flat::light as shade() returns it
};

// One vertex as the pixel shaders read it.
struct SVert {
    V3 p, n;
    V2 uv;
};

// Which of a triangle's vertices (v0, v1, v2 in fill_triangle_2's order) the
// two edges of a span of half `lower` run between: both edges share vertex s
// (v0 in the upper half, v2 in the lower one); the other end of the left edge
// is l, of the right edge r.  The long edge v0 -> v2 is the right one when
// `llr`.
__device__ __forceinline__ void sh_edge_ends(bool lower, bool llr, uint32_t g0, uint32_t g1, uint32_t g2, uint32_t &s,
                                             uint32_t &l, uint32_t &r)
{
    s = lower ? g2 : g0;
    const uint32_t o = lower ? g0 : g2; // the long edge's other end
    l = llr ? g1 : o;
    r = llr ? o : g1;
}

__device__ __forceinline__ V3 sel3(bool c, V3 a, V3 b) { return mk3(c ? a.x : b.x, c ? a.y : b.y, c ? a.z : b.z); }
__device__ __forceinline__ V2 sel2(bool c, V2 a, V2 b) { return mk2(c ? a.x : b.x, c ? a.y : b.y); }

// prepare_for_triangle, prepare_for_upper/lower_triangle, prepare_for_scanline
// (src/render/pixel_shaders.cpp:88-158,304-346) and the interpolation of
// shade(): position, normal and texture coordinates run along the left edge
// to progress pl, along the right edge to pr, and between the two to
// `progress`, each as start + (end - start) * progress.  Both lower edges end
// at s, both upper ones start there.  The reference negates the three normals
// of an `inverted` triangle before interpolating; every step commutes with
// that sign, so it is taken at the end.
__device__ __forceinline__ void sh_fragment(Shader &sh, const SVert &s, const SVert &l, const SVert &r, bool lower,
                                            bool inverted, float pl, float pr, float progress)
{
    {
        const V3 a = sel3(lower, l.p, s.p), b = sel3(lower, s.p, l.p);
        const V3 c = sel3(lower, r.p, s.p), d = sel3(lower, s.p, r.p);
        const V3 v = add3(a, mul3(sub3(b, a), pl));
        sh.center = add3(v, mul3(sub3(add3(c, mul3(sub3(d, c), pr)), v), progress));
    }
    {
        const V3 a = sel3(lower, l.n, s.n), b = sel3(lower, s.n, l.n);
        const V3 c = sel3(lower, r.n, s.n), d = sel3(lower, s.n, r.n);
        const V3 v = add3(a, mul3(sub3(b, a), pl));
        const V3 n = add3(v, mul3(sub3(add3(c, mul3(sub3(d, c), pr)), v), progress));
        sh.n = sel3(inverted, neg3(n), n);
    }
    {
        const float tw = (float)sh.tw, th = (float)sh.th;
        const V2 ts = mk2(s.uv.x * tw, s.uv.y * th), tl = mk2(l.uv.x * tw, l.uv.y * th),
                 tr = mk2(r.uv.x * tw, r.uv.y * th);
        const V2 a = sel2(lower, tl, ts), b = sel2(lower, ts, tl);
        const V2 c = sel2(lower, tr, ts), d = sel2(lower, ts, tr);
        const V2 v = add2(a, mul2(sub2(b, a), pl));
        sh.t = add2(v, mul2(sub2(add2(c, mul2(sub2(d, c), pr)), v), progress));
    }
}

// The sun and point-light sum of the Phong and the flat light shaders
// (src/render/pixel_shaders.cpp:159-205 per pixel, :33-84 per triangle): the
// same expressions at a point with a normal.
//
// A point light whose direction the reference would find behind the surface
// (alignment < 0, the light skipped) is skipped here before its division and
// normalisation when the unnormalised dot product already shows it with a
// margin that rounding cannot cross: with a_i = n_i * d_i (d = center minus
// the light), the float sum of the a_i is within 3 * 2^-24 * sum |a_i| of the
// exact dot product, and the reference's dot product of n with the
// normalised d (three IEEE divisions by the same length, three products, two
// sums) is within 2^-22 * sum |a_i| / length of the exact one divided by
// that length.  A float sum above 2^-20 * sum |a_i| therefore makes both
// positive, and the reference skips the light too (its test on the
// intensity / distance^2 ratio only skips more).  Sums below 2^-100 (where
// products could be subnormal), squared distances from 2^100 up (where the
// length could overflow) and NaNs take the full path.
//
// The specular power is left out where the term cannot change the diffuse one
// that it is added to: with b the base, the term is b^p p / 2 / d2, and where
// p log2(b) < log2(diffuse d2) - 36 it is below p / 2 * 2^-36 of the diffuse
// term, for p up to 1024 below 2^-27 of it, while half a unit in its last
// place is at least 2^-25 of it.  The factor of 4 between them holds what the
// approximate logarithms (2^-22 each, the first times p), the roundings of the
// test and a subnormal diffuse d2 can add, together less than a factor of 2.
// Only materials are held to 1024 at upload: a default material's exponent
// beyond it, or below 0, takes the power (without that bound 59,328 of the
// 2,000,000 sums of tests/shade_math/light_skip.cu differ).
__host__ __device__ __forceinline__ float light_sum(const LightsDev &L, V3 center, V3 normal, V3 camvec,
                                                    int shininess)
{
    float face_sun = -dot3(normal, mk3(L.sun[0], L.sun[1], L.sun[2]));
    if (face_sun < 0.0f)
        face_sun = 0.0f;
    else
        face_sun = face_sun * L.sun_intensity;
    float dyn = 0.0f;
    const float fp = (float)shininess;
    for (int l = 0; l < L.n; l++) {
        const float4 pl = L.pl[l];
        V3 ld = sub3(center, mk3(pl.x, pl.y, pl.z));
        const float d2 = ld.x * ld.x + ld.y * ld.y + ld.z * ld.z;
        const float ax = normal.x * ld.x, ay = normal.y * ld.y, az = normal.z * ld.z;
        const float mag = fabsf(ax) + fabsf(ay) + fabsf(az);
        if (ax + ay + az > 0x1p-20f * mag && mag > 0x1p-100f && d2 < 0x1p100f)
            continue; // behind the surface
        float diffuse = pl.w / d2;
        if (diffuse < 0.05f) // (double)diffuse < 0.05, see sgl_device.cuh
            continue;
        ld = normalize_fast(ld);
        const float alignment = -dot3(normal, ld);
        if (alignment < 0.0f)
            continue;
        diffuse = diffuse * alignment;
        const V3 reflection = add3(ld, mul3(normal, alignment * 2.0f));
        float specular = dot3(reflection, camvec);
        const bool unseen =
            fp * log2_approx(specular) < log2_approx(diffuse * d2) - 36.0f && (uint32_t)shininess <= 1024u;
        if (specular > 0.0f && !unseen) {
            specular = spec_pow(specular, shininess);
            specular = specular * fp / 2.0f;
            dyn = dyn + (diffuse + specular / d2);
        } else {
            dyn = dyn + diffuse;
        }
    }
    return L.ambient + face_sun + dyn;
}

// pixel_shader_lights_phong::shade (src/render/pixel_shaders.cpp:159-205)
__device__ __forceinline__ int sh_phong(const Shader &sh, const LightsDev &L, const ViewDev &v)
{
    const V3 normal = normalize_fast(sh.n);
    const V3 camvec = normalize_fast(sub3(mk3(v.campos[0], v.campos[1], v.campos[2]), sh.center));
    return f2i(65536.0f * light_sum(L, sh.center, normal, camvec, sh.shininess));
}

// pixel_shader_lights_flat::prepare_for_triangle (src/render/pixel_shaders.cpp:
// 33-84) on fill_triangle_2's vertex order: the face normal (cross()
// normalises; the unary minus of a normal_t builds a normal_t, normalised
// again), the centroid (v0 + v1 + v2) / 3 and the same light sum; shade()
// returns light * 65536 converted to int.
__device__ __forceinline__ int flat_light(const V3 w[3], bool inverted, const LightsDev &L, const ViewDev &v,
                                          int shininess)
{
    V3 normal = cross_n(sub3(w[1], w[0]), sub3(w[2], w[0]));
    if (inverted)
        normal = normalize3(neg3(normal));
    const V3 sum = add3(add3(w[0], w[1]), w[2]);
    const V3 center = mk3(sum.x / 3.0f, sum.y / 3.0f, sum.z / 3.0f);
    const V3 camvec = normalize3(sub3(mk3(v.campos[0], v.campos[1], v.campos[2]), center));
    float light = light_sum(L, center, normal, camvec, shininess);
    light = light * 65536.0f;
    return f2i(light);
}

// pixel_shader_texture::shade (src/render/pixel_shaders.cpp:276-281): the
// texel at (int)t % size, the int converted to unsigned by the unsigned width
// and height.
__device__ __forceinline__ uint32_t sh_nearest(const Shader &sh)
{
    const V2 t = sh.t;
    const uint32_t tw = (uint32_t)sh.tw, th = (uint32_t)sh.th;
    const uint32_t u = (uint32_t)f2i(t.x) % tw;
    const uint32_t vv = (uint32_t)f2i(t.y) % th;
    if (sh.tex && !in_bounds(u < tw && vv < th, CHK_TEXEL, (unsigned long long)vv * tw + u))
        return 0u;
    return sh.tex ? __ldg(sh.tex + vv * tw + u) : sh.color; // untextured: 1x1 of the colour
}

// The remainder of `i + n` by n as the reference's int arithmetic gives it
// (it keeps the sign of a negative dividend), without the division while i
// is in [-n, n).
__device__ __forceinline__ int wrap_texel(int i, int n)
{
    int m = i < 0 ? i + n : i;
    if ((uint32_t)m >= (uint32_t)n)
        m = (n & (n - 1)) == 0 && i >= 0 ? i & (n - 1) : (i + n) % n;
    return m;
}

// A sum of weighted bytes, 0 <= x < 2^22, rounded half away from zero
// (roundf): adding 2^23 rounds to the nearest integer with ties to even, and
// a tie that went down leaves a remainder of exactly 0.5.
__device__ __forceinline__ uint32_t round_byte(float x)
{
    const float t = x + 8388608.0f;
    return (__float_as_uint(t) + (x - (t - 8388608.0f) == 0.5f ? 1u : 0u)) & 0xFFu;
}

// pixel_shader_texture_bilinear::shade (src/render/pixel_shaders.cpp:348-384)
// with the pixel_colors_f sums of src/render/colors.cpp:11-30.  v comes from
// t.x and u from t.y, as in the reference.  FAST: both coordinates are below
// 2^22 in magnitude, so their conversions are in range, the weights lie in
// [0, 1] and the sums are bytes.
template <bool FAST>
__device__ __forceinline__ uint32_t bilinear_at(const uint32_t *tex, int tw, int th, uint32_t color, V2 t)
{
    float v = t.x;
    float u = t.y;
    // (float)(u - 0.5) in double equals u - 0.5f in float: 0.5 is exact and
    // double rounding is innocuous for a single subtraction.
    const float u1 = u - 0.5f, u2 = u + 0.5f, v1 = v - 0.5f, v2 = v + 0.5f;
    u = floorf(u2);
    v = floorf(v2);
    int v1m = FAST ? wrap_texel(__float2int_rz(v1), th) : (f2i(v1) + th) % th;
    int v2m = v1m + 1;
    if (v2m == th)
        v2m = 0;
    const int u1m = FAST ? wrap_texel(__float2int_rz(u1), tw) : (f2i(u1) + tw) % tw;
    int u2m = u1m + 1;
    if (u2m == tw)
        u2m = 0;
    const float w11 = (u - u1) * (v - v1), w21 = (u - u1) * (v2 - v), w12 = (u2 - u) * (v - v1),
                w22 = (u2 - u) * (v2 - v);
    uint32_t c11 = color, c21 = color, c12 = color, c22 = color; // untextured: 1x1 of the colour
    const long long row1 = (long long)v1m * tw, row2 = (long long)v2m * tw;
    if (!FAST || (v1m | u1m) < 0) { // (a negative remainder)
        const long long n = (long long)tw * th, i11 = row1 + u1m, i21 = row2 + u1m, i12 = row1 + u2m, i22 = row2 + u2m;
        if (i11 < 0 || i11 >= n || i21 < 0 || i21 >= n || i12 < 0 || i12 >= n || i22 < 0 || i22 >= n)
            return 0u; // the reference reads outside the texture here
    }
    if (tex) {
        // the two texels of a row are neighbours unless the column wraps: one
        // 8-byte load when the pair starts on an even texel (textures start
        // 256-byte aligned), else two 4-byte loads
        const uint32_t *r1 = tex + row1, *r2 = tex + row2;
        const bool pair = u2m == u1m + 1;
        if (pair && ((uintptr_t)(r1 + u1m) & 7) == 0) {
            const uint2 q = __ldg(reinterpret_cast<const uint2 *>(r1 + u1m));
            c11 = q.x;
            c12 = q.y;
        } else {
            c11 = __ldg(r1 + u1m);
            c12 = __ldg(r1 + u2m);
        }
        if (pair && ((uintptr_t)(r2 + u1m) & 7) == 0) {
            const uint2 q = __ldg(reinterpret_cast<const uint2 *>(r2 + u1m));
            c21 = q.x;
            c22 = q.y;
        } else {
            c21 = __ldg(r2 + u1m);
            c22 = __ldg(r2 + u2m);
        }
    }
    uint32_t out = 0;
#pragma unroll
    for (int ch = 0; ch < 4; ch++) {
        const int sft = 8 * ch;
        float acc = (float)((c11 >> sft) & 0xFFu) * w11;
        acc = acc + (float)((c21 >> sft) & 0xFFu) * w21;
        acc = acc + (float)((c12 >> sft) & 0xFFu) * w12;
        acc = acc + (float)((c22 >> sft) & 0xFFu) * w22;
        out |= (FAST ? round_byte(acc) : (uint32_t)f2i(roundf(acc)) & 0xFFu) << sft;
    }
    return out;
}

// texture coordinates of 2^22 texels and more, infinities and NaNs
__device__ __noinline__ uint32_t bilinear_far(const uint32_t *tex, int tw, int th, uint32_t color, float tx, float ty)
{
    return bilinear_at<false>(tex, tw, th, color, mk2(tx, ty));
}

__device__ __forceinline__ uint32_t sh_bilinear(const Shader &sh)
{
    if (!(fabsf(sh.t.x) < 4194304.0f && fabsf(sh.t.y) < 4194304.0f))
        return bilinear_far(sh.tex, sh.tw, sh.th, sh.color, sh.t.x, sh.t.y);
    return bilinear_at<true>(sh.tex, sh.tw, sh.th, sh.color, sh.t);
}

// The view's pixel shader (SGL_SHADER_*, include/sgl.h); the combinations are
// pixel_shader_light_and_texture::shade (swegl/render/pixel_shaders.hpp:159-178).
// ALL_MODES = false compiles the default Phong + bilinear shader alone.
template <bool ALL_MODES = true>
__device__ __forceinline__ uint32_t sh_shade(const Shader &sh, const LightsDev &L, const ViewDev &v)
{
    const int mode = ALL_MODES ? v.shader : SGL_SHADER_PHONG_BILINEAR;
    if (mode >= SGL_SHADER_COLOR) {
        switch (mode) {
        case SGL_SHADER_COLOR: return sh.color;
        case SGL_SHADER_BILINEAR: return sh_bilinear(sh);
        case SGL_SHADER_NEAREST: return sh_nearest(sh);
        case SGL_SHADER_PHONG: return (uint32_t)sh_phong(sh, L, v);
        default: return (uint32_t)sh.flat_light; // SGL_SHADER_FLAT
        }
    }
    const bool nearest = mode == SGL_SHADER_PHONG_NEAREST || mode == SGL_SHADER_FLAT_NEAREST;
    const bool flat = mode == SGL_SHADER_FLAT_BILINEAR || mode == SGL_SHADER_FLAT_NEAREST;
    uint32_t color = nearest ? sh_nearest(sh) : sh_bilinear(sh);
    // (float)(i / 65536.0): the int rounded to float, then an exact power-of-two scale
    float light = __int2float_rn(flat ? sh.flat_light : sh_phong(sh, L, v)) * (1.0f / 65536.0f);
    uint32_t out = color & 0xFF000000u;
    if (light < 1.0f) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const uint32_t c = (color >> (8 * k)) & 0xFFu;
            // (|light| <= 2^15: the conversion is in range)
            out |= ((uint32_t)__float2int_rz((float)c * light) & 0xFFu) << (8 * k);
        }
    } else {
        light = sqrtf(light);
        light = sqrtf(light);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const uint32_t c = (color >> (8 * k)) & 0xFFu;
            const uint32_t q = (uint32_t)__float2int_rz((float)(255u - c) / light) & 0xFFu;
            out |= ((255u - q) & 0xFFu) << (8 * k);
        }
    }
    return out;
}


} // namespace sgl
