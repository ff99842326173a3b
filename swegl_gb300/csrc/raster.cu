// raster.cu — sm_103a kernels of the swegl render path.
//
// Every kernel works on a batch of views (items: scene, camera, buffers) and
// is a persistent grid-stride kernel with a fixed grid that reads the batch
// totals from device memory, so one launch sequence (and one CUDA graph)
// serves any batch.  The plain one-frame-per-launch renderer is a batch of one.
//
//   k_geom        the next three for primitives of few vertices, a warp each
//   k_vertex      world -> view -> projection, |z'| divide      (vertex_shaders.hpp:35-52)
//   k_flags       visibility flags of triangles                  (renderer.cpp:86-185)
//   k_compact     drawable triangles -> the walk, tall or near-clip list
//   k_walk        scanline set-ups (TriRec) of 32 walk-list triangles, their
//                 rows dealt across a warp's lanes, fragment keys folded with
//                 an atomic min; then the warp's share of the near-clip
//                 triangles and of the tall triangles
//   k_spans       long spans binned by the walk, several lanes each
//   k_winners     winner records of binned spans and near-clip triangles
//                 (every span after a bin overflow)
//   k_shade       batches of several views, per pixel: background or the
//                 winner's colour, and depth; winners are queued so that
//                 shading runs on full warps
//   k_classify    single views: background, depth, the list of winners (and
//                 k_winners' records)
//   k_shade_wins  ... and the winners' colours
//   k_dof         depth-of-field gather of the items that ask for it
//
// Depth test.  The reference draws triangles in order and keeps a fragment
// when z < zbuffer (strict, src/render/renderer.cpp:489-499), so the earliest
// drawn of equal-depth fragments wins.  Each fragment here folds the 64-bit
// key (float bits of z << 32 | draw slot) into its pixel with atomicMin: z is
// above 0.001, so its bits order like the floats, and the draw slot
// (2 * draw-order triangle + clip sub-triangle) breaks ties in draw order.
// The shade kernel then replays the winner's row and pixel steps from the
// triangle's set-up record to recover the progress values the reference
// shaded with; spans too long to replay cheaply have them recorded by the
// span kernels instead.  The depth keys start every launch sequence empty:
// new key pools are filled once and the shade kernel empties what it reads.
#include <cstdint>

#include "sgl_cull.h"
#include "sgl_device.cuh"
#include "sgl_dof_taps.h"
#include "sgl_internal.h"
#include "sgl_shade.cuh"

namespace sgl {

// Index of the item owning global index x: largest i with base[i] <= x.
__device__ __forceinline__ int find_item(const uint32_t *base, int n, uint32_t x)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(base + mid) <= x)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// Walks a grid-stride range over the concatenated per-item ranges given by
// `base`, calling fn(item, local_index); the item is looked up only when the
// index leaves the previous item's range.
template <class Fn>
__device__ __forceinline__ void for_each_in_items(const BatchDev *b, const uint32_t *base, uint32_t total, Fn &&fn)
{
    int item = -1;
    uint32_t lo = 0, hi = 0;
    const int n = b->n_items;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
        if (g < lo || g >= hi) {
            item = find_item(base, n, g);
            lo = __ldg(base + item);
            hi = __ldg(base + item + 1);
        }
        fn(item, g - lo);
    }
}

// Depth-key reduction without a return value (red.global.min.u64): the
// 64-bit atomicMin() returns the old key, and a warp would wait for that round
// trip on every fragment.
__device__ __forceinline__ void key_min(unsigned long long *p, unsigned long long v)
{
    asm volatile("red.global.min.u64 [%0], %1;\n" ::"l"(p), "l"(v) : "memory");
}

// Asynchronous global -> shared copies of BYTES (cp.async), committed as groups.
template <int BYTES> __device__ __forceinline__ void cp_async(void *smem, const void *gmem)
{
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(sa), "l"(gmem), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ---------------------------------------------------------------- vertices --

// vertex_shader_t::original_to_world (swegl/render/vertex_shaders.hpp:16-33) and
// the view-independent normal of camera_to_frustum (:63): rotate() normalises,
// .normalize() again, and the normal_t assignment a third time.
__global__ void k_world(SceneDev s)
{
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= s.n_vertices)
        return;
    const uint32_t n = s.vnode[g];
    const float *M = s.node_world + 16 * n;
    const float *RS = s.node_rs + 16 * n;
    const float4 p = s.pos_u[g];
    const float4 q = s.nrm_v[g];
    const V3 w = transform3(mk3(p.x, p.y, p.z), M);
    const V3 nw = normalize_fast<true>(normalize_fast<true>(rotate_n(mk3(q.x, q.y, q.z), RS)));
    s.wpos[g] = make_float4(w.x, w.y, w.z, p.w);
    s.wnrm[g] = make_float4(nw.x, nw.y, nw.z, q.w);
}

// k_world for a batch's posed views: the same transforms under each view's own
// node matrices, into its own arrays, all views in one launch (a launch and a
// copy per view, half of a 16-view batch's passes before its first triangle,
// left the GPU idle between them).  Blocks beyond the vertices' make the boxes
// of the small primitives, each from its box before the transform (pose_box;
// a primitive is under one node): read back from the posed positions, a warp
// a primitive, they took a second pass (16 views of 50 spheres: 18 us beside
// the transforms' 32; now 32 together, the looser boxes cost k_geom nothing).
// One pass with a warp a primitive took 48: a strip's 66 vertices fill 69 % of
// its lanes, and the transforms are bound by instruction issue.
// Index of the pose whose blocks (`first`) hold block x.
template <uint32_t PoseDev::*FIRST> __device__ __forceinline__ int find_pose(const PoseDev *p, int n, uint32_t x)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (p[mid].*FIRST <= x)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}
__global__ void __launch_bounds__(256) k_pose(const PoseDev *poses, int n, uint32_t vertex_blocks)
{
    if (blockIdx.x >= vertex_blocks) {
        const uint32_t x = blockIdx.x - vertex_blocks;
        const PoseDev &p = poses[find_pose<&PoseDev::prim_block>(poses, n, x)];
        const uint32_t q = (x - p.prim_block) * kPosePrims + threadIdx.x;
        if (p.pbox && q < p.n_prims) {
            const uint4 gq = p.pgeo[q];
            float4 c = make_float4(NAN, 0.0f, 0.0f, 0.0f), h = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (gq.y && in_bounds(gq.x < p.n_vertices, CHK_NDC, gq.x))
                pose_box(p.node_world + 16 * p.vnode[gq.x], p.lbox[2 * q], p.lbox[2 * q + 1], c, h);
            p.pbox[2 * q] = c;
            p.pbox[2 * q + 1] = h;
        }
        return;
    }
    const PoseDev p = poses[find_pose<&PoseDev::vertex_block>(poses, n, blockIdx.x)];
    const uint32_t g0 = (blockIdx.x - p.vertex_block) * kPoseVertices + threadIdx.x;
    constexpr int kPer = kPoseVertices / 256;
    float4 a[kPer], q[kPer];
    uint32_t node[kPer];
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const uint32_t g = g0 + 256 * k;
        if (g < p.n_vertices) {
            a[k] = p.pos_u[g];
            q[k] = p.nrm_v[g];
            node[k] = p.vnode[g];
        }
    }
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const uint32_t g = g0 + 256 * k;
        if (g >= p.n_vertices)
            break;
        const V3 w = transform3(mk3(a[k].x, a[k].y, a[k].z), p.node_world + 16 * node[k]);
        const V3 nw = normalize_fast<true>(normalize_fast<true>(rotate_n(mk3(q[k].x, q[k].y, q[k].z), p.node_rs + 16 * node[k])));
        p.wpos[g] = make_float4(w.x, w.y, w.z, a[k].w);
        p.wnrm[g] = make_float4(nw.x, nw.y, nw.z, q[k].w);
    }
}

// The box of each primitive's world positions (a warp per primitive), for the
// fused pass's whole-primitive frustum test: pbox[2 q] = centre, pbox[2 q + 1]
// = half extent.  NaN coordinates are left out (a triangle with one fails
// each test of inside_camera_frustum that its other vertices fail, the
// comparisons with NaN being false); a box that is empty or not finite gets a
// NaN centre and is never culled.
__device__ __forceinline__ void primitive_box(uint4 gq, uint32_t n_vertices, const float4 *wpos, float4 *out)
{
    const uint32_t lane = threadIdx.x & 31;
    V3 lo = mk3(INFINITY, INFINITY, INFINITY), hi = mk3(-INFINITY, -INFINITY, -INFINITY);
    for (uint32_t i = lane; i < gq.y; i += 32) {
        if (!in_bounds(gq.x + i < n_vertices, CHK_NDC, gq.x + i))
            break;
        const float4 w = wpos[gq.x + i];
        lo = mk3(fminf(lo.x, w.x), fminf(lo.y, w.y), fminf(lo.z, w.z));
        hi = mk3(fmaxf(hi.x, w.x), fmaxf(hi.y, w.y), fmaxf(hi.z, w.z));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo.x = fminf(lo.x, __shfl_xor_sync(0xFFFFFFFFu, lo.x, o));
        lo.y = fminf(lo.y, __shfl_xor_sync(0xFFFFFFFFu, lo.y, o));
        lo.z = fminf(lo.z, __shfl_xor_sync(0xFFFFFFFFu, lo.z, o));
        hi.x = fmaxf(hi.x, __shfl_xor_sync(0xFFFFFFFFu, hi.x, o));
        hi.y = fmaxf(hi.y, __shfl_xor_sync(0xFFFFFFFFu, hi.y, o));
        hi.z = fmaxf(hi.z, __shfl_xor_sync(0xFFFFFFFFu, hi.z, o));
    }
    if (lane == 0) {
        float4 c, h;
        cull_box(make_float3(lo.x, lo.y, lo.z), make_float3(hi.x, hi.y, hi.z), c, h);
        out[0] = c;
        out[1] = h;
    }
}
// Counts of kAlphaSamples points a triangle those with an alpha below 255: the
// texels under its centroid and the points halfway from there to its corners,
// found as the bilinear shader finds them, or its material's colour.  (By
// triangles, not by texels: of a texture that many objects share, some may be
// opaque and others not.)
__device__ __forceinline__ void count_translucent(const SceneDev &s, uint32_t t)
{
    uint32_t n = 0;
    if (t < s.n_triangles) {
        const uint4 tri = s.tris[t];
        const PrimShade ps = s.pshade[tri.w];
        if (!ps.tex) {
            n = (ps.color >> 24) != 255u ? kAlphaSamples : 0u;
        } else {
            const V2 a = mk2(s.pos_u[tri.x].w, s.nrm_v[tri.x].w), b = mk2(s.pos_u[tri.y].w, s.nrm_v[tri.y].w),
                     c = mk2(s.pos_u[tri.z].w, s.nrm_v[tri.z].w);
            const V2 mid = mul2(add2(add2(a, b), c), 1.0f / 3.0f);
            // floor(x) modulo `size`, 0 where it has none
            auto wrap = [](float x, int size) {
                const float f = (float)size, r = x - floorf(x / f) * f;
                return r >= 0.0f && r < f ? min((int)r, size - 1) : 0;
            };
            static_assert(kAlphaSamples == 4, "the centroid and three points");
            const V2 at[kAlphaSamples] = {mid, mul2(add2(mid, a), 0.5f), mul2(add2(mid, b), 0.5f), mul2(add2(mid, c), 0.5f)};
#pragma unroll
            for (int k = 0; k < (int)kAlphaSamples; k++)
                n += (__ldg(ps.tex + (size_t)wrap(at[k].x * (float)ps.tw, ps.th) * ps.tw +
                            wrap(at[k].y * (float)ps.th, ps.tw)) >> 24) != 255u;
        }
    }
    n = __reduce_add_sync(0xFFFFFFFFu, n);
    if ((threadIdx.x & 31) == 0 && n)
        atomicAdd(s.translucent, (unsigned long long)n);
}

// The boxes, and at upload those of the positions before any transform
// (`lbox`) in the first `box_blocks` blocks, the translucent samples in the
// others.  (Launches and arrays of their own cost a small scene's upload: the
// textured cube 177 us, 149 so, 159 before there were samples and such boxes.)
__global__ void __launch_bounds__(256) k_box(SceneDev s, float4 *lbox, uint32_t box_blocks)
{
    if (blockIdx.x >= box_blocks) {
        count_translucent(s, (blockIdx.x - box_blocks) * 256 + threadIdx.x);
        return;
    }
    const uint32_t w = (blockIdx.x * 256 + threadIdx.x) >> 5;
    const bool local = w >= s.n_prims;
    const uint32_t q = local ? w - s.n_prims : w;
    if (q < s.n_prims && (!local || lbox))
        primitive_box(s.pgeo[q], s.n_vertices, local ? s.pos_u : s.wpos, (local ? lbox : s.pbox) + 2 * q);
}
// world_to_camera_or_frustum (vertex_shaders.hpp:35-52): view, projection
// (rows 0-2), x and y divided by |z'|; also clears the visibility flag.  The
// item's matrices stay in registers while the index is inside it.  Each
// thread takes kGeomPer vertices (a warp 32 * kGeomPer consecutive ones) and
// issues their loads first.
constexpr int kGeomPer = 4;
__global__ void __launch_bounds__(256) k_vertex(const BatchDev *b)
{
    uint32_t lo = 0, hi = 0;
    float m[24];
    const float4 *wpos = nullptr;
    float4 *ndc = nullptr;
    uint8_t *yes = nullptr;
    const uint8_t *vsmall = nullptr; // a mixed scene: vertices the fused pass transforms
    const uint32_t total = b->total_gvtx;
    auto bind = [&](uint32_t g) {
        const int item = find_item(b->g_vtx_base, b->n_items, g);
        lo = __ldg(b->g_vtx_base + item);
        hi = __ldg(b->g_vtx_base + item + 1);
        const ItemDev &it = b->items[item];
#pragma unroll
        for (int k = 0; k < 12; k++) {
            m[k] = it.v.view[k];
            m[12 + k] = it.v.proj[k];
        }
        wpos = it.s.wpos;
        ndc = it.ndc;
        yes = it.yes;
        vsmall = it.s.vsmall;
    };
    auto project = [&](uint32_t l, float4 w) {
        if (vsmall && vsmall[l])
            return;
        V3 p = transform3(mk3(w.x, w.y, w.z), m);
        p = transform3(p, m + 12);
        if (p.z != 0.0f) {
            p.x = p.x / fabsf(p.z);
            p.y = p.y / fabsf(p.z);
        }
        if (!in_bounds(l < hi - lo, CHK_NDC, l))
            return;
        ndc[l] = make_float4(p.x, p.y, p.z, 0.0f);
        yes[l] = below_near(p.z) ? kYesBehind : 0; // kYesDrawn is set by k_flags
    };
    // a warp takes 32 * kGeomPer consecutive vertices, lane + 32 u each
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t stride = gridDim.x * blockDim.x * kGeomPer;
    for (uint32_t g0 = ((blockIdx.x * blockDim.x + threadIdx.x) & ~31u) * kGeomPer + lane; g0 < total; g0 += stride) {
        const uint32_t glast = g0 + 32 * (kGeomPer - 1);
        if (g0 < lo || g0 >= hi)
            bind(g0);
        if (glast < hi && glast < total) {
            const uint32_t l = g0 - lo;
            float4 w[kGeomPer];
#pragma unroll
            for (int u = 0; u < kGeomPer; u++)
                w[u] = wpos[l + 32 * u];
#pragma unroll
            for (int u = 0; u < kGeomPer; u++)
                project(l + 32 * u, w[u]);
        } else {
            for (uint32_t g = g0; g <= glast && g < total; g += 32) {
                if (g < lo || g >= hi)
                    bind(g);
                project(g - lo, wpos[g - lo]);
            }
        }
    }
}

// inside_camera_frustum (src/render/renderer.cpp:58-70)
// (a >= k || b >= k || c >= k is max(a, b, c) >= k, NaNs ignored alike)
__device__ __forceinline__ bool inside_frustum(V3 a, V3 b, V3 c)
{
    return fmaxf(fmaxf(a.x, b.x), c.x) >= -1.0f && fmaxf(fmaxf(a.y, b.y), c.y) >= -1.0f &&
           fminf(fminf(a.x, b.x), c.x) < 1.0f && fminf(fminf(a.y, b.y), c.y) < 1.0f &&
           at_or_past_near(fmaxf(fmaxf(a.z, b.z), c.z)) && (a.x != b.x || a.x != c.x) && (a.y != b.y || a.y != c.y);
}

__device__ __forceinline__ V3 ld3(const float4 *a, uint32_t i)
{
    const float4 t = a[i];
    return mk3(t.x, t.y, t.z);
}

// Visibility flags (renderer.cpp:86-185): inside the frustum and (double sided
// or front facing, front_face_visible :72-75, on the draw-order triple).
constexpr int kFlagsPer = 2;
__global__ void __launch_bounds__(256) k_flags(const BatchDev *b)
{
    uint32_t lo = 0, hi = 0;
    const uint4 *tris = nullptr;
    const float4 *ndc = nullptr;
    uint8_t *yes = nullptr;
    const PrimDesc *prims = nullptr;
    const MatDesc *mats = nullptr;
    const uint8_t *psmall = nullptr; // a mixed scene: primitives of the fused pass
    int n_mats = 0;
    const uint32_t total = b->total_gtri;
    auto bind = [&](uint32_t g) {
        const int item = find_item(b->g_tri_base, b->n_items, g);
        lo = __ldg(b->g_tri_base + item);
        hi = __ldg(b->g_tri_base + item + 1);
        const ItemDev &it = b->items[item];
        tris = it.s.tris;
        ndc = it.ndc;
        yes = it.yes;
        prims = it.s.prims;
        mats = it.s.mats;
        n_mats = it.s.n_mats;
        psmall = it.s.psmall;
    };
    auto flag = [&](uint4 tri, V3 a, V3 c1, V3 c2) {
        if ((psmall && psmall[tri.w]) || !inside_frustum(a, c1, c2))
            return;
        // front facing, else double sided (the material is read only then)
        bool vis = cross_z_positive(sub3(c1, a), sub3(c2, a));
        if (!vis) {
            const int m = prims[tri.w].material;
            vis = m >= 0 && m < n_mats && mats[m].double_sided;
        }
        if (vis) {
            yes[tri.x] = kYesDrawn | (below_near(a.z) ? kYesBehind : 0);
            yes[tri.y] = kYesDrawn | (below_near(c1.z) ? kYesBehind : 0);
            yes[tri.z] = kYesDrawn | (below_near(c2.z) ? kYesBehind : 0);
        }
    };
    // a warp takes 32 * kFlagsPer consecutive triangles, lane + 32 u each,
    // and issues all their loads before the tests
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t stride = gridDim.x * blockDim.x * kFlagsPer;
    for (uint32_t g0 = ((blockIdx.x * blockDim.x + threadIdx.x) & ~31u) * kFlagsPer + lane; g0 < total; g0 += stride) {
        const uint32_t glast = g0 + 32 * (kFlagsPer - 1);
        if (g0 < lo || g0 >= hi)
            bind(g0);
        if (glast < hi && glast < total) {
            const uint32_t l = g0 - lo;
            uint4 t[kFlagsPer];
#pragma unroll
            for (int u = 0; u < kFlagsPer; u++)
                t[u] = tris[l + 32 * u];
            V3 a[kFlagsPer], c1[kFlagsPer], c2[kFlagsPer];
#pragma unroll
            for (int u = 0; u < kFlagsPer; u++) {
                a[u] = ld3(ndc, t[u].x);
                c1[u] = ld3(ndc, t[u].y);
                c2[u] = ld3(ndc, t[u].z);
            }
#pragma unroll
            for (int u = 0; u < kFlagsPer; u++)
                flag(t[u], a[u], c1[u], c2[u]);
        } else {
            for (uint32_t g = g0; g <= glast && g < total; g += 32) {
                if (g < lo || g >= hi)
                    bind(g);
                const uint4 tri = tris[g - lo];
                flag(tri, ld3(ndc, tri.x), ld3(ndc, tri.y), ld3(ndc, tri.z));
            }
        }
    }
}

// frustum_to_viewport (viewport.cpp:123-129) of a flagged vertex
__device__ __forceinline__ V3 load_vp(const ItemDev &it, uint32_t g)
{
    const float4 n = it.ndc[g];
    return mk3(it.v.vm00 * n.x + it.v.vm03, it.v.vm11 * n.y + it.v.vm13, n.z);
}

// The lanes' counts added to their items' counters (item_counters[2 item +
// which]: 0 drawn triangles, 1 fragments), one atomic per distinct item.
// Every lane of the warp calls it.
__device__ __forceinline__ void item_add(const BatchDev *b, int which, uint32_t item, unsigned long long n, bool valid)
{
    const unsigned act = __ballot_sync(0xFFFFFFFFu, valid && n);
    if (!(valid && n))
        return;
    if (__any_sync(act, n >> 26)) { // the sum of 32 might not fit
        atomicAdd(b->item_counters + 2 * (size_t)item + which, n);
        return;
    }
    const unsigned grp = __match_any_sync(act, item);
    const uint32_t sum = __reduce_add_sync(grp, (uint32_t)n);
    if ((threadIdx.x & 31) == __ffs(grp) - 1)
        atomicAdd(b->item_counters + 2 * (size_t)item + which, (unsigned long long)sum);
}

// The record slot of a near-clipped batch triangle: flags = kRecClip.
__device__ __forceinline__ void mark_clip(const BatchDev *b, uint32_t r)
{
    if (in_bounds(r < b->list_cap, CHK_REC, r))
        reinterpret_cast<uint32_t *>(b->recs + r)[kRecFlagsWord] = kRecClip;
}

// 32-bit batch counter w (C_*)
__device__ __forceinline__ uint32_t *counter32(const BatchDev *b, int w)
{
    return reinterpret_cast<uint32_t *>(b->counters) + w;
}

// Reserve n0 walk-list and n1 clip-list entries with one atomic: the two
// 32-bit counters C_LIST and C_CLIP are the halves of one 64-bit counter word
// (a list holds fewer than 2^31 entries, so the low half never carries).
// Returns the previous values (C_LIST low, C_CLIP high).
static_assert(C_LIST % 2 == 0 && C_CLIP == C_LIST + 1, "list counters share a 64-bit word");
__device__ __forceinline__ unsigned long long reserve_lists(const BatchDev *b, uint32_t n0, uint32_t n1)
{
    if (!(n0 | n1))
        return 0ull;
    return atomicAdd(b->counters + C_LIST / 2, ((unsigned long long)n1 << 32) | n0);
}

// The rows a triangle whose screen y range is lo_y .. hi_y walks in a view of
// rows y .. y_end are more than kTallRows (the first test settles most).
__device__ __forceinline__ bool tall_rows(float lo_y, float hi_y, int y, int y_end)
{
    if (hi_y - lo_y < kTallRows - 0.5f)
        return false;
    const int a = max(f2i(ceilf(lo_y)), y), z = min(f2i(ceilf(hi_y)), y_end);
    return z > a && z - a > kTallRows;
}

// A triangle of one row (its screen y range lo_y .. hi_y holds one whole
// number) whose row's span holds no pixel: no whole number between the
// crossings of the row with its two edges that span it, widened by `eps` to
// both sides.  Each crossing here is within 2^-20 mx (mx the largest |x|, below
// 2^20) of the exact one (differences, the hardware reciprocal, products and
// the sum: 7 roundings of 2^-24 of at most 2 mx), the reference's x within
// 18 * 2^-24 mx of it (its start has 6 roundings), and eps is at least 33 *
// 2^-23 mx, nearly twice both.  Such triangles are two fifths of the walk list
// of a batch of small views (2.8 M of 7.1 M of the 64 views of 200 spheres; a
// fifth of the 1080p frame's) and cost the walk a set-up each: 64 views, walk 470
// -> 347 us for 46 us more of geometry.  (k_compact does not ask: on terrains of
// 512 x 512 cells at 256 x 256 to 1920 x 1080 it took 0.7 us and saved none.)
__device__ __forceinline__ bool row_empty(float x0, float y0, float x1, float y1, float x2, float y2, float lo_y,
                                          float hi_y, float mx, float eps)
{
    const float y = ceilf(lo_y);
    if (!(y + 1.0f >= hi_y && mx < 0x1p20f && fabsf(y) < 0x1p20f))
        return false;
    float lo = INFINITY, hi = -INFINITY, sum = 0.0f;
    auto edge = [&](float xa, float ya, float xb, float yb) {
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(yb - ya));
        const float x = xa + (y - ya) * (xb - xa) * r;
        if ((ya <= y) != (yb <= y)) {
            lo = fminf(lo, x);
            hi = fmaxf(hi, x);
            sum = sum + x;
        }
    };
    edge(x0, y0, x1, y1);
    edge(x1, y1, x2, y2);
    edge(x2, y2, x0, y0);
    return fabsf(sum) < 0x1p22f && ceilf(lo - eps) >= hi + eps; // (the sum is NaN or infinite where a crossing is)
}

// Batch triangles r of the lanes that ask for it into the tall list, one
// atomic per warp.  Every lane of the warp calls it.
__device__ __forceinline__ void list_tall(const BatchDev *b, bool want, uint32_t r)
{
    const unsigned m = __ballot_sync(0xFFFFFFFFu, want);
    if (!m)
        return;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    uint32_t at = 0;
    if (lane == leader)
        at = atomicAdd(counter32(b, C_TALL), (uint32_t)__popc(m));
    at = __shfl_sync(0xFFFFFFFFu, at, leader) + __popc(m & ((1u << lane) - 1u));
    if (want && in_bounds(at < b->list_cap, CHK_REC, at))
        b->tall[at] = r;
}

// Drawable triangles (all three vertices flagged, renderer.cpp:248-253) into
// the walk list, or the tall list when they have many rows; triangles crossing
// the near plane go to their own list and are marked in their records.  One
// global atomic per list per block.
constexpr int kCompactBlock = 512;
__global__ void __launch_bounds__(kCompactBlock) k_compact(const BatchDev *b)
{
    __shared__ uint32_t cnt[2], base[2];
    const int lane = threadIdx.x & 31;
    int item = -1;
    uint32_t lo = 0, hi = 0;
    const uint4 *tris = nullptr;
    const uint8_t *yes = nullptr;
    const uint8_t *psmall = nullptr; // a mixed scene: primitives of the fused pass
    const uint32_t total = b->total_gtri;
    // every thread of the block runs the same number of iterations (barriers inside)
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t g0 = blockIdx.x * blockDim.x; g0 < total; g0 += stride) {
        if (threadIdx.x < 2)
            cnt[threadIdx.x] = 0;
        __syncthreads();
        const uint32_t g = g0 + threadIdx.x;
        int list = -1; // 0 walk list, 1 clip list, 2 tall list
        bool counted = false; // reached fill_triangle_2's set-up
        uint32_t t = 0;
        if (g < total) {
            if (g < lo || g >= hi) {
                item = find_item(b->g_tri_base, b->n_items, g);
                lo = __ldg(b->g_tri_base + item);
                hi = __ldg(b->g_tri_base + item + 1);
                const ItemDev &it = b->items[item];
                tris = it.s.tris;
                yes = it.yes;
                psmall = it.s.psmall;
            }
            t = g - lo;
            const uint4 tri = tris[t];
            const bool general = !psmall || !psmall[tri.w];
            const uint32_t ya = general ? yes[tri.x] : 0u, yb = general ? yes[tri.y] : 0u,
                           yc = general ? yes[tri.z] : 0u;
            if (ya & yb & yc & kYesDrawn) {
                // fill_triangle's cases (renderer.cpp:281-318): the smallest z' decides
                list = ((ya | yb | yc) & kYesBehind) ? 1 : 0;
                if (list == 0) {
                    const ItemDev &it = b->items[item];
                    const float y0 = it.v.vm11 * it.ndc[tri.x].y + it.v.vm13;
                    const float y1 = it.v.vm11 * it.ndc[tri.y].y + it.v.vm13;
                    const float y2 = it.v.vm11 * it.ndc[tri.z].y + it.v.vm13;
                    const float lo_y = fminf(y0, fminf(y1, y2)), hi_y = fmaxf(y0, fmaxf(y1, y2));
                    // (finite or infinite y only: with a NaN the set-up's sort decides)
                    if (y0 == y0 && y1 == y1 && y2 == y2) {
                        if (f2i(ceilf(lo_y)) == f2i(ceilf(hi_y))) {
                            // fill_triangle_2 draws nothing when its first and last
                            // rows coincide (ceil of the smallest and largest y,
                            // renderer.cpp:389-391): such a triangle never reaches
                            // the set-up or the walk, and is not counted
                            list = -1;
                        } else {
                            counted = true;
                            // No pixel column either: every row's span [ceil(xl),
                            // ceil(xr)) is empty when the triangle's x range, widened
                            // by the walk's rounding, holds no integer boundary.  The
                            // walked edge positions are the exact ones (inside the
                            // range) up to the start's rounding and one rounding per
                            // row step, (rows + 17) u (max |x| + eps) in all (u =
                            // 2^-24); eps is over twice that.  Such a triangle reached
                            // the set-up in the reference, so it is counted as drawn,
                            // but it covers no pixel and gets no set-up record.
                            const float x0 = it.v.vm00 * it.ndc[tri.x].x + it.v.vm03;
                            const float x1 = it.v.vm00 * it.ndc[tri.y].x + it.v.vm03;
                            const float x2 = it.v.vm00 * it.ndc[tri.z].x + it.v.vm03;
                            const float mx = fmaxf(fabsf(x0), fmaxf(fabsf(x1), fabsf(x2)));
                            const float rows = ceilf(hi_y) - ceilf(lo_y);
                            const float eps = (rows + 32.0f) * 0x1p-23f * (mx + 1.0f);
                            const float lo_x = fminf(x0, fminf(x1, x2)) - eps;
                            const float hi_x = fmaxf(x0, fmaxf(x1, x2)) + eps;
                            if (ceilf(lo_x) == ceilf(hi_x)) {
                                list = -1;
                                if (b->slot_flags)
                                    b->slot_flags[2 * t] = 1;
                            } else if (tall_rows(lo_y, hi_y, it.v.y, it.v.y + it.v.h)) {
                                list = 2;
                            }
                        }
                    }
                }
            }
        }
        list_tall(b, list == 2, list == 2 ? __ldg(b->tri_base + item) + t : 0u);
        item_add(b, 0, (uint32_t)item, 1u, counted);
        uint32_t pos = 0;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const unsigned m = __ballot_sync(0xFFFFFFFFu, list == k);
            if (!m)
                continue;
            uint32_t wb = 0;
            if (lane == 0)
                wb = atomicAdd(&cnt[k], (uint32_t)__popc(m));
            wb = __shfl_sync(0xFFFFFFFFu, wb, 0);
            if (list == k)
                pos = wb + __popc(m & ((1u << lane) - 1u));
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const unsigned long long old = reserve_lists(b, cnt[0], cnt[1]);
            base[0] = (uint32_t)old;
            base[1] = (uint32_t)(old >> 32);
        }
        __syncthreads();
        if (list == 1) {
            const uint32_t j = base[1] + pos;
            if (j < b->clip_cap)
                b->clip[b->clip_cap - 1 - j] = make_uint2(t, (uint32_t)item); // filled from the end
            mark_clip(b, __ldg(b->tri_base + item) + t);
        } else if (list == 0) {
            const uint32_t j = base[0] + pos;
            if (j < b->list_cap)
                b->list[j] = make_uint2(__ldg(b->tri_base + item) + t, (uint32_t)item);
        }
        __syncthreads();
    }
}

// The geometry of fused scenes (every primitive within kFuseVerts vertices
// and kFuseTris triangles): one warp per primitive runs k_vertex, k_flags and
// k_compact on it with the vertex positions and flags in shared memory.  A
// primitive owns its vertices (no two vertex ranges overlap), so its
// triangles are the only ones that flag them (renderer.cpp:86-185 flags a
// node's primitives before any is drawn, and each primitive's vertices are
// its own), and its compaction needs nothing from other warps.
//
// Items are taken in groups that read the same vertex data (the views of one
// scene in the batch; the reference likewise transforms a scene to world
// space once for all the viewports of a render call, renderer.hpp:27-34).  A
// block takes kGeomWarps consecutive primitives and up to kGeomItems items of
// a group and runs each warp's primitive for each of the items: the primitive's first 64 triangles stay in registers as local vertex
// indices and its world positions are read again per item (from L1 after the
// first).  Per item the warp records its walk-list and clip-list decisions as
// ballot masks, and at the end one global atomic reserves both lists for all
// the unit's items and warps (reserve_lists).
//
// The pass is bound by instruction issue and by the latency of its load chain
// (about 1,000 instructions a primitive and view before, at 49 % issue).  So a
// vertex is one 16-byte word of shared memory with its flags in w, the
// unit's cameras are staged once for the block, a primitive without a
// visible triangle (about half of a closed mesh's) stops after the visibility
// test, and projected vertices are stored only for primitives with an entry
// in a list, which are all that the later passes read: 64 views 691 -> 573 us,
// of 200 spheres.  Blocks are of four warps, as all of a block wait for its
// slowest primitive and for the reservation, and the first item's world
// positions are copied beside the triangles: 1080p 27.5 -> 25.5 us, 64 views
// 595 -> 579 us (with row_empty); eight warps 27.2 and 583, two 27.0 and 602.
// The grid is eight waves of blocks: 64 views take 643 us in two, 679 in one.
constexpr int kGeomVerts = 2;           // vertices of a lane with loads in flight (four spill registers: 683 us for 573)
constexpr int kGeomTG = kFuseTris / 32; // groups of 32 triangles
constexpr int kGeomBlocks = 32 / kGeomWarps; // resident blocks per SM the pass is compiled for
// words of an item's camera in shared memory: view and projection rows 0-2, then
enum { GV_VM00 = 24, GV_VM03, GV_VM11, GV_VM13, GV_Y, GV_YEND, GV_ITEM, GV_TRI, kGeomViewWords };
static_assert(kGeomViewWords == 32, "a warp stages an item's camera, a word per lane");
struct GeomShared {
    float4 pos[kGeomWarps][kFuseVerts];             // x, y, z' and flags of each vertex (for the item in hand)
    float view[kGeomItems][kGeomViewWords];         // the unit's cameras
    float4 *ndc[kGeomItems];                        // ... and projected vertices
    uint32_t walk[kGeomItems][kGeomWarps][kGeomTG]; // per 32 triangles: ballot of the walk list
    uint32_t clip[kGeomItems][kGeomWarps][kGeomTG]; // ... of the clip list
    uint32_t cnt[kGeomItems * kGeomWarps];          // entries: walk list | clip list << 16
    uint32_t off[kGeomItems * kGeomWarps];          // ... of the items and warps before
    uint32_t nx[kGeomItems * kGeomWarps];           // triangles that reach fill_triangle_2's set-up
    uint32_t base[2];                               // the block's first position in each list
};
static_assert(kFuseVerts <= 256, "local vertex indices are bytes");
static_assert(kGeomItems * kGeomWarps <= 64 && kGeomWarps % 2 == 0 && 64 * kFuseTris < 65536,
              "a warp scans the counts, two of one item a lane, in 16 bits");
constexpr size_t kGeomSmem = sizeof(GeomShared);

// The local vertex indices of triangle t of a fused primitive (a | b << 8 | c << 16).
__device__ __forceinline__ uint32_t geom_tri(const uint4 *tris, uint4 gq, uint32_t t)
{
    const uint4 tri = tris[gq.z + t];
    in_bounds(tri.x - gq.x < gq.y && tri.y - gq.x < gq.y && tri.z - gq.x < gq.y, CHK_LOCAL, gq.z + t);
    return (tri.x - gq.x) | ((tri.y - gq.x) << 8) | ((tri.z - gq.x) << 16);
}

// Bit i (i < n <= 8) set when item grp_items[v0 + i] sees none of the
// triangles of primitive q (box pbox[2 q], pbox[2 q + 1]): the box is in the
// region z' > 0 and in one beyond a side plane (ViewDev::cull).  Lane 4 i + r
// tests item i's side r; the mask is the same in every lane.  A box with a
// NaN is in no region.
__device__ __forceinline__ uint32_t geom_unseen(const BatchDev *b, const float4 *pbox, uint32_t q, uint32_t v0,
                                                uint32_t n, uint32_t lane)
{
    bool out = false;
    if ((lane >> 2) < n) {
        const float4 *cull = &b->items[__ldg(b->grp_items + v0 + (lane >> 2))].v.cull[0][0];
        const float4 bc = pbox[2 * q], bh = pbox[2 * q + 1];
        const float4 ba = make_float4(fabsf(bc.x) + bh.x, fabsf(bc.y) + bh.y, fabsf(bc.z) + bh.z, 0.0f);
        out = cull_region(cull + 2 * (lane & 3), bc, bh, ba) < 0.0f && cull_region(cull + 8, bc, bh, ba) < 0.0f;
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, out);
    uint32_t u = 0;
#pragma unroll
    for (int i = 0; i < kGeomItems; i++)
        u |= ((m >> (4 * i)) & 15u) ? 1u << i : 0u;
    return u;
}

__global__ void __launch_bounds__(kGeomWarps * 32, kGeomBlocks) k_geom(const BatchDev *b)
{
    extern __shared__ __align__(16) unsigned char geom_smem[];
    GeomShared &S = *reinterpret_cast<GeomShared *>(geom_smem);
    const int warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    float4 *pos = S.pos[warp];
    uint32_t c_lo = 0, c_hi = 0, g_lo = 0, g_n = 0, passes = 1, i_lo = 0xFFFFFFFFu;
    int nv = 0;
    const uint32_t total = b->total_chunks;
    // every thread of the block runs the same iterations (barriers inside)
    for (uint32_t c = blockIdx.x; c < total; c += gridDim.x) {
        __syncthreads(); // the previous unit's masks and cameras are read
        if (c < c_lo || c >= c_hi) {
            const int g = find_item(b->grp_chunk_base, b->n_groups, c);
            c_lo = __ldg(b->grp_chunk_base + g);
            c_hi = __ldg(b->grp_chunk_base + g + 1);
            g_lo = __ldg(b->grp_item_base + g);
            g_n = __ldg(b->grp_item_base + g + 1) - g_lo;
            passes = (g_n + kGeomItems - 1) / kGeomItems;
        }
        const uint32_t chunk = passes == 1 ? c - c_lo : (c - c_lo) / passes, first = (c - c_lo - chunk * passes) * kGeomItems;
        if (g_lo + first != i_lo) {
            i_lo = g_lo + first;
            nv = (int)min((uint32_t)kGeomItems, g_n - first);
            // a warp stages an item's camera at a time
            for (int sv = warp; sv < nv; sv += kGeomWarps) {
                const uint32_t item = __ldg(b->grp_items + i_lo + sv);
                const ItemDev &it = b->items[item];
                float x;
                if (lane < 12)
                    x = it.v.view[lane];
                else if (lane < 24)
                    x = it.v.proj[lane - 12];
                else if (lane < GV_Y)
                    x = (&it.v.vm00)[lane - GV_VM00];
                else
                    x = __uint_as_float(lane == GV_Y      ? (uint32_t)it.v.y
                                        : lane == GV_YEND ? (uint32_t)(it.v.y + it.v.h)
                                        : lane == GV_ITEM ? item
                                                          : __ldg(b->tri_base + item));
                S.view[sv][lane] = x;
                if (lane == 0)
                    S.ndc[sv] = it.ndc;
            }
        }
        const SceneDev &sc = b->items[__ldg(b->grp_items + i_lo)].s; // vertex data shared by the group
        const uint32_t q = chunk * kGeomWarps + warp;                  // this warp's primitive
        const bool has = q < sc.n_prims && (!sc.psmall || sc.psmall[q]); // (a mixed scene's larger ones: general passes)
        uint4 gq = make_uint4(0u, 0u, 0u, 0u); // first vertex, vertex count, first triangle, triangle count
        bool ds = false;
        uint32_t tr0 = 0, tr1 = 0; // the first 64 triangles, local vertex indices
        uint32_t unseen = 0;       // bit vi: item vi sees none of the primitive
        const float4 *wpos = sc.wpos;
        const uint4 *tris = sc.tris;
        if (has) {
            gq = sc.pgeo[q];
            gq.y = min(gq.y, kFuseVerts); // (a fused scene's primitives are within both limits)
            gq.w = min(gq.w, kFuseTris);
            if (sc.pbox)
                unseen = geom_unseen(b, sc.pbox, q, i_lo, (uint32_t)nv, lane);
            // the first item's world positions go where its vertices will be
            // (each lane transforms those it copied)
            if (!(unseen & 1u))
                for (uint32_t i = lane; i < gq.y; i += 32)
                    cp_async<16>(pos + i, wpos + gq.x + i);
            if (lane < gq.w)
                tr0 = geom_tri(tris, gq, lane);
            if (lane + 32 < gq.w)
                tr1 = geom_tri(tris, gq, lane + 32);
            ds = sc.pshade[q].double_sided != 0;
        }
        wpos += gq.x;
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads(); // the cameras are staged
        for (int vi = 0; vi < nv; vi++) {
            uint32_t entries = 0, nx = 0;
            if (has && !((unseen >> vi) & 1u)) {
                const float *vw = S.view[vi];
                __syncwarp(); // the previous item's reads of pos are done
                // world_to_camera_or_frustum (vertex_shaders.hpp:35-52), as
                // k_vertex; kGeomVerts vertices a lane and round, their loads issued first
                bool behind = false;
                {
                    float m[24];
#pragma unroll
                    for (int k = 0; k < 6; k++)
                        reinterpret_cast<float4 *>(m)[k] = reinterpret_cast<const float4 *>(vw)[k];
                    for (uint32_t i0 = 0; i0 < gq.y; i0 += 32 * kGeomVerts) {
                        float4 w[kGeomVerts];
#pragma unroll
                        for (int k = 0; k < kGeomVerts; k++)
                            if (i0 + lane + 32 * k < gq.y)
                                w[k] = vi ? wpos[i0 + lane + 32 * k] : pos[i0 + lane + 32 * k];
#pragma unroll
                        for (int k = 0; k < kGeomVerts; k++) {
                            const uint32_t i = i0 + lane + 32 * k;
                            if (i < gq.y) {
                                V3 v = transform3(mk3(w[k].x, w[k].y, w[k].z), m);
                                v = transform3(v, m + 12);
                                if (v.z != 0.0f) {
                                    v.x = v.x / fabsf(v.z);
                                    v.y = v.y / fabsf(v.z);
                                }
                                const bool near = below_near(v.z);
                                behind |= near;
                                pos[i] = make_float4(v.x, v.y, v.z, __uint_as_float(near ? kYesBehind : 0u));
                            }
                        }
                    }
                }
                behind = __any_sync(0xFFFFFFFFu, behind);
                // visibility flags (renderer.cpp:86-185), as k_flags; every
                // store to a vertex writes the same value
                bool any = false;
                for (uint32_t t = lane; t < gq.w; t += 32) {
                    const uint32_t tp = t < 32 ? tr0 : (t < 64 ? tr1 : geom_tri(tris, gq, t));
                    float4 &pa = pos[tp & 0xFFu], &pb = pos[(tp >> 8) & 0xFFu], &pc = pos[tp >> 16];
                    const float4 fa = pa, fb = pb, fc = pc;
                    const V3 a = mk3(fa.x, fa.y, fa.z), c1 = mk3(fb.x, fb.y, fb.z), c2 = mk3(fc.x, fc.y, fc.z);
                    if (inside_frustum(a, c1, c2) && (ds || cross_z_positive(sub3(c1, a), sub3(c2, a)))) {
                        any = true;
                        pa.w = __uint_as_float(__float_as_uint(fa.w) | kYesDrawn);
                        pb.w = __uint_as_float(__float_as_uint(fb.w) | kYesDrawn);
                        pc.w = __uint_as_float(__float_as_uint(fc.w) | kYesDrawn);
                    }
                }
                if (__any_sync(0xFFFFFFFFu, any)) {
                    __syncwarp();
                    // the compaction's decisions, as k_compact
                    const float vm00 = vw[GV_VM00], vm03 = vw[GV_VM03], vm11 = vw[GV_VM11], vm13 = vw[GV_VM13];
                    bool listed = false;
                    for (uint32_t t0 = 0; t0 < gq.w; t0 += 32) {
                        const uint32_t t = t0 + lane;
                        int d = 0; // 0 none, 1 walk list, 2 clip list, 3 no pixel column, 4 tall list
                        bool counted = false;
                        if (t < gq.w) {
                            const uint32_t tp = t < 32 ? tr0 : (t < 64 ? tr1 : geom_tri(tris, gq, t));
                            const float4 fa = pos[tp & 0xFFu], fb = pos[(tp >> 8) & 0xFFu], fc = pos[tp >> 16];
                            const uint32_t ya = __float_as_uint(fa.w), yb = __float_as_uint(fb.w),
                                           yc = __float_as_uint(fc.w);
                            if (ya & yb & yc & kYesDrawn) {
                                if (behind && ((ya | yb | yc) & kYesBehind)) {
                                    d = 2;
                                } else {
                                    d = 1;
                                    const float y0 = vm11 * fa.y + vm13, y1 = vm11 * fb.y + vm13,
                                                y2 = vm11 * fc.y + vm13;
                                    const float lo_y = fminf(y0, fminf(y1, y2)), hi_y = fmaxf(y0, fmaxf(y1, y2));
                                    if (y0 == y0 && y1 == y1 && y2 == y2) {
                                        if (f2i(ceilf(lo_y)) == f2i(ceilf(hi_y))) {
                                            d = 0; // no row
                                        } else {
                                            counted = true;
                                            const float x0 = vm00 * fa.x + vm03, x1 = vm00 * fb.x + vm03,
                                                        x2 = vm00 * fc.x + vm03;
                                            const float mx = fmaxf(fabsf(x0), fmaxf(fabsf(x1), fabsf(x2)));
                                            const float rows = ceilf(hi_y) - ceilf(lo_y);
                                            const float eps = (rows + 32.0f) * 0x1p-23f * (mx + 1.0f);
                                            const float lo_x = fminf(x0, fminf(x1, x2)) - eps;
                                            const float hi_x = fmaxf(x0, fmaxf(x1, x2)) + eps;
                                            if (ceilf(lo_x) == ceilf(hi_x) ||
                                                row_empty(x0, y0, x1, y1, x2, y2, lo_y, hi_y, mx, eps)) {
                                                d = 3; // no pixel column, or no pixel in its row
                                                if (b->slot_flags)
                                                    b->slot_flags[2 * (gq.z + t)] = 1;
                                            } else if (tall_rows(lo_y, hi_y, __float_as_int(vw[GV_Y]),
                                                                 __float_as_int(vw[GV_YEND]))) {
                                                d = 4;
                                            }
                                        }
                                    }
                                }
                            }
                        }
                        if (__any_sync(0xFFFFFFFFu, d == 4)) {
                            list_tall(b, d == 4, __float_as_uint(vw[GV_TRI]) + gq.z + t);
                            listed = true;
                        }
                        const unsigned m1 = __ballot_sync(0xFFFFFFFFu, d == 1);
                        const unsigned m2 = behind ? __ballot_sync(0xFFFFFFFFu, d == 2) : 0u;
                        const unsigned m3 = __ballot_sync(0xFFFFFFFFu, counted);
                        if (lane == 0) {
                            S.walk[vi][warp][t0 >> 5] = m1;
                            S.clip[vi][warp][t0 >> 5] = m2;
                        }
                        entries += __popc(m1) | (__popc(m2) << 16);
                        nx += __popc(m3);
                    }
                    // the later passes read the projected vertices of listed
                    // triangles alone
                    if (listed || entries) {
                        float4 *ndc = S.ndc[vi] + gq.x;
                        for (uint32_t i = lane; i < gq.y; i += 32)
                            if (in_bounds(gq.x + i < sc.n_vertices, CHK_NDC, gq.x + i))
                                ndc[i] = pos[i];
                    }
                }
            }
            if (lane == 0) {
                S.cnt[vi * kGeomWarps + warp] = entries;
                S.nx[vi * kGeomWarps + warp] = nx;
            }
        }
        __syncthreads();
        if (warp == 0) {
            // first positions per item and warp (two a lane), one reservation
            const int k = 2 * (int)lane;
            const uint32_t a = k < nv * kGeomWarps ? S.cnt[k] : 0u, z = k < nv * kGeomWarps ? S.cnt[k + 1] : 0u;
            uint32_t incl = a + z;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                if ((int)lane >= d)
                    incl += u;
            }
            if (k < kGeomItems * kGeomWarps) {
                S.off[k] = incl - a - z;
                S.off[k + 1] = incl - z;
            }
            if (lane == 31) {
                const unsigned long long old = reserve_lists(b, incl & 0xFFFFu, incl >> 16);
                S.base[0] = (uint32_t)old;
                S.base[1] = (uint32_t)(old >> 32);
            }
            // the items' drawn triangles (kGeomWarps / 2 lanes hold one item's)
            uint32_t x = k < nv * kGeomWarps ? S.nx[k] + S.nx[k + 1] : 0u;
#pragma unroll
            for (int d = 1; d < kGeomWarps / 2; d <<= 1)
                x += __shfl_xor_sync(0xFFFFFFFFu, x, d);
            if (lane % (kGeomWarps / 2) == 0 && x)
                atomicAdd(b->item_counters + 2 * (size_t)__float_as_uint(S.view[lane / (kGeomWarps / 2)][GV_ITEM]),
                          (unsigned long long)x);
        }
        __syncthreads();
        if (has) {
            const uint32_t list_cap = b->list_cap, base0 = S.base[0], base1 = S.base[1];
            uint2 *list = b->list;
            for (int vi = 0; vi < nv; vi++) {
                const uint32_t n = S.cnt[vi * kGeomWarps + warp];
                if (!n)
                    continue;
                const uint32_t off = S.off[vi * kGeomWarps + warp];
                const uint32_t item = __float_as_uint(S.view[vi][GV_ITEM]), tlo = __float_as_uint(S.view[vi][GV_TRI]);
                uint32_t o0 = base0 + (off & 0xFFFFu);
                for (uint32_t t0 = 0; t0 < gq.w; t0 += 32) {
                    const unsigned m1 = S.walk[vi][warp][t0 >> 5];
                    const uint32_t j = o0 + __popc(m1 & below);
                    if (((m1 >> lane) & 1u) && j < list_cap)
                        list[j] = make_uint2(tlo + gq.z + t0 + lane, item);
                    o0 += __popc(m1);
                }
                if (!(n >> 16))
                    continue;
                uint32_t o1 = base1 + (off >> 16);
                for (uint32_t t0 = 0; t0 < gq.w; t0 += 32) {
                    const unsigned m2 = S.clip[vi][warp][t0 >> 5];
                    if ((m2 >> lane) & 1u) {
                        const uint32_t j = o1 + __popc(m2 & below);
                        if (j < b->clip_cap)
                            b->clip[b->clip_cap - 1 - j] = make_uint2(gq.z + t0 + lane, item); // from the end
                        mark_clip(b, tlo + gq.z + t0 + lane);
                    }
                    o1 += __popc(m2);
                }
            }
        }
    }
}

// ------------------------------------------------------------ triangle walk --

// fill_triangle's sort of the vertex pointers by z' descending
// (renderer.cpp:264-279), on values; pa/pb/pc track which input landed where.
__device__ __forceinline__ bool sort_z_desc(V3 &a, V3 &b, V3 &c, int &pa, int &pb, int &pc)
{
    bool inv = false;
    V3 t;
    int q;
    if (b.z > a.z) { t = a; a = b; b = t; q = pa; pa = pb; pb = q; inv = !inv; }
    if (c.z > b.z) { t = b; b = c; c = t; q = pb; pb = pc; pc = q; inv = !inv; }
    if (b.z > a.z) { t = a; a = b; b = t; q = pa; pa = pb; pb = q; inv = !inv; }
    return inv;
}

// fill_triangle_2's sort by screen y ascending (renderer.cpp:375-387)
__device__ __forceinline__ void sort_y_asc(V3 &a, V3 &b, V3 &c, int &pa, int &pb, int &pc)
{
    V3 t;
    int q;
    if (b.y < a.y) { t = a; a = b; b = t; q = pa; pa = pb; pb = q; }
    if (c.y < b.y) { t = b; b = c; c = t; q = pb; pb = pc; pc = q; }
    if (b.y < a.y) { t = a; a = b; b = t; q = pa; pa = pb; pb = q; }
}

// fill_half_triangle row loop (renderer.cpp:462-558): per row the span
// [x1, x2) clipped to the viewport goes to the visitor, then both edges step.
template <class Vis>
__device__ __forceinline__ void walk_half(const ViewDev &v, int y, int y_end, Side &Ls, Side &Rs, uint32_t bits,
                                          Vis &vis)
{
    for (; y < y_end && vis.active(); y++) {
        int x1 = f2i(ceilf(Ls.x));
        if (x1 < v.x)
            x1 = v.x;
        int x2 = f2i(ceilf(Rs.x));
        if (x2 > v.x + v.w)
            x2 = v.x + v.w;
        if (x1 < x2)
            vis.span(y, x1, x2, Ls, Rs, bits);
        Ls.x = Ls.x + Ls.ratio;
        Rs.x = Rs.x + Rs.ratio;
        Ls.it.step();
        Rs.it.step();
    }
}

// fill_triangle_2 (src/render/renderer.cpp:361-460) on screen positions, in
// the vertex order fill_triangle passes them: edge setup and both halves.
// Span bits: kBitLower for the lower half, kBitLLR for long_line_on_right.
template <class Vis>
__device__ __forceinline__ void walk_sub(const ViewDev &v, V3 a, V3 b, V3 c, Vis &vis)
{
    int pa = 0, pb = 1, pc = 2;
    sort_y_asc(a, b, c, pa, pb, pc);
    const V3 v0 = a, v1 = b, v2 = c;
    const int y0 = f2i(ceilf(v0.y));
    const int y1 = f2i(ceilf(v1.y));
    const int y2 = f2i(ceilf(v2.y));
    if (y0 == y2)
        return;
    Side lng, sht;
    lng.ratio = (v2.x - v0.x) / (v2.y - v0.y);
    lng.it.init_self(v2.y - v0.y, v0.z, v2.z);
    if (y0 < v.y) {
        lng.it.displace((float)v.y - v0.y);
        lng.x = v0.x + lng.ratio * ((float)v.y - v0.y);
    } else {
        lng.it.displace((float)y0 - v0.y);
        lng.x = v0.x + lng.ratio * ((float)y0 - v0.y);
    }
    vis.drawn();
    if (y1 >= v.y) {
        sht.ratio = (v1.x - v0.x) / (v1.y - v0.y);
        sht.it.init_self(v1.y - v0.y, v0.z, v1.z);
        const int y = y0 > v.y ? y0 : v.y;
        const int y_end = y1 < v.y + v.h ? y1 : v.y + v.h;
        sht.it.displace((float)y - v0.y);
        sht.x = v0.x + sht.ratio * ((float)y - v0.y);
        const bool llr = lng.ratio > sht.ratio;
        const uint32_t bits = llr ? kBitLLR : 0u;
        if (llr)
            walk_half(v, y, y_end, sht, lng, bits, vis);
        else
            walk_half(v, y, y_end, lng, sht, bits, vis);
    }
    if (y1 < v.y + v.h) {
        sht.ratio = (v2.x - v1.x) / (v2.y - v1.y);
        sht.it.init_self(v2.y - v1.y, v1.z, v2.z);
        const int y = y1 > v.y ? y1 : v.y;
        const int y_end = y2 < v.y + v.h ? y2 : v.y + v.h;
        sht.it.displace((float)y - v1.y);
        sht.x = v1.x + sht.ratio * ((float)y - v1.y);
        const bool llr = lng.ratio < sht.ratio;
        const uint32_t bits = kBitLower | (llr ? kBitLLR : 0u);
        if (llr)
            walk_half(v, y, y_end, sht, lng, bits, vis);
        else
            walk_half(v, y, y_end, lng, sht, bits, vis);
    }
}

// The per-pixel loop of fill_half_triangle for one span: qpixel set up over
// the span (renderer.cpp:476-480) and stepped per pixel (:486).  `op(x, z,
// progress)` gets each pixel nearer than the near plane and the clear depth.
template <class Op>
__device__ __forceinline__ void span_pixels(int x1, int x2, const Side &Ls, const Side &Rs, Op &op)
{
    Interp q;
    q.init_self(Rs.x - Ls.x, Ls.it.value(), Rs.it.value());
    q.displace((float)x1 - Ls.x);
    for (; x1 < x2; x1++, q.step()) {
        const float z = q.value();
        if (below_near(z)) // (double)z <= 0.001
            continue;
        if (__float_as_uint(z) >= kMaxZBits)
            continue; // z >= the cleared depth never passes
        op(x1, z, q.alpha);
    }
}

__device__ __forceinline__ unsigned long long make_key(float z, uint32_t slot)
{
    return ((unsigned long long)__float_as_uint(z) << 32) | slot;
}

// The span bins: span i's interpolator, edge values and place as three
// 16-byte words in arrays of span_cap entries, then its item, with
// kSpanRecorded when the shade cannot replay its pixels and their winners are
// recorded (a capture span: its first pool entry).
constexpr uint32_t kSpanRecorded = 1u << 31; // (a batch has at most 4,096 items)
struct SpanRec {
    float4 q; // the qpixel interpolator of fill_half_triangle after its displacement to x1: top, tstep, bottom, bstep
    float4 e; // ... v0, dv; the row's edge progress progL, progR (prepare_for_scanline)
    uint4 at; // slot, y | kBitLower | kBitLLR, x1, x2
};
__device__ __forceinline__ void store_span(const BatchDev *b, uint32_t i, uint32_t item, uint32_t slot, uint32_t y_bits,
                                           int x1, int x2, const Interp &q, float pl, float pr)
{
    float4 *p = static_cast<float4 *>(b->spans) + i;
    const size_t cap = b->span_cap;
    p[0] = make_float4(q.top, q.tstep, q.bottom, q.bstep);
    p[cap] = make_float4(q.v0, q.dv, pl, pr);
    reinterpret_cast<uint4 *>(p)[2 * cap] = make_uint4(slot, y_bits, (uint32_t)x1, (uint32_t)x2);
    reinterpret_cast<uint32_t *>(static_cast<float4 *>(b->spans) + 3 * cap)[i] = item;
}
__device__ __forceinline__ SpanRec load_span(const BatchDev *b, uint32_t i)
{
    const float4 *p = static_cast<const float4 *>(b->spans) + i;
    const size_t cap = b->span_cap;
    return SpanRec{p[0], p[cap], reinterpret_cast<const uint4 *>(p)[2 * cap]};
}
__device__ __forceinline__ uint32_t load_span_item(const BatchDev *b, uint32_t i)
{
    return reinterpret_cast<const uint32_t *>(static_cast<const float4 *>(b->spans) + 3 * (size_t)b->span_cap)[i];
}

// Bin a long span: the qpixel state after its displacement to x1.
__device__ __forceinline__ bool bin_span(const BatchDev *b, uint32_t item, uint32_t slot, int y, int x1, int x2,
                                         const Side &Ls, const Side &Rs, uint32_t bits)
{
    const uint32_t i = atomicAdd(counter32(b, C_SPANS), 1u);
    if (i >= b->span_cap) {
        atomicExch(counter32(b, C_OVERFLOW), 1u);
        return false;
    }
    Interp q;
    q.init_self(Rs.x - Ls.x, Ls.it.value(), Rs.it.value());
    q.displace((float)x1 - Ls.x);
    store_span(b, i, item | kSpanRecorded, slot, (uint32_t)y | bits, x1, x2, q, Ls.it.alpha, Rs.it.alpha);
    return true;
}

struct DepthVisitor {
    const BatchDev *b;
    const ItemDev *it;
    uint32_t item;
    uint32_t slot;
    int inline_span;
    uint32_t drawn_n;
    unsigned long long fragments;

    __device__ __forceinline__ bool active() const { return true; }
    __device__ __forceinline__ void drawn()
    {
        drawn_n++;
        if (b->slot_flags)
            b->slot_flags[slot] = 1;
    }
    __device__ __forceinline__ void span(int y, int x1, int x2, const Side &Ls, const Side &Rs, uint32_t bits)
    {
        fragments += (unsigned long long)(x2 - x1);
        if (x2 - x1 > inline_span && bin_span(b, item, slot, y, x1, x2, Ls, Rs, bits))
            return;
        const ViewDev &v = it->v;
        unsigned long long *row = it->key + ((long long)(y - v.y) * v.w - v.x);
        const uint32_t sl = slot;
        auto op = [&](int x, float z, float) {
            if (in_bounds(x >= v.x && x < v.x + v.w && y >= v.y && y < v.y + v.h, CHK_KEY,
                          (unsigned long long)(uint32_t)y << 32 | (uint32_t)x))
                key_min(row + x, make_key(z, sl));
        };
        span_pixels(x1, x2, Ls, Rs, op);
    }
};

// Records the winner's progress values (the overflow fallback and the
// near-clip triangles, whose winners the shade kernel does not replay).
struct WinnerVisitor {
    const ItemDev *it;
    uint32_t slot;
    int inline_span;
    bool all_spans; // bins overflowed: record every span here

    __device__ __forceinline__ bool active() const { return true; }
    __device__ __forceinline__ void drawn() {}
    __device__ __forceinline__ void span(int y, int x1, int x2, const Side &Ls, const Side &Rs, uint32_t bits)
    {
        if (x2 - x1 > inline_span && !all_spans)
            return; // recorded by the winner span kernel from the bins
        const ViewDev &v = it->v;
        const long long base = (long long)(y - v.y) * v.w - v.x;
        const unsigned long long *row = it->key + base;
        float4 *rec = it->prec + base;
        const uint32_t sl = slot;
        const float pl = Ls.it.alpha, pr = Rs.it.alpha;
        auto op = [&](int x, float z, float progress) {
            if (row[x] == make_key(z, sl))
                rec[x] = make_float4(progress, pl, pr, __uint_as_float(bits));
        };
        span_pixels(x1, x2, Ls, Rs, op);
    }
};

// ------------------------------------------------------- row-parallel walk --
//
// The walk of fill_triangle_2 is serial only along its edges: row k needs the
// edges after k steps (x += ratio, top += tstep, bottom += bstep, renderer.cpp
// :553-556), and each span needs the qpixel chain from its left end.  The
// steps are float additions, so any thread can reach row k by repeating them
// from the set-up; the divisions of a row (edge progress, span set-up) and of
// its pixels then run wherever that row is.  A warp takes 32 triangles, each
// lane makes its triangle's set-up (the TriRec), and the warp's rows are
// dealt out across the lanes.  Triangles with more than kTallRows rows have
// a list of their own (the geometry passes know their rows): each is walked
// by a whole warp, 32 rows at a time, and every one of its spans goes to the
// long-span kernels.
//
// The set-up is made here, in the shared memory that the rows are read from.
// As a pass of its own it spent its time on the stores of its records (51 MB
// on the 1080p frame) and the walk on reading them back; made here, only the
// records of triangles with fragments are stored, for the shade, as whole
// lines: set-up and walk 49.0 -> 37.4 us (1080p), 854 -> 682 us (64 views).
// Both were bound by latency and issue (20 % and 48 % of the issue slots).

constexpr int kWalkWarps = 4;
#ifndef SGL_WALK_MIN_BLOCKS
#define SGL_WALK_MIN_BLOCKS 5 // resident blocks per SM the walk is compiled for (caps its registers: 4, 5, 6 and 7
                              // blocks walk the 1080p frame in 39.5, 37.4, 40.2 and 51.5 us)
#endif
// Per-warp set-ups in shared memory, S[field][lane]: fields 0-31 are the
// words of TriRec in order; the row is padded to 33 words so that both the
// per-lane and the per-record accesses are free of bank conflicts.
enum {
    F_LX, F_LT, F_LB, F_LR, F_LTS, F_LBS, // long edge: x, top, bottom, ratio, tstep, bstep
    F_Z0, F_Z2,
    F_UX, F_UT, F_UB, F_UR, F_UTS, F_UBS, // upper short edge
    F_SLOT, F_ITEM,
    F_DX, F_DT, F_DB, F_DR, F_DTS, F_DBS, // lower short edge
    F_YL, F_ND,
    F_Z1, F_YS, F_NU, F_FLAGS, F_G0, F_G1, F_G2, F_PRIM,
    F_FRAGS, // fragments of the lane's triangle (shared atomics of the lanes walking its rows)
    F_INCL,  // inclusive prefix of the rows dealt out, per lane
    F_VX, F_VW, F_KEY, // the item's view: x, w and its key pointer (two words), in batches of several views
    kWalkFields = F_KEY + 2
};
constexpr int kWalkPitch = 33;
static_assert(F_PRIM == 31 && sizeof(TriRec) == 32 * sizeof(uint32_t), "shared set-up fields follow TriRec");
static_assert(offsetof(TriRec, slot) == 4 * F_SLOT && offsetof(TriRec, dx) == 4 * F_DX &&
                  offsetof(TriRec, flags) == 4 * F_FLAGS,
              "shared set-up fields follow TriRec");

// interpolator_g<1>::InitSelf then DisplaceStartingPoint (interpolator.hpp:
// 60-84), with 1/z1 and 1/z2 passed in (the same divisions, made once per
// vertex).  The progress of the displaced state is not formed here: every
// reader divides top by bottom itself, as step() would have.
__device__ __forceinline__ void edge_init(float dist, float rz1, float rz2, float move, float &top, float &bot,
                                          float &ts, float &bs)
{
    const float alphastep = 1.0f / dist;
    bot = rz1;
    top = 0.0f;
    top = top * bot;
    ts = (1.0f * rz2 - top) * alphastep;
    bs = (rz2 - bot) * alphastep;
    top = top + ts * move;
    bot = bot + bs * move;
}

// f2i(ceilf(x)) in one conversion where it is in range.
__device__ __forceinline__ int ceil_i(float x) { return fabsf(x) < 2147483520.0f ? __float2int_ru(x) : f2i(ceilf(x)); }

// The inputs of one walked row: both edges at the half's first row with
// their constants, the steps to take, the row and its span bits.
struct RowIn {
    float lx, lt, lb, lr, lts, lbs, lz, ldv; // long edge; value() = lz + ldv * progress
    float sx, st, sb, sr, sts, sbs, sz, sdv; // short edge of the row's half
    int y, ls, ss;
    bool llr;
    uint32_t bits;
};

// Row k of a set-up (k < n_u: upper half): `lg` is the long edge (x, top,
// bottom, ratio, tstep, bstep), `sh` the short edge of the row's half.
__device__ __forceinline__ void row_in(RowIn &r, int k, const float lg[6], const float sh[6], float z0, float z1,
                                       float z2, int y_s, int y_l, int n_u, uint32_t flags)
{
    r.lx = lg[0]; r.lt = lg[1]; r.lb = lg[2]; r.lr = lg[3]; r.lts = lg[4]; r.lbs = lg[5];
    r.sx = sh[0]; r.st = sh[1]; r.sb = sh[2]; r.sr = sh[3]; r.sts = sh[4]; r.sbs = sh[5];
    r.lz = z0;
    r.ldv = z2 - z0;
    r.ls = k;
    if (k < n_u) {
        r.sz = z0;
        r.sdv = z1 - z0;
        r.y = y_s + k;
        r.ss = k;
        r.llr = (flags & kRecLLRUpper) != 0u;
        r.bits = r.llr ? kBitLLR : 0u;
    } else {
        r.sz = z1;
        r.sdv = z2 - z1;
        r.y = y_l + (k - n_u);
        r.ss = k - n_u;
        r.llr = (flags & kRecLLRLower) != 0u;
        r.bits = kBitLower | (r.llr ? kBitLLR : 0u);
    }
}

// A row after its steps: the span [x1, x2) clipped to the viewport
// (renderer.cpp:466-472) and the left and right edge (Ls, Rs).
struct RowSpan {
    int x1, x2;
    float Lx, Lt, Lb, Lz, Ldv, Rx, Rt, Rb, Rz, Rdv;
};

__device__ __forceinline__ void row_span(RowIn &r, int vx, int vw, RowSpan &o)
{
    for (int k = 0; k < r.ls; k++) {
        r.lx = r.lx + r.lr;
        r.lt = r.lt + r.lts;
        r.lb = r.lb + r.lbs;
    }
    for (int k = 0; k < r.ss; k++) {
        r.sx = r.sx + r.sr;
        r.st = r.st + r.sts;
        r.sb = r.sb + r.sbs;
    }
    if (r.llr) {
        o.Lx = r.sx; o.Lt = r.st; o.Lb = r.sb; o.Lz = r.sz; o.Ldv = r.sdv;
        o.Rx = r.lx; o.Rt = r.lt; o.Rb = r.lb; o.Rz = r.lz; o.Rdv = r.ldv;
    } else {
        o.Lx = r.lx; o.Lt = r.lt; o.Lb = r.lb; o.Lz = r.lz; o.Ldv = r.ldv;
        o.Rx = r.sx; o.Rt = r.st; o.Rb = r.sb; o.Rz = r.sz; o.Rdv = r.sdv;
    }
    o.x1 = ceil_i(o.Lx);
    if (o.x1 < vx)
        o.x1 = vx;
    o.x2 = ceil_i(o.Rx);
    if (o.x2 > vx + vw)
        o.x2 = vx + vw;
}

// The qpixel interpolator of a span after its displacement to x1, and the
// progress of both edges (renderer.cpp:474-480, prepare_for_scanline).  With
// `steps` > 0 the interpolator is also stepped that many pixels: top and
// bottom take every addition of the reference's per-pixel steps, and alpha,
// which each step recomputes from them alone, is divided out once at the end
// (the same value as the last step's).
__device__ __forceinline__ void span_interp(const RowSpan &o, Interp &q, float &pl, float &pr, int steps = 0)
{
    pl = o.Lt / o.Lb;
    pr = o.Rt / o.Rb;
    q.init_self(o.Rx - o.Lx, o.Lz + o.Ldv * pl, o.Rz + o.Rdv * pr);
    const float move = (float)o.x1 - o.Lx;
    q.top = q.top + q.tstep * move; // Interp::displace without its division
    q.bottom = q.bottom + q.bstep * move;
    for (int k = 0; k < steps; k++) {
        q.top = q.top + q.tstep;
        q.bottom = q.bottom + q.bstep;
    }
    q.alpha = q.top / q.bottom;
}

// Bins the spans of the lanes that ask for it (one atomic per warp).  Every
// lane of the warp calls it; returns whether this lane's span was binned.
__device__ __forceinline__ bool bin_span_warp(const BatchDev *b, bool want, uint32_t item, uint32_t slot, int y,
                                              const RowSpan &o, const Interp &q, float pl, float pr, uint32_t bits)
{
    const unsigned m = __ballot_sync(0xFFFFFFFFu, want);
    if (!m)
        return false;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if (lane == leader)
        base = atomicAdd(counter32(b, C_SPANS), (uint32_t)__popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    if (!want)
        return false;
    const uint32_t i = base + __popc(m & ((1u << lane) - 1u));
    if (i >= b->span_cap) {
        atomicExch(counter32(b, C_OVERFLOW), 1u);
        return false;
    }
    store_span(b, i, item, slot, (uint32_t)y | bits, o.x1, o.x2, q, pl, pr);
    return true;
}

// One span's pixels into the depth keys (the opaque branch of
// fill_half_triangle, renderer.cpp:484-499, as a key reduction).
// The view fields the walk needs of an item.
struct WalkView {
    int x, w;
    long long origin;         // of the view's pixels, y * w + x of its top left: pixel (X, Y) is Y * w + X - origin
    unsigned long long *key;  // depth keys less `origin`
    __device__ __forceinline__ void load(const ItemDev &it)
    {
        x = it.v.x;
        w = it.v.w;
        origin = (long long)it.v.y * w + x;
        key = it.key - origin;
    }
};

__device__ __forceinline__ bool key_in_view(const BatchDev *b, uint32_t item, int x, int y)
{
#ifdef SGL_BOUNDS_CHECK
    const ViewDev &v = b->items[item].v;
    return in_bounds(x >= v.x && x < v.x + v.w && y >= v.y && y < v.y + v.h, CHK_KEY,
                     (unsigned long long)(uint32_t)y << 32 | (uint32_t)x);
#else
    return true;
#endif
}

// One pixel of a span at the interpolator's top and bottom.
__device__ __forceinline__ void pixel_depth(const BatchDev *b, uint32_t item, unsigned long long *row, int x, int y,
                                            uint32_t slot, float top, float bottom, float v0, float dv)
{
    const float z = v0 + dv * (top / bottom);
    if (!below_near(z) && __float_as_uint(z) < kMaxZBits && key_in_view(b, item, x, y))
        key_min(row + x, make_key(z, slot));
}

__device__ __forceinline__ void span_depth(const BatchDev *b, const WalkView &v, uint32_t item, int y, uint32_t slot,
                                           int x1, int x2, const Interp &q)
{
    unsigned long long *row = v.key + (long long)y * v.w;
    float top = q.top, bottom = q.bottom;
    for (int x = x1; x < x2; x++) {
        pixel_depth(b, item, row, x, y, slot, top, bottom, q.v0, q.dv);
        top = top + q.tstep;
        bottom = bottom + q.bstep;
    }
}

// A span's pixels by L lanes, the `sub`-th of them pixels x1 + sub, + L, ...:
// each lane repeats the chain's additions up to its own pixels.  (Eight lanes
// where there are spans enough: the additions a lane repeats are 8 per 8 pixels
// instead of 32 per 32, so that four spans side by side take a third of the
// instructions of one after another.)
constexpr int kSpanLanes = 8;
template <int L, class Op>
__device__ __forceinline__ void span_by(int x1, int x2, int sub, float top, float tstep, float bottom, float bstep,
                                        Op &&op)
{
#pragma unroll
    for (int bit = L / 2; bit; bit >>= 1)
        if (sub & bit) {
#pragma unroll
            for (int k = 0; k < bit; k++) {
                top = top + tstep;
                bottom = bottom + bstep;
            }
        }
    for (int x = x1 + sub; x < x2; x += L) {
        op(x, top, bottom);
#pragma unroll
        for (int k = 0; k < L; k++) {
            top = top + tstep;
            bottom = bottom + bstep;
        }
    }
}

// The spans of the lanes that ask for it, four at a time by eight lanes each.
// Every lane of the warp calls it.
__device__ __forceinline__ void spans_depth_warp(const BatchDev *b, bool want, const WalkView &v, uint32_t item, int y,
                                                 uint32_t slot, int x1, int x2, const Interp &q)
{
    unsigned m = __ballot_sync(0xFFFFFFFFu, want);
    if (!m)
        return;
    const int lane = threadIdx.x & 31, sub = lane & (kSpanLanes - 1);
    unsigned long long *row = v.key + (long long)y * v.w;
    while (m) {
        unsigned mine = m; // this lane's span: the (lane / 8)-th of those left
#pragma unroll
        for (int k = 0; k < 32 / kSpanLanes - 1; k++)
            if (lane >= kSpanLanes * (k + 1))
                mine &= mine - 1;
        const int src = mine ? __ffs(mine) - 1 : 0;
        const float top = __shfl_sync(0xFFFFFFFFu, q.top, src), tstep = __shfl_sync(0xFFFFFFFFu, q.tstep, src);
        const float bottom = __shfl_sync(0xFFFFFFFFu, q.bottom, src), bstep = __shfl_sync(0xFFFFFFFFu, q.bstep, src);
        const float v0 = __shfl_sync(0xFFFFFFFFu, q.v0, src), dv = __shfl_sync(0xFFFFFFFFu, q.dv, src);
        const int xa = __shfl_sync(0xFFFFFFFFu, x1, src), xb = __shfl_sync(0xFFFFFFFFu, x2, src);
        const int ys = __shfl_sync(0xFFFFFFFFu, y, src);
        const uint32_t sl = __shfl_sync(0xFFFFFFFFu, slot, src), si = __shfl_sync(0xFFFFFFFFu, item, src);
        unsigned long long *rs = reinterpret_cast<unsigned long long *>(
            __shfl_sync(0xFFFFFFFFu, reinterpret_cast<unsigned long long>(row), src));
        if (mine)
            span_by<kSpanLanes>(xa, xb, sub, top, tstep, bottom, bstep, [&](int x, float t, float bt) {
                pixel_depth(b, si, rs, x, ys, sl, t, bt, v0, dv);
            });
#pragma unroll
        for (int k = 0; k < 32 / kSpanLanes; k++)
            m &= m - 1;
    }
}

// Fragment capture of a view with transparency layers (a layered batch has
// one item): the pool counter and its per-pixel chains.
__device__ __forceinline__ unsigned long long *frag_counter(const BatchDev *b)
{
    return b->counters + C_FRAGS / 2;
}

// One span's fragments stored from pool entry `at` on, each with its view
// pixel in the `next` field (k_link chains them afterwards); pixels skipped
// at the near plane are stored as holes (kFragEnd).
__device__ __forceinline__ void span_frags(const BatchDev *b, uint32_t row_px, uint32_t slot, int x1, int x2,
                                           Interp q, float pl, float pr, uint32_t bits, uint32_t at)
{
    Frag *pool = b->frags;
    const float fb = __uint_as_float(bits);
    for (int x = x1; x < x2; x++, q.step()) {
        const float z = q.value();
        const bool keep = !below_near(z) && __float_as_uint(z) < kMaxZBits;
        const uint32_t k = at + (uint32_t)(x - x1);
        reinterpret_cast<float4 *>(pool + k)[0] = make_float4(q.alpha, pl, pr, fb);
        reinterpret_cast<uint4 *>(pool + k)[1] =
            make_uint4(__float_as_uint(z), slot, keep ? row_px + (uint32_t)x : kFragEnd, 0u);
    }
}

typedef uint32_t WalkRow[kWalkPitch];

__device__ __forceinline__ float smf(const WalkRow *S, int f, int o) { return __uint_as_float(S[f][o]); }

__device__ __forceinline__ void smem_row_in(RowIn &r, const WalkRow *S, int o, int k)
{
    const int n_u = (int)S[F_NU][o];
    const int sf = k < n_u ? F_UX : F_DX;
    float lg[6], sh[6];
#pragma unroll
    for (int f = 0; f < 6; f++) {
        lg[f] = smf(S, F_LX + f, o);
        sh[f] = smf(S, sf + f, o);
    }
    row_in(r, k, lg, sh, smf(S, F_Z0, o), smf(S, F_Z1, o), smf(S, F_Z2, o), (int)S[F_YS][o], (int)S[F_YL][o], n_u,
           S[F_FLAGS][o]);
}

// Set-up of triangle t (vertices `tri`, projected n0, n1, n2) of `item`:
// fill_triangle's z sort (renderer.cpp:264-279), fill_triangle_2's y sort,
// edges and halves (:375-460), into column `c` of the warp's set-ups.  A
// triangle that does not reach scanline set-up (y0 == y2) has no rows.
// Returns whether it did and was not counted by the geometry pass (a NaN y).
__device__ __forceinline__ bool tri_setup(const BatchDev *b, const ViewDev &v, uint32_t item, uint32_t t, uint4 tri,
                                          float4 n0, float4 n1, float4 n2, uint32_t extra_flags, WalkRow *S, int c)
{
    auto put = [&](int f, float x) { S[f][c] = __float_as_uint(x); };
    auto vp = [&](float4 n) { return mk3(v.vm00 * n.x + v.vm03, v.vm11 * n.y + v.vm13, n.z); }; // as load_vp
    V3 a = vp(n0), c1 = vp(n1), c2 = vp(n2);
    const bool ffv = cross_z_negative(sub3(c1, a), sub3(c2, a));
    int pa = 0, pb = 1, pc = 2;
    // (the order by z' decides only where the order by y leaves a tie)
    if (!(a.y < c1.y || a.y > c1.y) || !(a.y < c2.y || a.y > c2.y) || !(c1.y < c2.y || c1.y > c2.y))
        sort_z_desc(a, c1, c2, pa, pb, pc);
    sort_y_asc(a, c1, c2, pa, pb, pc);
    const V3 v0 = a, v1 = c1, v2 = c2;
    const int y0 = ceil_i(v0.y), y1 = ceil_i(v1.y), y2 = ceil_i(v2.y);
    S[F_ITEM][c] = item;
    S[F_SLOT][c] = 2 * t;
    S[F_NU][c] = 0;
    S[F_ND][c] = 0;
    S[F_FLAGS][c] = extra_flags;
    if (y0 == y2)
        return false;
    if (b->slot_flags)
        b->slot_flags[2 * t] = 1;
    S[F_G0][c] = pa == 0 ? tri.x : (pa == 1 ? tri.y : tri.z);
    S[F_G1][c] = pb == 0 ? tri.x : (pb == 1 ? tri.y : tri.z);
    S[F_G2][c] = pc == 0 ? tri.x : (pc == 1 ? tri.y : tri.z);
    S[F_PRIM][c] = tri.w;
    put(F_Z0, v0.z);
    put(F_Z1, v1.z);
    put(F_Z2, v2.z);
    const float rz0 = 1.0f / v0.z, rz1 = 1.0f / v1.z, rz2 = 1.0f / v2.z;
    const int ys = y0 < v.y ? v.y : y0;
    S[F_YS][c] = (uint32_t)ys;
    const float lmove = (float)ys - v0.y;
    const float lratio = (v2.x - v0.x) / (v2.y - v0.y);
    float top, bot, ts, bs;
    auto edge = [&](int f, float x, float ratio) {
        put(f, x);
        put(f + 1, top);
        put(f + 2, bot);
        put(f + 3, ratio);
        put(f + 4, ts);
        put(f + 5, bs);
    };
    edge_init(v2.y - v0.y, rz0, rz2, lmove, top, bot, ts, bs);
    edge(F_LX, v0.x + lratio * lmove, lratio);
    uint32_t flags = extra_flags | (ffv ? kRecFFV : 0u);
    if (y1 >= v.y) {
        const float ratio = (v1.x - v0.x) / (v1.y - v0.y);
        const int yend = y1 < v.y + v.h ? y1 : v.y + v.h;
        edge_init(v1.y - v0.y, rz0, rz1, lmove, top, bot, ts, bs);
        edge(F_UX, v0.x + ratio * lmove, ratio);
        if (lratio > ratio)
            flags |= kRecLLRUpper;
        S[F_NU][c] = yend > ys ? (uint32_t)(yend - ys) : 0u;
    }
    if (y1 < v.y + v.h) {
        const float ratio = (v2.x - v1.x) / (v2.y - v1.y);
        const int y = y1 > v.y ? y1 : v.y;
        const int yend = y2 < v.y + v.h ? y2 : v.y + v.h;
        const float move = (float)y - v1.y;
        edge_init(v2.y - v1.y, rz1, rz2, move, top, bot, ts, bs);
        edge(F_DX, v1.x + ratio * move, ratio);
        if (lratio < ratio)
            flags |= kRecLLRLower;
        S[F_YL][c] = (uint32_t)y;
        S[F_ND][c] = yend > y ? (uint32_t)(yend - y) : 0u;
    }
    S[F_FLAGS][c] = flags;
    return v0.y != v0.y || v1.y != v1.y || v2.y != v2.y;
}

// Wide spans per round of rows that the walk keeps: the bins' atomic costs a
// round trip, which more spans share (walk of a terrain's 1080p frame: 32.6,
// 30.8, 30.0, 27.6 and 28.2 us for 0, 1, 2, 4 and 8).
constexpr int kWarpSpans = 4;
// One row of triangle `slot` of `item` (view v) on this lane; every lane of
// the warp calls it (act = this lane has a row).  A lane walks its span alone
// up to inline_span pixels; wider ones are walked by eight lanes each, here
// or (when there are many, they are wider than kReplaySpan, or the triangle is
// tall) in the long-span kernels.  Returns the row's fragments.  With FRAGS (a view with transparency
// layers) every fragment is stored instead: the warp reserves its lanes'
// fragments with one atomic per round of rows, spans beyond inline_span are
// binned, and a binned span carries its first pool entry in place of its item.
template <bool FRAGS>
__device__ __forceinline__ int walk_row(const BatchDev *b, const WalkView &v, int inline_span, uint32_t item,
                                        uint32_t slot, RowIn &r, bool act, bool bin_all)
{
    RowSpan sp;
    sp.x1 = sp.x2 = 0;
    if (act)
        row_span(r, v.x, v.w, sp);
    const bool has = act && sp.x1 < sp.x2;
    Interp q;
    float pl = 0.0f, pr = 0.0f;
    if (has)
        span_interp(sp, q, pl, pr);
    const int len = has ? sp.x2 - sp.x1 : 0;
    if constexpr (FRAGS) {
        const int lane = threadIdx.x & 31;
        const uint32_t n = (uint32_t)len;
        uint32_t incl = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d)
                incl += u;
        }
        unsigned long long base = 0;
        if (lane == 31 && incl)
            base = atomicAdd(frag_counter(b), (unsigned long long)incl);
        base = __shfl_sync(0xFFFFFFFFu, base, 31);
        const unsigned long long at = base + incl - n;
        const bool fits = at + n <= (unsigned long long)b->frag_cap; // else counted only: the view is redone
        const bool want = has && (bin_all || len > inline_span);
        if (!bin_span_warp(b, want && fits, (uint32_t)at, slot, r.y, sp, q, pl, pr, r.bits) && has && fits)
            span_frags(b, (uint32_t)((long long)r.y * v.w - v.origin), slot, sp.x1, sp.x2, q, pl, pr, r.bits,
                       (uint32_t)at);
    } else {
        // Wide spans: up to kWarpSpans of a round are walked by this warp at
        // once, more (or longer than the shade replays) go to the bins, whose
        // atomic's round trip and second kernel they are worth.
        bool wide = has && (bin_all || len > inline_span);
        const unsigned m = __ballot_sync(0xFFFFFFFFu, wide);
        const bool record = bin_all || len > kReplaySpan;
        const bool want = wide && (record || __popc(m) > kWarpSpans);
        if (bin_span_warp(b, want, record ? item | kSpanRecorded : item, slot, r.y, sp, q, pl, pr, r.bits))
            wide = false;
        else if (has && !wide)
            span_depth(b, v, item, r.y, slot, sp.x1, sp.x2, q);
        spans_depth_warp(b, wide, v, item, r.y, slot, sp.x1, sp.x2, q);
    }
    return len;
}

// n <= 31 repeated additions x += d of three chains; every lane takes its own
// n.  The additions of a chain are all alike, so a lane's n of them can be
// taken in any grouping: 16, 8, 4, 2, 1 by the bits of n.
__device__ __forceinline__ void step3(float &x, float &t, float &b, float dx, float dt, float db, int n)
{
#pragma unroll
    for (int bit = 16; bit; bit >>= 1)
        if (n & bit) {
#pragma unroll
            for (int k = 0; k < bit; k++) {
                x = x + dx;
                t = t + dt;
                b = b + db;
            }
        }
}
// The same additions n times by every lane alike.
__device__ __forceinline__ void advance3(float &x, float &t, float &b, float dx, float dt, float db, int n)
{
#pragma unroll 8
    for (int k = 0; k < n; k++) {
        x = x + dx;
        t = t + dt;
        b = b + db;
    }
}

// A tall triangle (set-up in column 0 of S), walked by `share` warps, this one
// the `sub`-th: each takes 32 rows in share * 32, its lanes a row each, from
// the state of the first of the 32, to which the warp repeats the additions
// from its last.  Every span is binned.  Returns this lane's fragments.
template <bool FRAGS>
__device__ __forceinline__ unsigned long long walk_tall(const BatchDev *b, const WalkRow *S, int sub, int share)
{
    const int lane = threadIdx.x & 31;
    const int n_u = (int)S[F_NU][0], n = n_u + (int)S[F_ND][0];
    const uint32_t slot = S[F_SLOT][0], item = S[F_ITEM][0];
    unsigned long long frags = 0;
    WalkView v;
    v.load(b->items[item]);
    float lx = smf(S, F_LX, 0), lt = smf(S, F_LT, 0), lb = smf(S, F_LB, 0);
    // the short edge in hand (the upper one until row n_u) and the row of its state
    bool upper = n_u > 0;
    int sf = upper ? F_UX : F_DX, at = 0;
    float sx = smf(S, sf, 0), st = smf(S, sf + 1, 0), sb = smf(S, sf + 2, 0);
    for (int r0 = 32 * sub; r0 < n; r0 += 32 * share) {
        advance3(lx, lt, lb, smf(S, F_LR, 0), smf(S, F_LTS, 0), smf(S, F_LBS, 0), r0 - at);
        if (upper && r0 >= n_u) { // on to the lower edge, from its first row
            upper = false;
            sf = F_DX;
            sx = smf(S, sf, 0), st = smf(S, sf + 1, 0), sb = smf(S, sf + 2, 0);
            at = n_u;
        }
        advance3(sx, st, sb, smf(S, sf + 3, 0), smf(S, sf + 4, 0), smf(S, sf + 5, 0), r0 - at);
        at = r0;
        const int k = r0 + lane;
        const bool act = k < n;
        RowIn r;
        smem_row_in(r, S, 0, act ? k : 0);
        r.lx = lx; r.lt = lt; r.lb = lb;
        step3(r.lx, r.lt, r.lb, r.lr, r.lts, r.lbs, lane);
        // rows of the half in hand continue its chain; a row beyond it starts
        // on the lower short edge (smem_row_in's state)
        const bool cont = (k < n_u) == upper;
        if (cont) {
            r.sx = sx; r.st = st; r.sb = sb;
        }
        step3(r.sx, r.st, r.sb, r.sr, r.sts, r.sbs, cont ? lane : k - n_u);
        r.ls = 0;
        r.ss = 0;
        frags += (unsigned long long)walk_row<FRAGS>(b, v, kSpanLanes, item, slot, r, act, true);
    }
    return frags;
}

// the rare depth walks, defined with the near-clip code below
__device__ __noinline__ void walk_clip_depth(const BatchDev *b);
template <bool FRAGS>
__device__ __noinline__ void walk_tall_all(const BatchDev *b, WalkRow *S);

// One warp's shared memory: the set-ups of the group in hand, and what is
// copied in ahead for the next groups: list entries (three ahead), their
// triangles (two ahead) and the triangles' projected vertices (one ahead).
// Each lane reads only what it copied itself, except the entries' batch
// triangles.
struct WalkShared {
    WalkRow S[kWalkFields];
    __align__(16) float4 ndc[3][32];
    uint4 tri[2][32];
    uint2 entry[4][32];
};

// Fragments of the lanes' triangles added to the block's sums of the first
// kWalkItems items, or (when the warp holds another, or a triangle of 2^26
// fragments) to the items' counters: one addition per item of the warp.  Few
// items' counters meet all the warps that walk the same view; more items'
// spread over as many addresses (32 views of 512 x 384, of 200 spheres, take
// 752 us in all with the sums and 812 with counters alone; from 64 views on the
// walk is as long either way, 364 and 366 us, and sums of 256 or 1,024 items
// change nothing at 96 to 4,096 views).  Additions by lane were what cost:
// 96 views 1,950 us, 548 now.  Every lane of the warp calls it.
constexpr int kWalkItems = 64;
__device__ __forceinline__ void block_add(const BatchDev *b, uint32_t *sums, uint32_t item, uint32_t n)
{
    if (__any_sync(0xFFFFFFFFu, n && ((n >> 26) || item >= (uint32_t)kWalkItems))) {
        item_add(b, 1, item, n, true);
        return;
    }
    const unsigned act = __ballot_sync(0xFFFFFFFFu, n != 0u);
    if (!n)
        return;
    const unsigned grp = __match_any_sync(act, item);
    const uint32_t sum = __reduce_add_sync(grp, n);
    if ((threadIdx.x & 31) == __ffs(grp) - 1 && atomicAdd(sums + item, sum) >> 31) {
        const uint32_t all = atomicExch(sums + item, 0u); // (well before it overflows)
        atomicAdd(b->item_counters + 2 * (size_t)item + 1, (unsigned long long)all);
    }
}

// Set-up and depth walk of the drawable triangles wholly in front of the near
// plane (fill_triangle's normal case, renderer.cpp:281-285: one sub-triangle,
// slot 2t).  Each warp takes groups of 32 list entries (warp-strided): a lane
// makes its entry's set-up in shared memory, the group's rows are dealt across
// the lanes, and the set-ups with fragments are stored as whole records for
// the shade.  FRAGS: the fragment capture of a layered view (the near-clipped
// triangles are captured by k_frags).
template <bool FRAGS, bool STRIDED>
__global__ void __launch_bounds__(kWalkWarps * 32, SGL_WALK_MIN_BLOCKS) k_walk(const BatchDev *b)
{
    __shared__ WalkShared shared[kWalkWarps];
    __shared__ uint32_t item_frags[STRIDED ? 1 : kWalkItems]; // fragments of the batch's first items, walked by this block
    WalkShared &W = shared[threadIdx.x >> 5];
    WalkRow *S = W.S;
    const int lane = threadIdx.x & 31;
    const uint32_t n_raw = *counter32(b, C_LIST);
    const uint32_t n = n_raw < b->list_cap ? n_raw : b->list_cap;
    const uint32_t n_groups = (n + 31) / 32;
    // STRIDED (a batch of one view, kSeqOne): group g holds entries
    // g + j * n_groups (j < 32), so every group samples the whole list and the
    // large triangles of nearby primitives, which sit together in list order,
    // spread over all groups and warps (1080p frame: 41.7 -> 30.3 us).  In a
    // batch of several views a strided group would mix the views' triangles,
    // whose view parameters each row then reloads (serving: 5.5 -> 12.3 us
    // per request), so there group g holds entries 32 g + j.
    auto index = [&](uint32_t g) -> uint32_t { return STRIDED ? g + (uint32_t)lane * n_groups : 32 * g + (uint32_t)lane; };
    // the copies of group g's entries, triangles and vertices (q: the group's
    // place in this warp's sequence, which picks the buffers)
    auto fetch_entry = [&](uint32_t g, int q) {
        if (g < n_groups && index(g) < n)
            cp_async<8>(&W.entry[q & 3][lane], b->list + index(g));
    };
    auto fetch_tri = [&](uint32_t g, int q) {
        if (g < n_groups && index(g) < n) {
            const uint2 e = W.entry[q & 3][lane];
            cp_async<16>(&W.tri[q & 1][lane], b->items[e.y].s.tris + (e.x - __ldg(b->tri_base + e.y)));
        }
    };
    auto fetch_ndc = [&](uint32_t g, int q) {
        if (g < n_groups && index(g) < n) {
            const ItemDev &it = b->items[W.entry[q & 3][lane].y];
            const uint4 t = W.tri[q & 1][lane];
            if (in_bounds(t.x < it.s.n_vertices && t.y < it.s.n_vertices && t.z < it.s.n_vertices, CHK_NDC, t.x)) {
                cp_async<16>(&W.ndc[0][lane], it.ndc + t.x);
                cp_async<16>(&W.ndc[1][lane], it.ndc + t.y);
                cp_async<16>(&W.ndc[2][lane], it.ndc + t.z);
            }
        }
    };
    const int summed = min(b->n_items, kWalkItems);
    if (!STRIDED) {
        for (int i = (int)threadIdx.x; i < summed; i += kWalkWarps * 32)
            item_frags[i] = 0u;
        __syncthreads();
    }
    const int inline_span = b->inline_span;
    WalkView view{};
    if (STRIDED)
        view.load(b->items[0]);
    unsigned long long fragments = 0; // STRIDED: of this lane's triangles
    // Warps take groups g, g + G, g + 2G, ... (G warps in the grid; work
    // queues were measured slower: 41 -> 48 us on the 1080p frame).
    const uint32_t G = (gridDim.x * blockDim.x) >> 5;
    uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (g < n_groups) {
        fetch_entry(g, 0);
        fetch_entry(g + G, 1);
        fetch_entry(g + 2 * G, 2);
        cp_async_commit();
        cp_async_wait<0>();
        fetch_tri(g, 0);
        fetch_tri(g + G, 1);
        cp_async_commit();
        cp_async_wait<0>();
        fetch_ndc(g, 0);
        cp_async_commit();
    }
    for (int q = 0; g < n_groups; q++, g += G) {
        cp_async_wait<0>();
        const bool valid = index(g) < n;
        bool late = false;
        S[F_FRAGS][lane] = 0;
        if (valid) {
            const uint2 e = W.entry[q & 3][lane];
            const float4 n0 = W.ndc[0][lane], n1 = W.ndc[1][lane], n2 = W.ndc[2][lane];
            if (!STRIDED) {
                WalkView v;
                v.load(b->items[e.y]);
                const unsigned long long kp = reinterpret_cast<unsigned long long>(v.key);
                S[F_VX][lane] = (uint32_t)v.x;
                S[F_VW][lane] = (uint32_t)v.w;
                S[F_KEY][lane] = (uint32_t)kp;
                S[F_KEY + 1][lane] = (uint32_t)(kp >> 32);
            }
            late = tri_setup(b, b->items[e.y].v, e.y, e.x - __ldg(b->tri_base + e.y), W.tri[q & 1][lane], n0, n1, n2,
                              0u, S, lane);
        } else {
            S[F_NU][lane] = 0;
            S[F_ND][lane] = 0;
        }
        // rows dealt across the lanes
        int incl = (int)(S[F_NU][lane] + S[F_ND][lane]);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d)
                incl += u;
        }
        S[F_INCL][lane] = (uint32_t)incl;
        __syncwarp();
        // the vertices, triangles and entries of the groups ahead (this
        // group's are consumed)
        fetch_ndc(g + G, q + 1);
        fetch_tri(g + 2 * G, q + 2);
        fetch_entry(g + 3 * G, q + 3);
        cp_async_commit();
        const int total = (int)S[F_INCL][31];
        for (int p0 = 0; p0 < total; p0 += 32) {
            const int p = p0 + lane;
            int o = 0;
#pragma unroll
            for (int st = 16; st >= 1; st >>= 1)
                if ((int)S[F_INCL][o + st - 1] <= p)
                    o += st;
            o = o > 31 ? 31 : o;
            const bool act = p < total;
            RowIn r;
            if (act) {
                const int ex = o > 0 ? (int)S[F_INCL][o - 1] : 0;
                smem_row_in(r, S, o, p - ex);
            }
            if (!STRIDED) {
                view.x = (int)S[F_VX][o];
                view.w = (int)S[F_VW][o];
                view.key = reinterpret_cast<unsigned long long *>((unsigned long long)S[F_KEY][o] |
                                                                  ((unsigned long long)S[F_KEY + 1][o] << 32));
            }
            const int fr = walk_row<FRAGS>(b, view, inline_span, S[F_ITEM][o], S[F_SLOT][o], r, act, false);
            if (fr)
                atomicAdd(&S[F_FRAGS][o], (uint32_t)fr);
        }
        __syncwarp();
        const uint32_t fr = S[F_FRAGS][lane];
        if (STRIDED)
            fragments += fr;
        else
            block_add(b, item_frags, valid ? S[F_ITEM][lane] : 0u, fr);
        if (__any_sync(0xFFFFFFFFu, late))
            item_add(b, 0, late ? S[F_ITEM][lane] : 0u, 1u, late);
        // the records with fragments, four per round (a 128-byte line by eight
        // lanes): written by one lane each, as eight 16-byte stores to its own
        // line, the stores' 32 lines per instruction throttled the set-up
        // (20 us at 20 % issue on the 1080p frame)
        const unsigned kept = __ballot_sync(0xFFFFFFFFu, fr != 0u);
#pragma unroll
        for (int j0 = 0; j0 < 32; j0 += 4) {
            if (!((kept >> j0) & 15u))
                continue;
            const int j = j0 + (lane >> 3), w = 4 * (lane & 7);
            if ((kept >> j) & 1u) {
                const uint32_t r = W.entry[q & 3][j].x;
                if (in_bounds(r < b->list_cap, CHK_REC, r))
                    reinterpret_cast<uint4 *>(b->recs + r)[lane & 7] =
                        make_uint4(S[w][j], S[w + 1][j], S[w + 2][j], S[w + 3][j]);
            }
        }
        __syncwarp();
    }
    cp_async_wait<0>();
    // then this warp's share of the near-clip and the tall triangles
    if (STRIDED) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            fragments += __shfl_xor_sync(0xFFFFFFFFu, fragments, o);
        if (lane == 0 && fragments)
            atomicAdd(b->item_counters + 1, fragments);
    }
    if (!FRAGS)
        walk_clip_depth(b);
    walk_tall_all<FRAGS>(b, S);
    if (!STRIDED) {
        __syncthreads();
        for (int i = (int)threadIdx.x; i < summed; i += kWalkWarps * 32)
            if (item_frags[i])
                atomicAdd(b->item_counters + 2 * (size_t)i + 1, (unsigned long long)item_frags[i]);
    }
}

// ------------------------------------------------------------- near clip --

// A vertex with everything fill_triangle's clip branches need (mesh_vertex_t,
// swegl/data/model.hpp:20-29).
struct TV {
    V3 vp;     // v_viewport: screen x, y and z'
    V3 world;  // v_world
    V3 normal; // object-space normal
    V3 nworld; // normal_world
    V2 uv;
};

__device__ __forceinline__ void load_tv(const ItemDev &it, uint32_t g, TV &o)
{
    o.vp = load_vp(it, g);
    const float4 w = it.s.wpos[g];
    o.world = mk3(w.x, w.y, w.z);
    const float4 nv = it.s.nrm_v[g];
    o.normal = mk3(nv.x, nv.y, nv.z);
    const float4 nw = it.s.wnrm[g];
    o.nworld = mk3(nw.x, nw.y, nw.z);
    o.uv = mk2(w.w, nw.w);
}

// world_to_viewport (vertex_shaders.hpp:54-59) of a near-clip vertex
__device__ __forceinline__ void world_to_viewport(const ViewDev &v, TV &o, const float *rs)
{
    V3 p = transform3(o.world, v.view);
    o.nworld = normalize_fast<true>(normalize_fast<true>(rotate_n(o.normal, rs)));
    p = transform3(p, v.proj);
    if (p.z != 0.0f) {
        p.x = p.x / fabsf(p.z);
        p.y = p.y / fabsf(p.z);
    }
    p.x = v.vm00 * p.x + v.vm03;
    p.y = v.vm11 * p.y + v.vm13;
    o.vp = p;
}

// near-clip vertex a + (b - a) * cut (renderer.cpp:290-297)
__device__ __forceinline__ void clip_vertex(const ViewDev &v, TV &o, const TV &a, const TV &b, float cut,
                                            const float *rs)
{
    o.world = add3(a.world, mul3(sub3(b.world, a.world), cut));
    o.uv = add2(a.uv, mul2(sub2(b.uv, a.uv), cut));
    if (b.normal.x == a.normal.x && b.normal.y == a.normal.y && b.normal.z == a.normal.z)
        o.normal = a.normal;
    else
        o.normal = normalize3(add3(a.normal, mul3(sub3(b.normal, a.normal), cut)));
    world_to_viewport(v, o, rs);
}

// fill_triangle (src/render/renderer.cpp:240-359) for a triangle with a vertex
// behind the near plane: calls emit(slot, a, b, c, front_face_visible) for the
// fill_triangle_2 calls it makes, in order.  Only the rare near-clip triangles
// come here, so its register and stack use stay off the common walk.
template <class Emit>
__device__ __forceinline__ void clip_triangle(const ItemDev &it, uint32_t t, Emit &emit)
{
    const uint4 tri = it.s.tris[t];
    TV tv[3];
    load_tv(it, tri.x, tv[0]);
    load_tv(it, tri.y, tv[1]);
    load_tv(it, tri.z, tv[2]);
    const float *rs = it.s.node_rs + 16 * it.s.prims[tri.w].node;
    const ViewDev &v = it.v;
    const TV *a = &tv[0], *b = &tv[1], *c = &tv[2], *tp;
    bool ffv = cross_z_negative(sub3(b->vp, a->vp), sub3(c->vp, a->vp));
    bool inverted_order = false;
    if (b->vp.z > a->vp.z) { tp = a; a = b; b = tp; inverted_order = !inverted_order; }
    if (c->vp.z > b->vp.z) { tp = b; b = c; c = tp; inverted_order = !inverted_order; }
    if (b->vp.z > a->vp.z) { tp = a; a = b; b = tp; inverted_order = !inverted_order; }
    const V3 v0 = a->vp, v1 = b->vp, v2 = c->vp;
    if (at_or_past_near(v2.z)) {
        emit(2 * t, *a, *b, *c, ffv); // not reached: compaction sent it to the main list
    } else if (below_near(v1.z)) {
        TV n1, n2;
        clip_vertex(v, n1, *a, *b, (v0.z - 0.001f) / (v0.z - v1.z), rs);
        clip_vertex(v, n2, *a, *c, (v0.z - 0.001f) / (v0.z - v2.z), rs);
        ffv = cross_z_negative(sub3(n1.vp, v0), sub3(n2.vp, v0));
        if (inverted_order)
            ffv = !ffv;
        emit(2 * t, *a, n1, n2, ffv);
    } else {
        TV n1, n2;
        clip_vertex(v, n1, *a, *c, (v0.z - 0.001f) / (v0.z - v2.z), rs);
        clip_vertex(v, n2, *b, *c, (v1.z - 0.001f) / (v1.z - v2.z), rs);
        ffv = cross_z_negative(sub3(v1, v0), sub3(n2.vp, v0));
        if (inverted_order)
            ffv = !ffv;
        emit(2 * t, *a, *b, n2, ffv);
        ffv = cross_z_negative(sub3(n2.vp, v0), sub3(n1.vp, v0));
        if (inverted_order)
            ffv = !ffv;
        emit(2 * t + 1, *a, n2, n1, ffv);
    }
}

// Depth walk of the near-clip triangles (fill_triangle's clip cases), one
// thread each, over a warp-strided share of the clip list.  Out of line: rare,
// and its register and stack use stay off the row walk.
__device__ __noinline__ void walk_clip_depth(const BatchDev *b)
{
    const uint32_t n_raw = *counter32(b, C_CLIP);
    const uint32_t n = n_raw < b->clip_cap ? n_raw : b->clip_cap;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, n_warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t i0 = 32 * gw; i0 < n; i0 += 32 * n_warps) {
        const uint32_t i = i0 + lane;
        const bool valid = i < n;
        DepthVisitor dvis{b, nullptr, 0u, 0u, b->inline_span, 0u, 0ull};
        if (valid) {
            const uint2 e = b->clip[b->clip_cap - 1 - i];
            const ItemDev &it = b->items[e.y];
            dvis.item = e.y;
            dvis.it = &it;
            auto emit = [&](uint32_t slot, const TV &a, const TV &c1, const TV &c2, bool) {
                dvis.slot = slot;
                walk_sub(it.v, a.vp, c1.vp, c2.vp, dvis);
            };
            clip_triangle(it, e.x, emit);
        }
        item_add(b, 0, dvis.item, dvis.drawn_n, valid);
        item_add(b, 1, dvis.item, dvis.fragments, valid);
    }
}

// Set-up and depth walk (or fragment capture) of the tall triangles, a warp
// each, or several where there are warps to spare: one triangle of 300 rows
// was ten turns of one warp, most of a small frame's walk (640 x 480 cube: 14.5 ->
// 7.4 us).
template <bool FRAGS>
__device__ __noinline__ void walk_tall_all(const BatchDev *b, WalkRow *S)
{
    const uint32_t nt_raw = *counter32(b, C_TALL);
    const uint32_t nt = nt_raw < b->list_cap ? nt_raw : b->list_cap;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, n_warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t share = nt && nt < n_warps ? n_warps / nt : 1u;
    for (uint32_t k = gw; k < nt * share; k += n_warps) {
        const uint32_t r = b->tall[k % nt], sub = k / nt;
        const uint32_t item = (uint32_t)find_item(b->tri_base, b->n_items, r), t = r - __ldg(b->tri_base + item);
        const ItemDev &it = b->items[item];
        const uint4 tri = it.s.tris[t];
        __syncwarp();
        // (every lane writes the same values)
        tri_setup(b, it.v, item, t, tri, it.ndc[tri.x], it.ndc[tri.y], it.ndc[tri.z], kRecTall, S, 0);
        __syncwarp();
        if (sub == 0 && in_bounds(r < b->list_cap, CHK_REC, r))
            reinterpret_cast<uint32_t *>(b->recs + r)[lane] = S[lane][0];
        item_add(b, 1, item, walk_tall<FRAGS>(b, S, (int)sub, (int)share), true);
    }
}

// Winner records of what the shade kernel does not replay, after the depth
// keys are final: binned spans (one warp each, the qpixel chain as in
// k_spans), near-clip triangles (one thread each) and, after a bin overflow,
// every span of the walk list.
template <bool WINNER> __device__ __forceinline__ void spans_pass(const BatchDev *b);

__device__ __noinline__ void winner_clip(const BatchDev *b, bool overflow)
{
    const uint32_t n_raw = *counter32(b, C_CLIP);
    const uint32_t n = n_raw < b->clip_cap ? n_raw : b->clip_cap;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint2 e = b->clip[b->clip_cap - 1 - i];
        const ItemDev &it = b->items[e.y];
        WinnerVisitor wvis{&it, 0u, b->inline_span, overflow};
        auto emit = [&](uint32_t slot, const TV &a, const TV &c1, const TV &c2, bool) {
            wvis.slot = slot;
            walk_sub(it.v, a.vp, c1.vp, c2.vp, wvis);
        };
        clip_triangle(it, e.x, emit);
    }
}

__device__ __noinline__ void winner_overflow(const BatchDev *b)
{
    const uint32_t n_raw = *counter32(b, C_LIST), nt_raw = *counter32(b, C_TALL);
    const uint32_t n = n_raw < b->list_cap ? n_raw : b->list_cap, nt = nt_raw < b->list_cap ? nt_raw : b->list_cap;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n + nt; i += gridDim.x * blockDim.x) {
        const uint32_t r = i < n ? b->list[i].x : b->tall[i - n];
        const uint32_t item = i < n ? b->list[i].y : (uint32_t)find_item(b->tri_base, b->n_items, r);
        const ItemDev &it = b->items[item];
        const uint32_t t = r - __ldg(b->tri_base + item);
        WinnerVisitor vis{&it, 2 * t, b->inline_span, true};
        const uint4 tri = it.s.tris[t];
        V3 a = load_vp(it, tri.x), c1 = load_vp(it, tri.y), c2 = load_vp(it, tri.z);
        int pa = 0, pb = 1, pc = 2;
        sort_z_desc(a, c1, c2, pa, pb, pc);
        walk_sub(it.v, a, c1, c2, vis);
    }
}

__device__ __noinline__ void winner_records(const BatchDev *b)
{
    const bool overflow = *counter32(b, C_OVERFLOW) != 0u;
    if (overflow) {
        winner_overflow(b); // records every span, the binned ones included
    } else {
        spans_pass<true>(b);
    }
    winner_clip(b, overflow);
}

__global__ void __launch_bounds__(256, 4) k_winners(const BatchDev *b) { winner_records(b); }

// ------------------------------------------------------------- long spans --

// Binned spans, L lanes each (span_by).  WINNER: the fragments of the recorded
// ones whose key won record their progress values; else the keys are folded.
template <bool WINNER, int L> __device__ __forceinline__ void spans_pass_by(const BatchDev *b, uint32_t n)
{
    const uint32_t step = gridDim.x * blockDim.x / L;
    const int sub = (int)threadIdx.x & (L - 1);
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / L; i < n; i += step) {
        const uint32_t flagged = load_span_item(b, i);
        if (WINNER && !(flagged & kSpanRecorded))
            continue;
        const SpanRec r = load_span(b, i);
        const uint32_t item = flagged & ~kSpanRecorded, slot = r.at.x;
        const ItemDev &it = b->items[item];
        const int y = (int)(r.at.y & kYMask), x2 = (int)r.at.w;
        const long long base = (long long)(y - it.v.y) * it.v.w - it.v.x;
        unsigned long long *row = it.key + base;
        float4 *prec = it.prec + base;
        // WINNER: the keys of a lane's next four pixels are in flight at once
        unsigned long long keys[4] = {};
        int j = 0;
        span_by<L>((int)r.at.z, x2, sub, r.q.x, r.q.y, r.q.z, r.q.w, [&](int x, float top, float bottom) {
            if (WINNER) {
                if ((j & 3) == 0) {
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        keys[k] = x + L * k < x2 ? row[x + L * k] : 0ull;
                } else {
                    keys[0] = keys[1];
                    keys[1] = keys[2];
                    keys[2] = keys[3];
                }
                j++;
            }
            const float alpha = top / bottom;
            const float z = r.e.x + r.e.y * alpha;
            if (below_near(z) || __float_as_uint(z) >= kMaxZBits)
                return;
            if (!in_bounds(x >= it.v.x && x < it.v.x + it.v.w && y >= it.v.y && y < it.v.y + it.v.h,
                           WINNER ? CHK_PREC : CHK_KEY, (unsigned long long)(uint32_t)y << 32 | (uint32_t)x))
                return;
            const unsigned long long key = make_key(z, slot);
            if (!WINNER)
                key_min(row + x, key);
            else if (keys[0] == key)
                prec[x] = make_float4(alpha, r.e.z, r.e.w, __uint_as_float(r.at.y & ~kYMask));
        });
    }
}

// A span takes a warp while there are warps for all of them: its pixels are
// then the longest chain left (640 x 480 cube: spans 4.4 -> 3.2 us, their records
// 2 us less).
template <bool WINNER> __device__ __forceinline__ void spans_pass(const BatchDev *b)
{
    const uint32_t n_raw = *counter32(b, C_SPANS);
    const uint32_t n = n_raw < b->span_cap ? n_raw : b->span_cap;
    if (32ull * n <= (unsigned long long)gridDim.x * blockDim.x)
        spans_pass_by<WINNER, 32>(b, n);
    else
        spans_pass_by<WINNER, kSpanLanes>(b, n);
}

__global__ void __launch_bounds__(256) k_spans(const BatchDev *b) { spans_pass<false>(b); }

// ------------------------------------------------------------------ shade --

__device__ __forceinline__ void bind_material(const SceneDev &s, uint32_t prim, Shader &sh)
{
    const uint4 *p = reinterpret_cast<const uint4 *>(s.pshade + prim); // PrimShade: one 32-byte load
    const uint4 a = p[0], c = p[1];
    sh.tex = reinterpret_cast<const uint32_t *>((unsigned long long)a.x | ((unsigned long long)a.y << 32));
    sh.tw = (int)a.z;
    sh.th = (int)a.w;
    sh.color = c.x;
    sh.shininess = (int)c.y;
}

// Whether a pixel shader's light is per triangle (pixel_shader_lights_flat).
__device__ __forceinline__ bool flat_mode(int shader)
{
    return shader == SGL_SHADER_FLAT_BILINEAR || shader == SGL_SHADER_FLAT_NEAREST || shader == SGL_SHADER_FLAT;
}

// A winner of a near-clipped triangle: the clip vertices are rebuilt exactly
// as fill_triangle makes them; the progress values were recorded by the
// near-clip winner walk.  Rare, so kept out of line.
__device__ __noinline__ uint32_t shade_clip_rec(const ItemDev &it, uint32_t slot, float4 rec)
{
    Shader sh;
    bool done = false;
    auto emit = [&](uint32_t sl, const TV &a, const TV &c1, const TV &c2, bool ffv) {
        if (sl != slot || done)
            return;
        const TV *p0 = &a, *p1 = &c1, *p2 = &c2, *t;
        if (p1->vp.y < p0->vp.y) { t = p0; p0 = p1; p1 = t; }
        if (p2->vp.y < p1->vp.y) { t = p1; p1 = p2; p2 = t; }
        if (p1->vp.y < p0->vp.y) { t = p0; p0 = p1; p1 = t; }
        bind_material(it.s, it.s.tris[slot >> 1].w, sh);
        const uint32_t bits = __float_as_uint(rec.w);
        const bool lower = (bits & kBitLower) != 0u;
        uint32_t is, il, ir;
        sh_edge_ends(lower, (bits & kBitLLR) != 0u, 0u, 1u, 2u, is, il, ir);
        auto vert = [&](uint32_t k) {
            const TV *p = k == 0u ? p0 : (k == 1u ? p1 : p2);
            return SVert{p->world, p->nworld, p->uv};
        };
        sh_fragment(sh, vert(is), vert(il), vert(ir), lower, !ffv, rec.y, rec.z, rec.x);
        if (flat_mode(it.v.shader)) {
            const V3 sw[3] = {p0->world, p1->world, p2->world};
            sh.flat_light = flat_light(sw, !ffv, *it.s.lights, it.v, sh.shininess);
        }
        done = true;
    };
    clip_triangle(it, slot >> 1, emit);
    return done ? sh_shade(sh, *it.s.lights, it.v) : 0u;
}

__device__ __forceinline__ uint32_t shade_clip_px(const ItemDev &it, uint32_t i, uint32_t slot)
{
    return shade_clip_rec(it, slot, it.prec[i]);
}

// 32 bytes in one load: a quarter of a record, or a fragment.
struct Quarter {
    uint32_t w[8];
};
__device__ __forceinline__ Quarter load_quarter(const void *p)
{
    Quarter q;
    asm("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(q.w[0]), "=r"(q.w[1]), "=r"(q.w[2]), "=r"(q.w[3]), "=r"(q.w[4]), "=r"(q.w[5]), "=r"(q.w[6]), "=r"(q.w[7])
        : "l"(p));
    return q;
}
__device__ __forceinline__ Quarter load_quarter(const TriRec *rp, int k)
{
    return load_quarter(reinterpret_cast<const char *>(rp) + 32 * k);
}

// The progress values of pixel (X, Y) (surface coordinates) from its winning
// triangle's set-up (`d`: the record's last quarter): the row's edges after their steps, the span and the
// qpixel chain up to X (renderer.cpp:474-493).  False when the span was wide
// enough to be binned (its winners were recorded by the span kernels).
__device__ __forceinline__ bool rec_replay(const TriRec *rp, const Quarter &d, const ViewDev &v, int X, int Y, float4 &out)
{
    const Quarter a = load_quarter(rp, 0);
    const int y_s = (int)d.w[1], n_u = (int)d.w[2];
    const uint32_t flags = d.w[3];
    const bool upper = Y >= y_s && Y < y_s + n_u;
    const Quarter s = load_quarter(rp, upper ? 1 : 2);
    const int y_l = (int)s.w[6]; // (read in the lower half)
    const int k = upper ? Y - y_s : n_u + (Y - y_l);
    float lg[6], sh[6];
#pragma unroll
    for (int f = 0; f < 6; f++) {
        lg[f] = __uint_as_float(a.w[f]);
        sh[f] = __uint_as_float(s.w[f]);
    }
    RowIn r;
    row_in(r, k, lg, sh, __uint_as_float(a.w[6]), __uint_as_float(d.w[0]), __uint_as_float(a.w[7]), y_s, y_l, n_u, flags);
    RowSpan sp;
    row_span(r, v.x, v.w, sp);
    if (sp.x2 - sp.x1 > kReplaySpan)
        return false;
    Interp it;
    float pl, pr;
    span_interp(sp, it, pl, pr, X - sp.x1);
    out = make_float4(it.alpha, pl, pr, __uint_as_float(r.bits));
    return true;
}

template <bool ALL_MODES>
__device__ __forceinline__ uint32_t shade_rec(const ItemDev &it, uint4 q7, uint32_t flags, float4 rec);

// The colour of one winning fragment: pixel i of item `item`, won by `slot`.
template <bool ALL_MODES>
__device__ __forceinline__ uint32_t shade_winner_impl(const BatchDev *b, uint32_t item, uint32_t i, uint32_t slot,
                                                     bool overflow)
{
    const ItemDev &it = b->items[item];
    const ViewDev &v = it.v;
    const uint32_t r = __ldg(b->tri_base + item) + (slot >> 1);
    if (!in_bounds(r < b->list_cap, CHK_REC, r))
        return 0u;
    const TriRec *rp = b->recs + r;
    const Quarter d = load_quarter(rp, 3);
    const uint32_t flags = d.w[3];
    if (flags == kRecClip)
        return shade_clip_px(it, i, slot);
    const int y = (int)(i / (uint32_t)v.w), x = (int)(i - (uint32_t)y * (uint32_t)v.w);
    float4 rec;
    if (overflow || (flags & kRecTall) || !rec_replay(rp, d, v, x + v.x, y + v.y, rec))
        rec = it.prec[i]; // recorded by the span kernels (or the overflow winner walk)
    return shade_rec<ALL_MODES>(it, make_uint4(d.w[4], d.w[5], d.w[6], d.w[7]), flags, rec);
}

__device__ __forceinline__ SVert load_svert(const ItemDev &it, uint32_t g)
{
    const float4 w = it.s.wpos[g], n = it.s.wnrm[g];
    return SVert{mk3(w.x, w.y, w.z), mk3(n.x, n.y, n.z), mk2(w.w, n.w)};
}

// The colour of a fragment of a set-up triangle (vertices and primitive
// `q7`, TriRec flags `flags`) at the progress values `rec`.
template <bool ALL_MODES>
__device__ __forceinline__ uint32_t shade_rec(const ItemDev &it, uint4 q7, uint32_t flags, float4 rec)
{
    const ViewDev &v = it.v;
    Shader sh;
    bind_material(it.s, q7.w, sh);
    const uint32_t bits = __float_as_uint(rec.w);
    const bool lower = (bits & kBitLower) != 0u, llr = (bits & kBitLLR) != 0u, inverted = (flags & kRecFFV) == 0u;
    uint32_t is, il, ir;
    sh_edge_ends(lower, llr, q7.x, q7.y, q7.z, is, il, ir);
    const SVert s = load_svert(it, is), l = load_svert(it, il), r = load_svert(it, ir);
    sh_fragment(sh, s, l, r, lower, inverted, rec.y, rec.z, rec.x);
    if (ALL_MODES && flat_mode(v.shader)) {
        const V3 v1 = llr ? l.p : r.p, o = llr ? r.p : l.p;
        const V3 sw[3] = {lower ? o : s.p, v1, lower ? s.p : o};
        sh.flat_light = flat_light(sw, inverted, *it.s.lights, v, sh.shininess);
    }
    return sh_shade<ALL_MODES>(sh, *it.s.lights, v);
}

// Per pixel: the background of viewport_t::clear (viewport.cpp:88-113) or the
// colour of the winning fragment, and its depth.  A block takes TILE x TILE
// tiles; background pixels are written at once and winners are queued in
// shared memory, so that the shading runs on full warps.  The depth keys read
// are reset to empty for the next launch sequence (unless kept for debug).
constexpr int kShadeThreads = 256;
#ifndef SGL_SHADE_MIN_BLOCKS
#define SGL_SHADE_MIN_BLOCKS 5 // resident blocks per SM the winner-list shade is compiled for
#endif
#ifndef SGL_TILE_MIN_BLOCKS
#define SGL_TILE_MIN_BLOCKS 6 // ... and the tiled shade, which also hides its key loads and barriers with them (64
                              // views: 511, 451 and 433 us at 4, 5 and 6 blocks)
#endif
template <int TILE, bool ALL_MODES>
__global__ void __launch_bounds__(kShadeThreads, SGL_TILE_MIN_BLOCKS) k_shade(const BatchDev *b)
{
    __shared__ uint4 queue[2 * kShadeThreads];
    __shared__ int qn;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0)
        qn = 0;
    __syncthreads();
    __shared__ uint32_t tile_next;
    const bool overflow = *counter32(b, C_OVERFLOW) != 0u;
    const bool keep = b->keep_keys != 0;
    int item = -1;
    uint32_t lo = 0, hi = 0;
    // Tiles come from kQueues queues (queue q holds tiles q, q + kQueues,
    // ...; block b draws from queue b % kQueues); the next tile is fetched
    // while this one is shaded (the barriers of the loop order the exchange).
    const uint32_t qb = blockIdx.x % kQueues;
    uint32_t *tile_q = counter32(b, C_SHADE_Q + 32 * (int)qb);
    if (threadIdx.x == 0)
        tile_next = qb + kQueues * atomicAdd(tile_q, 1u);
    __syncthreads();
    for (;;) {
        const uint32_t tg = tile_next;
        if (tg >= b->total_tiles)
            break;
        __syncthreads(); // every thread has read tile_next
        if (threadIdx.x == 0)
            tile_next = qb + kQueues * atomicAdd(tile_q, 1u);
        if (tg < lo || tg >= hi) {
            item = find_item(b->tile_base, b->n_items, tg);
            lo = __ldg(b->tile_base + item);
            hi = __ldg(b->tile_base + item + 1);
        }
        const ItemDev &it = b->items[item];
        const uint32_t tl = tg - lo;
        const int tx = (int)(tl % (uint32_t)it.tiles_x), ty = (int)(tl / (uint32_t)it.tiles_x);
        for (int p0 = 0; p0 < TILE * TILE; p0 += kShadeThreads) {
            const int p = p0 + (int)threadIdx.x;
            const int x = tx * TILE + p % TILE, y = ty * TILE + p / TILE;
            bool win = false;
            uint32_t i = 0;
            unsigned long long k = kEmptyKey;
            if (p < TILE * TILE && x < it.v.w && y < it.v.h) {
                i = (uint32_t)y * (uint32_t)it.v.w + (uint32_t)x;
                k = it.key[i];
                if (k == kEmptyKey) {
                    it.pixels[(long long)y * it.pitch_px + x] = 0u;
                    if (it.zbuf)
                        it.zbuf[i] = __uint_as_float(kMaxZBits);
                } else {
                    win = true;
                    if (it.zbuf)
                        it.zbuf[i] = __uint_as_float((uint32_t)(k >> 32));
                    if (!keep)
                        it.key[i] = kEmptyKey;
                }
            }
            const unsigned m = __ballot_sync(0xFFFFFFFFu, win);
            int wb = 0;
            if (lane == 0 && m)
                wb = atomicAdd(&qn, __popc(m));
            wb = __shfl_sync(0xFFFFFFFFu, wb, 0);
            if (win)
                queue[wb + __popc(m & ((1u << lane) - 1u))] = make_uint4(i, (uint32_t)item, (uint32_t)k, 0u);
            __syncthreads();
            const int have = qn;
            if (have >= kShadeThreads) {
                const uint4 e = queue[threadIdx.x];
                const ItemDev &ie = b->items[e.y];
                const ViewDev &ve = ie.v;
                const uint32_t c = shade_winner_impl<ALL_MODES>(b, e.y, e.x, e.z, overflow);
                const int yy = (int)(e.x / (uint32_t)ve.w), xx = (int)(e.x - (uint32_t)yy * (uint32_t)ve.w);
                if (in_bounds(yy < ve.h, CHK_PIXEL, e.x))
                    ie.pixels[(long long)yy * ie.pitch_px + xx] = c;
                __syncthreads();
                if ((int)threadIdx.x < have - kShadeThreads)
                    queue[threadIdx.x] = queue[kShadeThreads + threadIdx.x];
                __syncthreads();
                if (threadIdx.x == 0)
                    qn = have - kShadeThreads;
            }
            __syncthreads();
        }
    }
    if ((int)threadIdx.x < qn) {
        const uint4 e = queue[threadIdx.x];
        const ItemDev &ie = b->items[e.y];
        const uint32_t c = shade_winner_impl<ALL_MODES>(b, e.y, e.x, e.z, overflow);
        const int yy = (int)(e.x / (uint32_t)ie.v.w), xx = (int)(e.x - (uint32_t)yy * (uint32_t)ie.v.w);
        if (in_bounds(yy < ie.v.h, CHK_PIXEL, e.x))
            ie.pixels[(long long)yy * ie.pitch_px + xx] = c;
    }
}

// The same per-pixel work for a batch of one view (kSeqWinList), in
// two passes.  k_classify streams the view's depth keys, four consecutive
// pixels a thread: background colour and every pixel's depth are written at
// once, and the winners appended to the winner list in pixel order, with one
// atomic per block pass; it also makes k_winners' records (nothing it does
// depends on them, and a pass of its own cost a launch).  k_shade_wins then
// shades one winner per thread, without tiles or barriers, and resets its key
// to empty (unless kept for debug).
//
// Bound by the latency of its stream (40 % issue) as single keys, with an
// integer division a pixel; where the target's rows are contiguous and
// aligned (a whole frame, a staged or depth-of-field view) a thread reads its
// keys as 32 bytes and writes colour and depth as 16, without rows.
// Classify and records: 1080p 14.8 -> 10.0 us, 4K 45.8 -> 37.1 us (132 MB of keys,
// colour and depth).  Taking the records last in every other block, beside the
// stream, measured slower (42.5 us).
constexpr int kClassifyPx = 4;   // consecutive pixels of a thread
constexpr int kClassifyRuns = 2; // ... and runs of them in flight per block pass

__global__ void __launch_bounds__(256, 4) k_classify(const BatchDev *b)
{
    winner_records(b);
    __shared__ uint32_t at[kClassifyRuns * 8]; // per (run, warp): winners, then their first list index
    __shared__ uint32_t base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const ItemDev &it = b->items[0];
    const uint32_t total = b->total_px, w = (uint32_t)it.v.w;
    const unsigned long long *keys = b->key_pool;
    uint32_t *pixels = it.pixels;
    float *zbuf = it.zbuf;
    const bool whole = it.pitch_px == it.v.w && ((reinterpret_cast<uintptr_t>(pixels) & 15) == 0) &&
                       ((reinterpret_cast<uintptr_t>(zbuf) & 15) == 0);
    const uint32_t pass = 256u * kClassifyPx * kClassifyRuns;
    for (uint32_t c0 = blockIdx.x * pass; c0 < total; c0 += gridDim.x * pass) {
        unsigned long long k[kClassifyRuns][kClassifyPx];
#pragma unroll
        for (int r = 0; r < kClassifyRuns; r++) {
            const uint32_t g = c0 + (r * 256u + threadIdx.x) * kClassifyPx;
            if (g + kClassifyPx <= total) { // (the key pool is 256-byte aligned)
                asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                             : "=l"(k[r][0]), "=l"(k[r][1]), "=l"(k[r][2]), "=l"(k[r][3])
                             : "l"(keys + g));
            } else {
#pragma unroll
                for (int j = 0; j < kClassifyPx; j++)
                    k[r][j] = g + j < total ? keys[g + j] : kEmptyKey;
            }
        }
        uint32_t first[kClassifyRuns]; // this lane's winners follow so many of its warp's
#pragma unroll
        for (int r = 0; r < kClassifyRuns; r++) {
            const uint32_t g = c0 + (r * 256u + threadIdx.x) * kClassifyPx;
            float z[kClassifyPx];
            uint32_t n = 0;
#pragma unroll
            for (int j = 0; j < kClassifyPx; j++) {
                const bool win = k[r][j] != kEmptyKey;
                z[j] = __uint_as_float(win ? (uint32_t)(k[r][j] >> 32) : kMaxZBits);
                n += win;
            }
            if (whole && g + kClassifyPx <= total) {
                // (a winner's colour is written by the shade)
                *reinterpret_cast<uint4 *>(pixels + g) = make_uint4(0u, 0u, 0u, 0u);
                if (zbuf)
                    *reinterpret_cast<float4 *>(zbuf + g) = make_float4(z[0], z[1], z[2], z[3]);
            } else {
#pragma unroll
                for (int j = 0; j < kClassifyPx; j++)
                    if (g + j < total) {
                        const uint32_t y = (g + j) / w, x = g + j - y * w;
                        pixels[(long long)y * it.pitch_px + x] = 0u;
                        if (zbuf)
                            zbuf[g + j] = z[j];
                    }
            }
            uint32_t incl = n;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                if (lane >= d)
                    incl += t;
            }
            first[r] = incl - n;
            if (lane == 31)
                at[r * 8 + warp] = incl;
        }
        __syncthreads();
        if (warp == 0) {
            // exclusive prefix of the counts in (run, warp) order, which is pixel order
            const uint32_t a = lane < kClassifyRuns * 8 ? at[lane] : 0u;
            uint32_t incl = a;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                if (lane >= d)
                    incl += t;
            }
            if (lane < kClassifyRuns * 8)
                at[lane] = incl - a;
            if (lane == 31)
                base = incl ? atomicAdd(counter32(b, C_WINS), incl) : 0u;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kClassifyRuns; r++) {
            uint32_t e = base + at[r * 8 + warp] + first[r];
#pragma unroll
            for (int j = 0; j < kClassifyPx; j++)
                if (k[r][j] != kEmptyKey && in_bounds(e < total, CHK_PIXEL, e))
                    b->wins[e++] = make_uint2(c0 + (r * 256u + threadIdx.x) * kClassifyPx + j, (uint32_t)k[r][j]);
        }
        __syncthreads(); // `at` and `base` are reused by the next pass
    }
}

template <bool ALL_MODES>
__global__ void __launch_bounds__(kShadeThreads, SGL_SHADE_MIN_BLOCKS) k_shade_wins(const BatchDev *b)
{
    const uint32_t n = *counter32(b, C_WINS);
    const bool overflow = *counter32(b, C_OVERFLOW) != 0u, keep = b->keep_keys != 0;
    const ItemDev &it = b->items[0];
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const uint2 wn = b->wins[e];
        const uint32_t i = wn.x;
        const uint32_t c = shade_winner_impl<ALL_MODES>(b, 0u, i, wn.y, overflow);
        const uint32_t y = i / (uint32_t)it.v.w, x = i - y * (uint32_t)it.v.w;
        if (in_bounds(y < (uint32_t)it.v.h, CHK_PIXEL, i)) {
            it.pixels[(long long)y * it.pitch_px + x] = c;
            if (!keep)
                b->key_pool[i] = kEmptyKey;
        }
    }
}

// ------------------------------------------------------------ depth of field --

// The fragment pool was too small: nothing is written, the host renders again.
__device__ __forceinline__ bool frags_overflowed(const BatchDev *b)
{
    return *frag_counter(b) > (unsigned long long)b->frag_cap;
}

__constant__ float2 c_dof_taps[SGL_DOF_TAPS];

// Circle of confusion at depth zp of a depth-of-field item.
__device__ __forceinline__ float dof_radius_at(const ItemDev &it, float zp)
{
    const float zv = (zp - it.p23) / it.p22;
    float r = (it.dof_ka * fabsf(zv - it.dof_focus)) / zv;
    if (!(r >= 0.0f && r <= it.dof_rmax))
        r = it.dof_rmax;
    return r;
}

// ... with `far` the radius of an empty pixel (the cleared depth), whose huge
// operands would take both divisions through their slow path.
__device__ __forceinline__ float dof_radius(const ItemDev &it, float zp, float far)
{
    return __float_as_uint(zp) == kMaxZBits ? far : dof_radius_at(it, zp);
}

__device__ __forceinline__ uint32_t dof_average(uint32_t centre, uint32_t sb, uint32_t sg, uint32_t sr)
{
    return (centre & 0xFF000000u) | (((sr + 16u) / 32u) << 16) | (((sg + 16u) / 32u) << 8) | ((sb + 16u) / 32u);
}

// 1.5 * 2^23: a float of magnitude below 2^22 added to it is rounded to the
// nearest integer (ties to even, as __float2int_rn), which is the sum's bits
// less kTapBias.  One full-rate addition, where the conversion unit takes a
// warp per two cycles: with two conversions a tap that unit bound the gather
// of pixels of unlike radius.
constexpr float kTapRound = 12582912.0f;
constexpr uint32_t kTapBias = 0x4B400000u;

// r * tap rounded to the nearest integers, each plus kTapBias (|r| < 2^22).
// (Paired single-precision instructions would halve these four, but a paired
// product, even as a fused multiply-add with -0, and a paired addition came
// out contracted: offsets one off in a pixel of a million.)
__device__ __forceinline__ uint2 tap_offset(float r, float2 t)
{
    return make_uint2(__float_as_uint(__fadd_rn(__fmul_rn(r, t.x), kTapRound)),
                      __float_as_uint(__fadd_rn(__fmul_rn(r, t.y), kTapRound)));
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// Depth-of-field gather (replaces post_shader_depth_box,
// swegl/render/post_shaders.hpp:51-132).  Per pixel: view-space depth from the
// z-buffer, z = (z' - P23) / P22; circle of confusion r = K*A*|z - F| / z
// pixels, clamped to [0, max]; the mean of 32 taps of the golden-angle
// pattern (sgl_dof_taps.h) at offsets r * tap rounded to the nearest integer
// (ties to even: one conversion instruction), clamped to the
// viewport, with integer sums rounded half up.  Every step is exact integer
// or IEEE float arithmetic, so the CPU oracle gives the same bits.
//
// A block takes kDofTile x kDofTile tiles of the items that ask for the
// gather and stages the tile with its halo (the taps reach at most
// ceil(max_radius) pixels: every tap component is below 1), clamped to the
// view as the taps are, in shared memory; the 32 taps of each pixel then read
// shared memory without further clamping.  Halos of up to 16 pixels (the usual
// radius) take half the shared memory, and the next tile's halo is copied in
// (and its depths loaded) while this one is gathered; wider ones are staged
// before each tile.  Inside the view a halo is copied as 16-byte words, where
// the source's rows are aligned to them.  Views whose reach exceeds
// kDofMaxHalo gather from the colour buffer.
//
// Bound by integer issue (two ALU instructions and a shared-memory read a
// pixel and tap); before, staging took a quarter of the instructions a word at
// a time and its latency was the main stall (a 3840 x 2160 frame of the spheres,
// radius 16: 60.9 M instructions and 87.4 us, now 52.0 M and 65.6 us; 2560 x
// 1440 of unlike radii up to 24: 64 -> 55 us).
constexpr int kDofBlocks = 5; // resident blocks per SM (shared memory: 37 KB each)
constexpr int kDofNear = 16;  // halo whose tiles are staged ahead
constexpr int kDofNearPitch = kDofTile + 2 * kDofNear;
static_assert(2 * kDofNearPitch * kDofNearPitch <= kDofPitch * kDofPitch, "two near tiles share the shared memory");
static_assert(kDofTile == 32 && kDofNear % 4 == 0 && kDofMaxHalo % 4 == 0, "16-byte words of a halo");

// The tile in hand: its item, place and, per thread, the pixels' depths and
// the staged pixel that a constant tile repeats.
struct DofTile {
    const ItemDev *it;
    int x0, y0, w, h;
    float z[4]; // of rows y0 + warp + 8 j, column x0 + lane (clamped into the view)
    uint32_t ref;

    __device__ __forceinline__ void load_depths()
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int x = x0 + lane < w ? x0 + lane : x0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int y = y0 + warp + 8 * j;
            z[j] = y < h ? it->zbuf[(uint32_t)y * (uint32_t)w + (uint32_t)x] : 0.0f;
        }
        ref = __ldg(it->dof_src + (size_t)y0 * it->dof_src_pitch + x0);
    }
};

// Copies the tile and PITCH-wide halo (view-clamped) into `halo` with
// cp.async (not committed); the tile's pixel (0, 0) lands at row and column
// (PITCH - kDofTile) / 2.
template <int PITCH> __device__ __forceinline__ void dof_stage(const DofTile &t, uint32_t *halo)
{
    constexpr int R = (PITCH - kDofTile) / 2, V = PITCH / 4; // 16-byte words of a row
    const uint32_t *src = t.it->dof_src;
    const int sp = t.it->dof_src_pitch;
    const int xa = t.x0 - R, ya = t.y0 - R;
    if (xa >= 0 && xa + PITCH <= t.w && (sp & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
        for (int i = (int)threadIdx.x; i < PITCH * V; i += 256) {
            const int yy = i / V, v = i - yy * V;
            const int sy = min(max(ya + yy, 0), t.h - 1);
            cp_async<16>(halo + yy * PITCH + 4 * v, src + (size_t)sy * sp + xa + 4 * v);
        }
    } else {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        for (int yy = warp; yy < PITCH; yy += 8) {
            const uint32_t *row = src + (size_t)min(max(ya + yy, 0), t.h - 1) * sp;
#pragma unroll
            for (int c = 0; c < PITCH; c += 32)
                cp_async<4>(halo + yy * PITCH + c + lane, row + min(max(xa + c + lane, 0), t.w - 1));
        }
    }
}

// Whether every word that this thread staged holds t.ref.
template <int PITCH> __device__ __forceinline__ bool dof_same(const DofTile &t, const uint32_t *halo)
{
    bool same = true;
    for (int i = (int)threadIdx.x; i < PITCH * PITCH / 4; i += 256) {
        const uint4 v = reinterpret_cast<const uint4 *>(halo)[i];
        same &= v.x == t.ref && v.y == t.ref && v.z == t.ref && v.w == t.ref;
    }
    return same;
}

// The gather of a staged tile; `far` as in dof_radius.
template <int PITCH> __device__ __forceinline__ void dof_gather(const DofTile &t, const uint32_t *halo, float far)
{
    constexpr int R = (PITCH - kDofTile) / 2;
    const ItemDev &it = *t.it;
    // Warp w takes rows w, w + 8, w + 16 and w + 24 of the tile, a lane
    // one column.  The sums are exact integers, so the taps may be
    // taken in any order: rb sums bytes 0 and 2 in two 16-bit lanes
    // (32 x 255 fits), g sums whole pixels modulo 2^32, so that bits
    // 8..23 of g - rb are the sum of byte 1 (below 2^24 after the
    // shift: byte 3's sum lands at bit 24 and up); alpha is the
    // centre's.
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int w = t.w, h = t.h, x0 = t.x0, y0 = t.y0, x = x0 + lane;
    if (y0 + warp >= h)
        return;
    const bool valid = x < w;
    const int xs = valid ? x : x0; // lanes past the view's right edge work on a pixel inside
    float r[4];
    bool uniform = true;
#pragma unroll
    for (int j = 0; j < 4; j++)
        r[j] = y0 + warp + 8 * j < h ? dof_radius(it, t.z[j], far) : 0.0f;
    const float r0 = __shfl_sync(0xFFFFFFFFu, r[0], 0);
#pragma unroll
    for (int j = 0; j < 4; j++)
        uniform &= !valid || y0 + warp + 8 * j >= h || r[j] == r0;
    // the halo holds the view-clamped pixels, so a tap needs no
    // clamp: |offset| <= ceil(r) <= R keeps it inside
    const uint32_t *c = halo + (warp + R) * PITCH + (xs - x0 + R);
    uint32_t rb[4] = {0u, 0u, 0u, 0u}, g[4] = {0u, 0u, 0u, 0u};
    if (__all_sync(0xFFFFFFFFu, uniform)) {
        // one radius for the warp's 128 pixels (the clamped radius,
        // or the empty background's): lane k makes tap k's offset
        // once, and each offset serves the four rows
        static_assert(SGL_DOF_TAPS == 32, "one tap per lane");
        const float2 tap = c_dof_taps[lane];
        const int off = __float2int_rn(r0 * tap.y) * PITCH + __float2int_rn(r0 * tap.x);
#pragma unroll 4
        for (int k = 0; k < SGL_DOF_TAPS; k += 2) {
            const uint32_t *q = c + __shfl_sync(0xFFFFFFFFu, off, k);
            const uint32_t *p = c + __shfl_sync(0xFFFFFFFFu, off, k + 1);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const uint32_t v = q[8 * j * PITCH], u = p[8 * j * PITCH];
                rb[j] += (v & 0x00FF00FFu) + (u & 0x00FF00FFu);
                g[j] += v + u;
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (y0 + warp + 8 * j >= h)
                break; // the whole warp
            const uint32_t *cj = c + 8 * j * PITCH;
            const float rj0 = __shfl_sync(0xFFFFFFFFu, r[j], 0);
            if (__all_sync(0xFFFFFFFFu, !valid || r[j] == rj0)) {
                const float2 tap = c_dof_taps[lane];
                const int off = __float2int_rn(rj0 * tap.y) * PITCH + __float2int_rn(rj0 * tap.x);
#pragma unroll 4
                for (int k = 0; k < SGL_DOF_TAPS; k += 2) {
                    const uint32_t v = cj[__shfl_sync(0xFFFFFFFFu, off, k)];
                    const uint32_t u = cj[__shfl_sync(0xFFFFFFFFu, off, k + 1)];
                    rb[j] += (v & 0x00FF00FFu) + (u & 0x00FF00FFu);
                    g[j] += v + u;
                }
            } else {
                // the pixel's shared address less the offsets' bias
                const uint32_t at = (uint32_t)__cvta_generic_to_shared(cj) - kTapBias * (4u + 4u * (uint32_t)PITCH);
#pragma unroll 8
                for (int k = 0; k < SGL_DOF_TAPS; k += 2) {
                    const uint2 a = tap_offset(r[j], c_dof_taps[k]), e = tap_offset(r[j], c_dof_taps[k + 1]);
                    const uint32_t v = lds32(at + a.y * (4u * (uint32_t)PITCH) + 4u * a.x);
                    const uint32_t u = lds32(at + e.y * (4u * (uint32_t)PITCH) + 4u * e.x);
                    rb[j] += (v & 0x00FF00FFu) + (u & 0x00FF00FFu);
                    g[j] += v + u;
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int y = y0 + warp + 8 * j;
        if (valid && y < h)
            it.dof_out[(size_t)y * it.dof_pitch + x] =
                dof_average(c[8 * j * PITCH], rb[j] & 0xFFFFu, ((g[j] - rb[j]) >> 8) & 0xFFFFu, rb[j] >> 16);
    }
}

// A tile whose staged pixels all hold t.ref: every tap of every pixel reads
// that value: 32 equal channels c sum to 32 c, and (32 c + 16) / 32 = c, alpha
// is the centre's: the gather leaves it unchanged.
__device__ __forceinline__ void dof_constant(const DofTile &t)
{
    const ItemDev &it = *t.it;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int x = t.x0 + lane, y = t.y0 + warp + 8 * j;
        if (x < t.w && y < t.h)
            it.dof_out[(size_t)y * it.dof_pitch + x] = t.ref;
    }
}

// A tile gathered from the colour buffer.
__device__ __noinline__ void dof_from_memory(const ItemDev &it, int x0, int y0, float far)
{
    const int w = it.v.w, h = it.v.h;
    for (int p = threadIdx.x; p < kDofTile * kDofTile; p += blockDim.x) {
        const int x = x0 + (p & (kDofTile - 1)), y = y0 + p / kDofTile;
        if (y >= h)
            continue; // the whole warp
        const bool valid = x < w;
        const int xs = valid ? x : x0;
        const float z = it.zbuf[(uint32_t)y * (uint32_t)w + (uint32_t)xs];
        const float r = dof_radius(it, z, far);
        uint32_t rb = 0, g = 0; // (as in dof_gather)
#pragma unroll 8
        for (int k = 0; k < SGL_DOF_TAPS; k++) {
            const uint2 o = tap_offset(r, c_dof_taps[k]);
            int sx = xs + (int)(o.x - kTapBias), sy = y + (int)(o.y - kTapBias);
            sx = sx < 0 ? 0 : (sx >= w ? w - 1 : sx);
            sy = sy < 0 ? 0 : (sy >= h ? h - 1 : sy);
            const uint32_t v = __ldg(it.dof_src + (size_t)sy * it.dof_src_pitch + sx);
            rb += v & 0x00FF00FFu;
            g += v;
        }
        if (valid)
            it.dof_out[(size_t)y * it.dof_pitch + x] = dof_average(it.dof_src[(size_t)y * it.dof_src_pitch + xs],
                                                                   rb & 0xFFFFu, ((g - rb) >> 8) & 0xFFFFu, rb >> 16);
    }
}

__global__ void __launch_bounds__(256, kDofBlocks) k_dof(const BatchDev *b)
{
    if (frags_overflowed(b))
        return; // a layered view whose fragment pool was too small: rendered again
    __shared__ __align__(16) uint32_t halo[kDofPitch * kDofPitch];
    __shared__ uint32_t claim[4]; // tiles of the next rounds (tiles cost from a copy to a full gather)
    const uint32_t total = b->total_dof_tiles;
    int item = -1;
    uint32_t lo = 0, hi = 0;
    float far = 0.0f, far_next = 0.0f; // the items' radii of an empty pixel
    // the place of tile tg
    auto locate = [&](uint32_t tg, DofTile &t) {
        if (tg < lo || tg >= hi) {
            item = find_item(b->dof_base, b->n_items, tg);
            lo = __ldg(b->dof_base + item);
            hi = __ldg(b->dof_base + item + 1);
            far_next = dof_radius_at(b->items[item], __uint_as_float(kMaxZBits));
        }
        t.it = b->items + item;
        t.w = t.it->v.w;
        t.h = t.it->v.h;
        const uint32_t tl = tg - lo, tx = (uint32_t)t.it->dof_tiles_x;
        t.y0 = (int)(tl / tx) * kDofTile;
        t.x0 = (int)(tl % tx) * kDofTile;
    };
    auto near = [](const DofTile &t) { return t.it->dof_halo >= 0 && t.it->dof_halo <= kDofNear; };
    if (threadIdx.x == 0) {
        claim[0] = atomicAdd(counter32(b, C_DOF_NEXT), 1u);
        claim[1] = atomicAdd(counter32(b, C_DOF_NEXT), 1u);
    }
    __syncthreads();
    DofTile t{}, next{};
    uint32_t tg = claim[0];
    if (tg < total) {
        locate(tg, t);
        far = far_next;
        if (near(t)) {
            dof_stage<kDofNearPitch>(t, halo);
            t.load_depths();
        }
    }
    cp_async_commit();
    for (int q = 0; tg < total; q++) {
        // this round's tile is in hand; claim the one after the next, and
        // start on the next
        const uint32_t tn = claim[(q + 1) & 3];
        if (threadIdx.x == 0)
            claim[(q + 2) & 3] = atomicAdd(counter32(b, C_DOF_NEXT), 1u);
        uint32_t *mine = halo + (q & 1) * kDofNearPitch * kDofNearPitch;
        const bool mine_near = near(t);
        bool next_near = false;
        if (tn < total) {
            locate(tn, next);
            next_near = near(next);
            if (next_near && mine_near) {
                dof_stage<kDofNearPitch>(next, halo + ((q + 1) & 1) * kDofNearPitch * kDofNearPitch);
                next.load_depths();
            }
        }
        cp_async_commit();
        if (mine_near) {
            cp_async_wait<1>();
            __syncthreads();
            if (__syncthreads_and(dof_same<kDofNearPitch>(t, mine)))
                dof_constant(t);
            else
                dof_gather<kDofNearPitch>(t, mine, far);
        } else if (t.it->dof_halo >= 0) {
            dof_stage<kDofPitch>(t, halo);
            t.load_depths();
            cp_async_commit();
            cp_async_wait<0>();
            __syncthreads();
            if (__syncthreads_and(dof_same<kDofPitch>(t, halo)))
                dof_constant(t);
            else
                dof_gather<kDofPitch>(t, halo, far);
        } else {
            dof_from_memory(*t.it, t.x0, t.y0, far);
        }
        __syncthreads(); // the halo is reused, claim[(q + 2) & 3] is written
        if (next_near && !mine_near) { // (its place was in use)
            dof_stage<kDofNearPitch>(next, halo + ((q + 1) & 1) * kDofNearPitch * kDofNearPitch);
            next.load_depths();
            cp_async_commit();
        }
        t = next;
        tg = tn;
        far = far_next;
    }
    cp_async_wait<0>();
}

// The gather's input for a view with transparency layers: its rectangle of
// the surface after the layer passes (the flatten and copy write the surface
// at the reference's offsets, so the rectangle is read back whole), copied
// to the scratch buffer, since the gather writes the rectangle in place.
__global__ void __launch_bounds__(256) k_dof_source(const BatchDev *b)
{
    if (frags_overflowed(b))
        return;
    const ItemDev &it = b->items[0];
    const int w = it.v.w;
    const uint32_t total = (uint32_t)w * (uint32_t)it.v.h;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int y = (int)(i / (uint32_t)w), x = (int)(i - (uint32_t)y * (uint32_t)w);
        it.dof_src[(size_t)y * it.dof_src_pitch + x] = it.dof_out[(long long)y * it.dof_pitch + x];
    }
}

// ------------------------------------------------------ transparency layers --
//
// A view with transparency layers (renderer.cpp:494-550) keeps per pixel the
// opaque depth and colour and up to `layers` transparent fragments sorted by
// depth, layer 0 the farthest.  The outcome depends on the draw order only
// through depth ties, so it can be computed from the pixel's fragments taken
// in any order:
//  - the screen gets the first drawn of the nearest opaque (alpha 255)
//    fragments, as without layers, and the depth buffer its depth;
//  - the layers hold the `layers` nearest transparent fragments strictly in
//    front of it, nearer meaning a smaller depth or, at equal depth, drawn
//    later (an insertion goes in front of the equal depths already there,
//    and when every layer is used the farthest is dropped).
// The capture stores every fragment, the linking chains those of a pixel (and
// shades them, or leaves that to the resolve: frags_on_demand), and the resolve
// takes a pixel's chain to that outcome.  The flatten and copy passes follow viewport_t::flatten
// (viewport.cpp:43-86) and post_shader_t's copy of the first layer to the
// screen (post_shaders.hpp:22-47).  A layered batch holds one view.


// blend (src/render/colors.cpp:39-57): back * (256 - a) / 256 + front * a / 256
// truncated, which is exact in integers (both terms are multiples of 1/256).
__device__ __forceinline__ uint32_t blend_px(uint32_t back, uint32_t front)
{
    const uint32_t a = front >> 24, ba = back >> 24;
    const uint32_t na = 255u - ((255u - a) * (255u - ba) / 255u);
    if (a == 255u)
        return (front & 0x00FFFFFFu) | (na << 24);
    if (a == 0u)
        return (back & 0x00FFFFFFu) | (na << 24);
    uint32_t out = na << 24;
#pragma unroll
    for (int c = 0; c < 24; c += 8) {
        const uint32_t bc = (back >> c) & 0xFFu, fc = (front >> c) & 0xFFu;
        out |= ((bc * (256u - a) + fc * a) >> 8) << c;
    }
    return out;
}

// The fragments a triangle reserves (one per span pixel): the walk of its
// edges without the pixel loops.
struct FragCount {
    uint32_t slot; // unused (the walk's emit sets it)
    unsigned long long n;

    __device__ __forceinline__ bool active() const { return true; }
    __device__ __forceinline__ void drawn() {}
    __device__ __forceinline__ void span(int, int x1, int x2, const Side &, const Side &, uint32_t)
    {
        n += (unsigned long long)(x2 - x1);
    }
};

// Stores every fragment of its spans from the triangle's reserved range at
// `at` on (span_frags).  Spans longer than kFragInline are binned for
// k_frag_spans.
constexpr int kFragInline = 32;
struct FragVisitor {
    const BatchDev *b;
    const ItemDev *it;
    uint32_t slot;
    uint32_t drawn_n;
    unsigned long long fragments;
    unsigned long long at;

    __device__ __forceinline__ bool active() const { return true; }
    __device__ __forceinline__ void drawn() { drawn_n++; }
    __device__ __forceinline__ void span(int y, int x1, int x2, const Side &Ls, const Side &Rs, uint32_t bits)
    {
        const unsigned long long n = (unsigned long long)(x2 - x1);
        fragments += n;
        const unsigned long long k = at;
        at += n;
        if (k + n > (unsigned long long)b->frag_cap)
            return; // counted, not stored: the pool is grown and the view rendered again
        if (n > (unsigned long long)kFragInline) {
            // a long span goes to the bins: its pixels are stored a warp at a time
            const uint32_t si = atomicAdd(counter32(b, C_SPANS), 1u);
            if (si < b->span_cap) {
                Interp q;
                q.init_self(Rs.x - Ls.x, Ls.it.value(), Rs.it.value());
                q.displace((float)x1 - Ls.x);
                // (item: the span's first fragment; a layered batch has one item)
                store_span(b, si, (uint32_t)k, slot, (uint32_t)y | bits, x1, x2, q, Ls.it.alpha, Rs.it.alpha);
                return;
            }
        }
        const ViewDev &v = it->v;
        Interp q;
        q.init_self(Rs.x - Ls.x, Ls.it.value(), Rs.it.value());
        q.displace((float)x1 - Ls.x);
        span_frags(b, (uint32_t)((y - v.y) * v.w - v.x), slot, x1, x2, q, Ls.it.alpha, Rs.it.alpha, bits,
                   (uint32_t)k);
    }
};

// Fragment capture of the near-clipped triangles (the walk list is captured
// by k_walk<true, true>): one thread per triangle runs fill_triangle's clip cases
// and the fill_triangle_2 walk.  Each lane first counts its triangle's
// fragments; the warp then reserves its lanes' ranges with one atomic and
// walks again to store them.  Bound by each thread's chain, not by the number
// of warps (sms * 2 blocks are launched): compiled for one block an SM it
// takes 91 registers without spills, left to the compiler 80 with (a call with
// 4,000 near-clipped triangles at 960 x 540 6.24 and 6.47 ms).
__global__ void __launch_bounds__(256, 1) k_frags(const BatchDev *b)
{
    const uint32_t c_raw = *counter32(b, C_CLIP);
    const uint32_t nc = c_raw < b->clip_cap ? c_raw : b->clip_cap;
    const int lane = threadIdx.x & 31;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; i0 < nc; i0 += stride) {
        const uint32_t i = i0 + (uint32_t)lane;
        const bool valid = i < nc;
        uint2 e = make_uint2(0u, 0u);
        if (valid)
            e = b->clip[b->clip_cap - 1 - i];
        const ItemDev &it = b->items[e.y];
        auto walk = [&](auto &vis) {
            if (!valid)
                return;
            auto emit = [&](uint32_t slot, const TV &a, const TV &c1, const TV &c2, bool) {
                vis.slot = slot;
                walk_sub(it.v, a.vp, c1.vp, c2.vp, vis);
            };
            clip_triangle(it, e.x, emit);
        };
        FragCount cnt{0u, 0ull};
        walk(cnt);
        unsigned long long incl = cnt.n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o)
                incl += up;
        }
        unsigned long long base = 0;
        if (lane == 31 && incl)
            base = atomicAdd(frag_counter(b), incl);
        base = __shfl_sync(0xFFFFFFFFu, base, 31);
        FragVisitor vis{b, &it, 0u, 0u, 0ull, base + incl - cnt.n};
        walk(vis);
        item_add(b, 0, e.y, vis.drawn_n, valid);
        item_add(b, 1, e.y, vis.fragments, valid);
    }
}

// The binned long spans of the capture, eight lanes each as in k_spans: every
// lane stores its pixels' fragments.
__global__ void __launch_bounds__(256) k_frag_spans(const BatchDev *b)
{
    if (frags_overflowed(b))
        return;
    const uint32_t n_raw = *counter32(b, C_SPANS);
    const uint32_t n = n_raw < b->span_cap ? n_raw : b->span_cap;
    const ItemDev &it = b->items[0];
    const ViewDev &v = it.v;
    Frag *pool = b->frags;
    const uint32_t step = gridDim.x * blockDim.x / kSpanLanes;
    const int sub = (int)threadIdx.x & (kSpanLanes - 1);
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / kSpanLanes; i < n; i += step) {
        const SpanRec r = load_span(b, i);
        const uint32_t first = load_span_item(b, i);
        const int y = (int)(r.at.y & kYMask), x1 = (int)r.at.z;
        const uint32_t row_px = (uint32_t)((y - v.y) * v.w - v.x);
        const float fb = __uint_as_float(r.at.y & ~kYMask);
        span_by<kSpanLanes>(x1, (int)r.at.w, sub, r.q.x, r.q.y, r.q.z, r.q.w, [&](int x, float top, float bottom) {
            const float alpha = top / bottom;
            const float z = r.e.x + r.e.y * alpha;
            const bool keep = !below_near(z) && __float_as_uint(z) < kMaxZBits;
            const uint32_t at = first + (uint32_t)(x - x1);
            reinterpret_cast<float4 *>(pool + at)[0] = make_float4(alpha, r.e.z, r.e.w, fb);
            reinterpret_cast<uint4 *>(pool + at)[1] =
                make_uint4(__float_as_uint(z), r.at.x, keep ? row_px + (uint32_t)x : kFragEnd, 0u);
        });
    }
}

// The colour of a captured fragment.
template <bool ALL_MODES>
__device__ __forceinline__ uint32_t shade_frag(const BatchDev *b, const ItemDev &it, uint32_t item, uint32_t slot,
                                               float4 rec)
{
    const Quarter d = load_quarter(b->recs + __ldg(b->tri_base + item) + (slot >> 1), 3);
    if (d.w[3] == kRecClip)
        return shade_clip_rec(it, slot, rec);
    return shade_rec<ALL_MODES>(it, make_uint4(d.w[4], d.w[5], d.w[6], d.w[7]), d.w[3], rec);
}

// Whether fragments are shaded when their pixel is resolved, nearest first
// until one is opaque, instead of all when they are linked.  In the pool's
// order neighbours share a triangle and every lane has a fragment, but hidden
// ones are shaded too; by pixel a warp takes as many turns as its deepest
// pixel, each a chain of dependent loads.  So it depends on the view's
// fragments a pixel, f, and on the share p of them that are translucent (of
// the scene's samples): k_link + k_layers, linked / on demand, us:
//   f 0.9  p 0: 61 / 62      .05: 61 / 84     .3: 65 / 109
//   f 1.8  p 0: 109 / 90     .02: 109 / 109   .05: 110 / 119
//   f 3.3  p 0: 196 / 123    .1: 202 / 177    .15: 204 / 196   .2: 205 / 211
//   f 6.4  p 0: 384 / 188    .1: 409 / 249    .3: 418 / 353
//   f 7.0  p 0: 78 / 46      .15: 84 / 80     .2: 84 / 88
//   f 13.5 p 0: 267 / 95     .15: 282 / 132   .3: 284 / 175
// (1280 x 720 but for 7.0 and 13.5).  The line f = 1.25 + 16 p lies between,
// and f = 1 where none is translucent: a pixel then takes one turn, else a warp
// takes those of its deepest (calls at 640 x 360, linked / on demand: f 1.0 to 1.25,
// p 0 258 / 246 us; f 1.4, p .02 159 / 169).  From a half on they are linked: the
// turns grow with the chain's length squared.
__device__ __forceinline__ bool frags_on_demand(const BatchDev *b, const ItemDev &it)
{
    const unsigned long long n = __ldg(it.s.translucent);
    const float p = (float)n / ((float)kAlphaSamples * (float)it.s.n_triangles);
    const float px = (float)it.v.w * (float)it.v.h;
    return p < 0.5f && (float)*frag_counter(b) > px * (n ? 1.25f + 16.0f * p : 1.0f);
}

// Chains the stored fragments to their pixels: one thread per pool entry
// swaps itself into its pixel's list head and keeps the previous head as its
// successor (the chain order is free: the resolve orders by depth and slot);
// and shades it, unless that waits for the resolve.
template <bool ALL_MODES>
__global__ void __launch_bounds__(256, SGL_SHADE_MIN_BLOCKS) k_link(const BatchDev *b)
{
    if (frags_overflowed(b))
        return;
    const uint32_t n = (uint32_t)*frag_counter(b);
    const ItemDev &it = b->items[0];
    const bool on_demand = frags_on_demand(b, it);
    uint32_t *head = it.frag_head;
    Frag *pool = b->frags;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const Quarter f = load_quarter(pool + i);
        const uint32_t px = f.w[6];
        if (px == kFragEnd)
            continue;
        const uint32_t next = atomicExch(head + px, i);
        uint32_t c = 0u;
        if (!on_demand)
            c = shade_frag<ALL_MODES>(b, it, 0u, f.w[5],
                                      make_float4(__uint_as_float(f.w[0]), __uint_as_float(f.w[1]),
                                                  __uint_as_float(f.w[2]), __uint_as_float(f.w[3])));
        reinterpret_cast<uint2 *>(pool + i)[3] = make_uint2(next, c);
    }
}

// A layered pixel's outcome: the opaque winner to the screen and the depth
// buffer, the transparent layers in front of it merged into the first one
// (viewport_t::flatten(front, back), viewport.cpp:43-51), `l0`.  ORIGIN: the
// view lies at the surface's top left, so its flatten and copy passes
// (k_flatten, k_copy_layer) read and write this pixel: made here.
template <bool ORIGIN>
__device__ __forceinline__ void write_pixel(const ItemDev &it, uint32_t i, uint32_t wz, uint32_t wc, uint32_t l0)
{
    const uint32_t w = (uint32_t)it.v.w, y = i / w, x = i - y * w;
    if (ORIGIN)
        wc = (l0 >> 24) ? blend_px(wc, l0) : wc;
    else
        it.layer0[i] = l0;
    it.pixels[(long long)y * it.pitch_px + x] = wc; // 0 = viewport_t::clear's background
    if (it.zbuf)
        it.zbuf[i] = __uint_as_float(wz);
}

// One pixel whose fragments are shaded: one run over its chain for the nearest
// opaque (the first drawn of equal depth), one for the transparent ones in
// front of it, kept nearest first (of equal depth the last drawn).  `first`:
// the second half of its head fragment (depth, slot, next, colour).
template <bool ORIGIN>
__device__ __forceinline__ void resolve_shaded(const BatchDev *b, const ItemDev &it, uint32_t i, uint4 first)
{
    const Frag *pool = b->frags;
    unsigned long long opaque = ((unsigned long long)kMaxZBits << 32) | 0xFFFFFFFFull;
    uint32_t wc = 0u, l0 = 0u, lone = 0u;
    int clear = 0; // transparent fragments, the last one's depth and colour
    for (uint4 m = first;;) {
        const unsigned long long key = ((unsigned long long)m.x << 32) | m.y;
        if ((m.w >> 24) != 255u) {
            clear++;
            lone = m.x;
            l0 = m.w;
        } else if (key < opaque) {
            opaque = key;
            wc = m.w;
        }
        if (m.z == kFragEnd)
            break;
        m = reinterpret_cast<const uint4 *>(pool + m.z)[1];
    }
    const uint32_t wz = (uint32_t)(opaque >> 32);
    if (clear == 1) { // most pixels: no order to find (30.7 -> 26.6 us)
        l0 = lone < wz ? l0 : 0u;
    } else if (clear) {
        l0 = 0u;
        unsigned long long lk[SGL_MAX_LAYERS]; // kept, nearest first: depth, then the complement of the slot
        uint32_t lc[SGL_MAX_LAYERS];
#pragma unroll
        for (int k = 0; k < SGL_MAX_LAYERS; k++) {
            lk[k] = ~0ull;
            lc[k] = 0u;
        }
        const int n_layers = it.layers;
        for (uint4 m = first;;) {
            if ((m.w >> 24) != 255u && m.x < wz) {
                unsigned long long key = ((unsigned long long)m.x << 32) | (uint32_t)~m.y;
                uint32_t c = m.w;
#pragma unroll
                for (int k = 0; k < SGL_MAX_LAYERS; k++)
                    if (k < n_layers && key < lk[k]) {
                        const unsigned long long tk = lk[k];
                        const uint32_t tc = lc[k];
                        lk[k] = key;
                        lc[k] = c;
                        key = tk;
                        c = tc;
                    }
            }
            if (m.z == kFragEnd)
                break;
            m = reinterpret_cast<const uint4 *>(pool + m.z)[1];
        }
        // the farthest kept is the first layer, the nearer ones blend onto it
        // (an unused place holds 0, which blends nothing)
#pragma unroll
        for (int k = SGL_MAX_LAYERS - 1; k >= 0; k--)
            if (lk[k] != ~0ull)
                l0 = (k == SGL_MAX_LAYERS - 1 || lk[k + 1 < SGL_MAX_LAYERS ? k + 1 : k] == ~0ull)
                         ? lc[k]
                         : ((lc[k] >> 24) ? blend_px(l0, lc[k]) : l0);
    }
    write_pixel<ORIGIN>(it, i, wz, wc, l0);
}

// One pixel whose fragments are not shaded yet: they are taken nearest first
// and shaded until one is opaque.
template <bool ALL_MODES, bool ORIGIN>
__device__ __forceinline__ void resolve_on_demand(const BatchDev *b, const ItemDev &it, uint32_t i)
{
    const int n_layers = it.layers;
    const Frag *pool = b->frags;
    const uint32_t head = it.frag_head[i];
    uint32_t lz[SGL_MAX_LAYERS], ls[SGL_MAX_LAYERS], lc[SGL_MAX_LAYERS]; // kept, nearest first
    int nt = 0;
    uint32_t wz = kMaxZBits, wc = 0u;
    unsigned long long prev = 0ull;
    bool first = true;
    // the first kChainRegs fragments of the chain are held in registers
    constexpr int kChainRegs = 4;
    unsigned long long ck[kChainRegs];
    uint32_t cf[kChainRegs];
    int held = 0;
    uint32_t rest = head; // the chain beyond the held fragments
#pragma unroll
    for (int k = 0; k < kChainRegs; k++) {
        if (rest != kFragEnd) {
            const uint4 m = reinterpret_cast<const uint4 *>(pool + rest)[1];
            ck[k] = ((unsigned long long)m.x << 32) | m.y;
            cf[k] = rest;
            held = k + 1;
            rest = m.z;
        }
    }
    for (;;) {
        // the next fragment in (depth, draw order)
        unsigned long long best = ~0ull;
        uint32_t bi = kFragEnd;
#pragma unroll
        for (int k = 0; k < kChainRegs; k++)
            if (k < held && (first || ck[k] > prev) && ck[k] < best) {
                best = ck[k];
                bi = cf[k];
            }
        for (uint32_t f = rest; f != kFragEnd;) {
            const uint4 m = reinterpret_cast<const uint4 *>(pool + f)[1];
            const unsigned long long key = ((unsigned long long)m.x << 32) | m.y;
            if ((first || key > prev) && key < best) {
                best = key;
                bi = f;
            }
            f = m.z;
        }
        if (bi == kFragEnd)
            break;
        first = false;
        prev = best;
        const uint32_t z = (uint32_t)(best >> 32), slot = (uint32_t)best;
        const uint32_t c = shade_frag<ALL_MODES>(b, it, 0u, slot, reinterpret_cast<const float4 *>(pool + bi)[0]);
        if ((c >> 24) == 255u) {
            wz = z;
            wc = c;
            while (nt > 0 && lz[nt - 1] == z)
                nt--; // not strictly in front
            break;
        }
        if (nt == n_layers && (z > lz[nt - 1] || (z == lz[nt - 1] && slot < ls[nt - 1])))
            continue; // farther than every kept layer
        int k = nt < n_layers ? nt : n_layers - 1;
        while (k > 0 && (lz[k - 1] > z || (lz[k - 1] == z && ls[k - 1] < slot))) {
            lz[k] = lz[k - 1];
            ls[k] = ls[k - 1];
            lc[k] = lc[k - 1];
            k--;
        }
        lz[k] = z;
        ls[k] = slot;
        lc[k] = c;
        if (nt < n_layers)
            nt++;
    }
    uint32_t l0 = nt > 0 ? lc[nt - 1] : 0u;
    for (int k = 1; k < nt; k++) {
        const uint32_t f = lc[nt - 1 - k];
        if (f >> 24)
            l0 = blend_px(l0, f);
    }
    write_pixel<ORIGIN>(it, i, wz, wc, l0);
    it.frag_head[i] = kFragEnd;
}

// Per pixel of the layered view (list heads are left empty for the next):
// pixels without fragments get the background at once, the others are resolved, those with fragments to shade queued in
// shared memory for full warps.
template <bool ALL_MODES, bool ORIGIN>
__global__ void __launch_bounds__(256, 4) k_layers(const BatchDev *b)
{
    if (frags_overflowed(b))
        return;
    const ItemDev &it = b->items[0];
    const uint32_t total = (uint32_t)it.v.w * (uint32_t)it.v.h;
    if (!frags_on_demand(b, it)) {
        // (a pixel's list head is loaded two turns ahead and its first fragment
        // one, so that a turn waits for neither: 26.6 -> 23.5 us; four consecutive
        // pixels a thread, with 16-byte accesses, 41.6 us)
        uint32_t *head = it.frag_head;
        const uint32_t step = gridDim.x * 256u;
        uint32_t i = blockIdx.x * 256u + threadIdx.x;
        auto fragment = [&](uint32_t f) {
            return f != kFragEnd ? reinterpret_cast<const uint4 *>(b->frags + f)[1] : make_uint4(0u, 0u, kFragEnd, 0u);
        };
        uint32_t h = i < total ? head[i] : kFragEnd, h1 = i + step < total ? head[i + step] : kFragEnd;
        uint4 m = fragment(h);
        for (; i < total; i += step) {
            const uint4 m1 = fragment(h1);
            const uint32_t h2 = i + 2 * step < total ? head[i + 2 * step] : kFragEnd;
            if (h == kFragEnd) {
                write_pixel<ORIGIN>(it, i, kMaxZBits, 0u, 0u);
            } else {
                resolve_shaded<ORIGIN>(b, it, i, m);
                head[i] = kFragEnd;
            }
            h = h1;
            m = m1;
            h1 = h2;
        }
        return;
    }
    __shared__ uint32_t queue[2 * 256];
    __shared__ int qn;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0)
        qn = 0;
    __syncthreads();
    for (uint32_t c0 = blockIdx.x * 256u; c0 < total; c0 += gridDim.x * 256u) {
        const uint32_t i = c0 + threadIdx.x;
        bool busy = false;
        if (i < total) {
            if (it.frag_head[i] == kFragEnd)
                write_pixel<ORIGIN>(it, i, kMaxZBits, 0u, 0u);
            else
                busy = true;
        }
        const unsigned m = __ballot_sync(0xFFFFFFFFu, busy);
        int wb = 0;
        if (lane == 0 && m)
            wb = atomicAdd(&qn, __popc(m));
        wb = __shfl_sync(0xFFFFFFFFu, wb, 0);
        if (busy)
            queue[wb + __popc(m & ((1u << lane) - 1u))] = i;
        __syncthreads();
        const int have = qn;
        if (have >= 256) {
            resolve_on_demand<ALL_MODES, ORIGIN>(b, it, queue[threadIdx.x]);
            __syncthreads();
            if ((int)threadIdx.x < have - 256)
                queue[threadIdx.x] = queue[256 + threadIdx.x];
            __syncthreads();
            if (threadIdx.x == 0)
                qn = have - 256;
        }
        __syncthreads();
    }
    if ((int)threadIdx.x < qn)
        resolve_on_demand<ALL_MODES, ORIGIN>(b, it, queue[threadIdx.x]);
}

// viewport_t::flatten(front) (viewport.cpp:53-79): view pixel (x, y) reads
// the surface at row y, column x.
__global__ void __launch_bounds__(256) k_flatten(const BatchDev *b)
{
    if (frags_overflowed(b))
        return;
    const ItemDev &it = b->items[0];
    const int w = it.v.w;
    const uint32_t total = (uint32_t)w * (uint32_t)it.v.h;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int y = (int)(i / (uint32_t)w), x = (int)(i - (uint32_t)y * (uint32_t)w);
        const uint32_t back = it.surface[(long long)y * it.pitch_px + x];
        const uint32_t f = it.layer0[i];
        it.layer0[i] = (f >> 24) ? blend_px(back, f) : back;
    }
}

// post_shader_t::copy_first_transparency_layer_to_screen
// (post_shaders.hpp:22-31): view pixel (x, y) to surface row y + view y,
// column x.
__global__ void __launch_bounds__(256) k_copy_layer(const BatchDev *b)
{
    if (frags_overflowed(b))
        return;
    const ItemDev &it = b->items[0];
    const int w = it.v.w;
    const uint32_t total = (uint32_t)w * (uint32_t)it.v.h;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int y = (int)(i / (uint32_t)w), x = (int)(i - (uint32_t)y * (uint32_t)w);
        it.surface[(long long)(y + it.v.y) * it.pitch_px + x] = it.layer0[i];
    }
}

// ---------------------------------------------------------------- launches --

static inline unsigned grid_for(uint64_t n, int block) { return (unsigned)((n + block - 1) / block); }

static int sm_count()
{
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
            n = 132;
    }
    return n;
}

cudaError_t launch_world(const SceneDev &s, bool uploaded, float4 *lbox, cudaStream_t st)
{
    if (s.n_vertices == 0)
        return cudaSuccess;
    k_world<<<grid_for(s.n_vertices, 256), 256, 0, st>>>(s);
    const unsigned boxes = s.pbox ? grid_for((uploaded ? 2ull : 1ull) * s.n_prims, 8) : 0u,
                   samples = uploaded ? grid_for(s.n_triangles, 256) : 0u;
    if (boxes + samples)
        k_box<<<boxes + samples, 256, 0, st>>>(s, uploaded ? lbox : nullptr, boxes);
    return cudaGetLastError();
}

cudaError_t launch_poses(const PoseDev *poses, int n, uint32_t vertex_blocks, uint32_t prim_blocks, cudaStream_t st)
{
    if (vertex_blocks + prim_blocks)
        k_pose<<<vertex_blocks + prim_blocks, 256, 0, st>>>(poses, n, vertex_blocks);
    return cudaGetLastError();
}

const char *prof_kernel_name(int k)
{
    static const char *names[kProfKernels] = {"k_geom",    "k_vertex",  "k_flags",  "k_compact", "k_walk",
                                                 "k_spans",   "k_winners", "k_shade",  "k_dof",
                                              "k_frags",   "k_layers",  "k_flatten", "k_copy_layer"};
    return (k >= 0 && k < kProfKernels) ? names[k] : "?";
}

// Fold the previous launch sequence's event timings into the totals.
static void prof_collect(Profiler *p)
{
    if (!p || !p->pending)
        return;
    if (cudaEventSynchronize(p->ev[kProfKernels]) == cudaSuccess) {
        for (int k = 0; k < kProfKernels; k++) {
            float ms = 0.0f;
            if (!(p->ran & (1u << k)))
                continue; // a stage this sequence skipped
            if (cudaEventElapsedTime(&ms, p->ev[k], p->ev[k + 1]) == cudaSuccess) {
                p->ms[k] += ms;
                p->launches[k]++;
            }
        }
    }
    cudaGetLastError();
    p->pending = false;
}

void prof_flush(Profiler *p) { prof_collect(p); }

// The fixed launch sequence of a batch.  Grids do not depend on the batch:
// every kernel strides over totals it reads from device memory.
// Constant tables of the current device (the depth-of-field taps); called
// before any launch or graph capture on that device.
cudaError_t init_device_constants()
{
    float2 taps[SGL_DOF_TAPS];
    for (int k = 0; k < SGL_DOF_TAPS; k++)
        taps[k] = make_float2(sgl_dof_taps[k][0], sgl_dof_taps[k][1]);
    cudaError_t e = cudaMemcpyToSymbol(c_dof_taps, taps, sizeof taps);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_geom, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGeomSmem);
    return e;
}

cudaError_t check_status(unsigned *code, unsigned long long *index, unsigned *count, bool reset, bool *compiled)
{
#ifdef SGL_BOUNDS_CHECK
    *compiled = true;
    unsigned long long first = 0;
    unsigned n = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&first, g_check_first, sizeof first);
    if (e == cudaSuccess)
        e = cudaMemcpyFromSymbol(&n, g_check_count, sizeof n);
    if (e == cudaSuccess && reset) {
        const unsigned long long z0 = 0;
        const unsigned z1 = 0;
        e = cudaMemcpyToSymbol(g_check_first, &z0, sizeof z0);
        if (e == cudaSuccess)
            e = cudaMemcpyToSymbol(g_check_count, &z1, sizeof z1);
    }
    *code = (unsigned)(first >> 48);
    *index = first & 0xFFFFFFFFFFFFull;
    *count = n;
    return e;
#else
    *compiled = false;
    *code = 0;
    *index = 0;
    *count = 0;
    (void)reset;
    return cudaSuccess;
#endif
}

cudaError_t launch_dof(const BatchDev *b, cudaStream_t st)
{
    k_dof<<<sm_count() * kDofBlocks, 256, 0, st>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_batch(const BatchDev *b, int tile, int flags, cudaStream_t st, int *launches, Profiler *prof)
{
    const bool timed = prof && prof->enabled;
    if (timed) {
        prof_collect(prof);
        for (int k = 0; k <= kProfKernels; k++)
            if (!prof->ev[k] && cudaEventCreate(&prof->ev[k]) != cudaSuccess)
                return cudaGetLastError();
    }
    if (timed)
        prof->ran = 0;
    auto mark = [&](int k) {
        if (timed)
            cudaEventRecord(prof->ev[k], st);
    };
    auto ran = [&](int k) {
        if (timed)
            prof->ran |= 1u << k;
    };
    const int sms = sm_count();
    int n = 0;
    mark(PK_GEOM);
    if (flags & kSeqFused) {
        k_geom<<<sms * kGeomBlocks * 8, kGeomWarps * 32, kGeomSmem, st>>>(b);
        ran(PK_GEOM);
        n++;
    }
    mark(PK_VERTEX);
    if (flags & kSeqSplit) {
        k_vertex<<<sms * 8, 256, 0, st>>>(b);
        ran(PK_VERTEX);
        mark(PK_FLAGS);
        k_flags<<<sms * 8, 256, 0, st>>>(b);
        ran(PK_FLAGS);
        mark(PK_COMPACT);
        k_compact<<<sms * 4, kCompactBlock, 0, st>>>(b);
        ran(PK_COMPACT);
        n += 3;
    } else {
        mark(PK_FLAGS);
        mark(PK_COMPACT);
    }
    if (flags & kSeqLayers) {
        for (int k = PK_WALK; k <= PK_DOF; k++)
            mark(k);
        mark(PK_FRAGS);
        k_walk<true, true><<<sms * SGL_WALK_MIN_BLOCKS, kWalkWarps * 32, 0, st>>>(b); // (one view)
        k_frags<<<sms * 2, 256, 0, st>>>(b);
        k_frag_spans<<<sms * 4, 256, 0, st>>>(b);
        const unsigned lg = sms * SGL_SHADE_MIN_BLOCKS;
        if (flags & kSeqShaders)
            k_link<true><<<lg, 256, 0, st>>>(b);
        else
            k_link<false><<<lg, 256, 0, st>>>(b);
        ran(PK_FRAGS);
        mark(PK_LAYERS);
        if (flags & kSeqShaders) {
            if (flags & kSeqOrigin)
                k_layers<true, true><<<sms * 4, 256, 0, st>>>(b);
            else
                k_layers<true, false><<<sms * 4, 256, 0, st>>>(b);
        } else {
            if (flags & kSeqOrigin)
                k_layers<false, true><<<sms * 4, 256, 0, st>>>(b);
            else
                k_layers<false, false><<<sms * 4, 256, 0, st>>>(b);
        }
        ran(PK_LAYERS);
        n += 5;
        mark(PK_FLATTEN);
        if (!(flags & kSeqOrigin)) {
            k_flatten<<<sms * 8, 256, 0, st>>>(b);
            ran(PK_FLATTEN);
            n++;
        }
        mark(PK_COPY);
        if (!(flags & kSeqOrigin)) {
            k_copy_layer<<<sms * 8, 256, 0, st>>>(b);
            ran(PK_COPY);
            n++;
        }
        if (flags & kSeqDof) { // the gather over the view's rectangle, from a copy of it (timed with the copy)
            k_dof_source<<<sms * 8, 256, 0, st>>>(b);
            k_dof<<<sms * kDofBlocks, 256, 0, st>>>(b);
            n += 2;
        }
        if (timed) {
            cudaEventRecord(prof->ev[kProfKernels], st);
            prof->pending = true;
        }
        if (launches)
            *launches += n;
        return cudaGetLastError();
    }
    mark(PK_WALK);
    if (flags & kSeqOne)
        k_walk<false, true><<<sms * SGL_WALK_MIN_BLOCKS, kWalkWarps * 32, 0, st>>>(b);
    else
        k_walk<false, false><<<sms * SGL_WALK_MIN_BLOCKS, kWalkWarps * 32, 0, st>>>(b);
    ran(PK_WALK);
    n++;
    mark(PK_SPANS);
    k_spans<<<sms * 4, 256, 0, st>>>(b);
    ran(PK_SPANS);
    n++;
    mark(PK_WINNER);
    if (!(flags & kSeqWinList)) { // (else by k_classify)
        k_winners<<<sms * 4, 256, 0, st>>>(b);
        ran(PK_WINNER);
        n++;
    }
    mark(PK_SHADE);
    // the kernel with every pixel shader only when a view asks for another
    // than the default, which then keeps all the registers
    const unsigned sg = sms * ((flags & kSeqWinList) ? SGL_SHADE_MIN_BLOCKS : SGL_TILE_MIN_BLOCKS);
    if (flags & kSeqWinList) {
        k_classify<<<sms * 4, 256, 0, st>>>(b);
        if (flags & kSeqShaders)
            k_shade_wins<true><<<sg, kShadeThreads, 0, st>>>(b);
        else
            k_shade_wins<false><<<sg, kShadeThreads, 0, st>>>(b);
        n++;
    } else if (flags & kSeqShaders) {
        if (tile == 8)
            k_shade<8, true><<<sg, kShadeThreads, 0, st>>>(b);
        else if (tile == 32)
            k_shade<32, true><<<sg, kShadeThreads, 0, st>>>(b);
        else
            k_shade<16, true><<<sg, kShadeThreads, 0, st>>>(b);
    } else {
        if (tile == 8)
            k_shade<8, false><<<sg, kShadeThreads, 0, st>>>(b);
        else if (tile == 32)
            k_shade<32, false><<<sg, kShadeThreads, 0, st>>>(b);
        else
            k_shade<16, false><<<sg, kShadeThreads, 0, st>>>(b);
    }
    ran(PK_SHADE);
    n++;
    mark(PK_DOF);
    if (flags & kSeqDof) {
        k_dof<<<sms * kDofBlocks, 256, 0, st>>>(b);
        ran(PK_DOF);
        n++;
    }
    for (int k = PK_FRAGS; k <= PK_COPY; k++)
        mark(k);
    if (timed) {
        cudaEventRecord(prof->ev[kProfKernels], st);
        prof->pending = true;
    }
    if (launches)
        *launches += n;
    return cudaGetLastError();
}

} // namespace sgl
