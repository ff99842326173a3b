// Scenarios over the library's host sources on the stand-in for the CUDA
// runtime (fake_cuda.h).  Each prints the counts that its test reads.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

#include "fake_cuda.h"
#include "sgl.h"

cudaStream_t test_stream();

static sgl_ctx *ctx;

static int upload()
{
    static const float pos[] = {0, 0, 0, 1, 0, 0, 0, 1, 0}, nrm[] = {0, 0, 1, 0, 0, 1, 0, 0, 1},
                       uv[] = {0, 0, 1, 0, 0, 1};
    static const uint32_t idx[] = {0, 1, 2}, texel[] = {0xFFFFFFFFu};
    sgl_node_desc node{};
    node.scale[0] = node.scale[1] = node.scale[2] = 1.0f;
    for (int k = 0; k < 4; k++)
        node.rotation[5 * k] = 1.0f;
    node.parent = -1;
    sgl_primitive_desc prim{0, SGL_TRIANGLES, 0, 0, 3, 0, 3};
    sgl_material_desc mat{0xFFFFFFFFu, 0, 0, 32};
    sgl_texture_desc tex{texel, 1, 1};
    sgl_scene_desc d{};
    d.n_nodes = d.n_primitives = d.n_materials = d.n_textures = 1;
    d.nodes = &node, d.primitives = &prim, d.materials = &mat, d.textures = &tex;
    d.n_vertices = d.n_indices = 3;
    d.positions = pos, d.normals = nrm, d.uvs = uv, d.indices = idx;
    d.default_material = mat;
    int id = 0;
    if (sgl_scene_upload(ctx, &d, &id) != SGL_OK)
        exit(2);
    return id;
}

static sgl_view view_of(int w, int h)
{
    sgl_view v{};
    v.w = w, v.h = h;
    for (int k = 0; k < 4; k++)
        v.view[5 * k] = v.proj[5 * k] = 1.0f;
    return v;
}

static std::vector<uint32_t> pixels(1 << 20);
static std::vector<float> depth(1 << 20);
static sgl_target target_of(int w, int h) { return sgl_target{pixels.data(), 4 * w, w, h, depth.data()}; }

static sgl_status frame(int id, cudaStream_t st, int w = 64, int h = 48)
{
    const sgl_view v = view_of(w, h);
    const sgl_target t = target_of(w, h);
    return sgl_render(ctx, id, &v, &t, 1, 1, st, nullptr);
}

static sgl_status batch(int id, cudaStream_t st, bool posed, bool graph = true)
{
    sgl_node_desc node{};
    node.scale[0] = node.scale[1] = node.scale[2] = 1.0f;
    node.parent = -1;
    static int turn = 0;
    node.translation[0] = (float)turn++; // another pose each time
    std::vector<sgl_batch_item> items(3);
    for (auto &it : items) {
        it.scene_id = id;
        it.view = view_of(64, 48);
        it.target = target_of(64, 48);
        it.nodes = posed ? &node : nullptr;
        it.n_nodes = posed ? 1 : 0;
    }
    const sgl_batch_opts o{0, 0, graph ? 1 : 0};
    return sgl_render_batch(ctx, items.data(), (int)items.size(), &o, st, nullptr);
}

// Calls on alternating streams without a wait of the caller's between them.
static int streams()
{
    const int id = upload();
    cudaStream_t a = test_stream(), b = test_stream();
    fake::unordered = 0;
    for (int k = 0; k < 6; k++) {
        if (frame(id, k & 1 ? b : a) != SGL_OK || batch(id, k & 1 ? a : b, k % 3 == 0) != SGL_OK)
            return 2;
    }
    sgl_batch_item it{};
    it.scene_id = id, it.view = view_of(64, 48), it.target = target_of(64, 48);
    sgl_batch_opts o{};
    if (frame(id, b) != SGL_OK || sgl_autotune(ctx, &it, 1, &o) != SGL_OK || frame(id, a) != SGL_OK)
        return 2;
    printf("%ld\n", fake::unordered);
    return 0;
}

// A context first used on the legacy default stream, then on its caller's and
// on its own (the tuner): only streams that it made are destroyed, once.
static int ownership()
{
    const int id = upload();
    cudaStream_t a = test_stream();
    sgl_batch_item it{};
    it.scene_id = id, it.view = view_of(64, 48), it.target = target_of(64, 48);
    sgl_batch_opts o{};
    if (frame(id, nullptr) != SGL_OK || frame(id, a) != SGL_OK)
        return 2;
    sgl_ctx *first = ctx;
    if (sgl_create(&ctx, 0) != SGL_OK)
        return 2;
    it.scene_id = upload();
    if (frame(it.scene_id, nullptr) != SGL_OK || sgl_autotune(ctx, &it, 1, &o) != SGL_OK)
        return 2;
    sgl_destroy(ctx);
    sgl_destroy(first);
    ctx = nullptr;
    printf("%ld %ld\n", fake::foreign_streams_destroyed, fake::streams_destroyed_twice);
    return 0;
}

int main(int argc, char **argv)
{
    if (sgl_create(&ctx, 0) != SGL_OK)
        return 2;
    int r = 2;
    if (argc > 1 && !strcmp(argv[1], "streams"))
        r = streams();
    else if (argc > 1 && !strcmp(argv[1], "ownership"))
        r = ownership();
    fake::auto_progress = true;
    sgl_destroy(ctx);
    return r;
}
