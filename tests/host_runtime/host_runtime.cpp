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

// Calls that fail after their staging was handed to an asynchronous copy, and
// the same calls again.
static int failures()
{
    const int id = upload();
    cudaStream_t a = test_stream();
    fake::overwritten = 0;
    for (int k = 0; k < 4; k++) {
        fake::fail_on = k % 2 ? "" : "launch_dof";
        sgl_view v = view_of(64 + k, 48);
        v.dof.enabled = 1, v.dof.max_radius = 4.0f;
        const sgl_target t = target_of(64 + k, 48);
        if ((sgl_dof(ctx, &v, &t, &t, 1, a) == SGL_OK) != (k % 2 == 1))
            return 2;
    }
    fake::drain_all();
    const long dof = fake::overwritten;
    for (int k = 0; k < 16; k++) {
        fake::fail_on = k < 12 ? (k % 2 ? "cudaGraphLaunch" : "launch_batch") : "";
        if ((batch(id, a, k % 3 == 0, k % 2 != 0) == SGL_OK) != (k >= 12))
            return 2;
    }
    fake::drain_all();
    const long batches = fake::overwritten - dof;
    // posed requests: the first fails when its sequence is launched
    fake::auto_progress = true;
    const sgl_serve_opts opts{0, 4, 1, 0};
    sgl_server *srv = nullptr;
    if (sgl_server_create(ctx, &opts, &srv) != SGL_OK)
        return 2;
    for (int k = 0; k < 4; k++) {
        sgl_node_desc node{};
        node.scale[0] = node.scale[1] = node.scale[2] = 1.0f;
        node.parent = -1;
        node.translation[0] = (float)k;
        sgl_request req{};
        req.scene_id = id, req.view = view_of(64, 48);
        req.nodes = &node, req.n_nodes = 1;
        uint64_t ticket = 0;
        sgl_request_result res{};
        fake::fail_on = k % 2 ? "" : "cudaGraphLaunch";
        if (sgl_server_submit(srv, &req, &ticket) != SGL_OK || sgl_server_wait(srv, ticket, 60.0, &res) != SGL_OK ||
            (res.status == SGL_OK) != (k % 2 == 1))
            return 2;
    }
    sgl_server_destroy(srv);
    fake::drain_all();
    printf("%ld %ld %ld\n", dof, batches, fake::overwritten - dof - batches);
    return 0;
}

// One request on a server whose budget is the least that admits it: the device
// bytes that it allocates beyond the budget, without and with depth of field,
// then with the budget of two and with four times as much.
static int budget()
{
    const int id = upload();
    fake::auto_progress = true;
    for (int k = 0; k < 4; k++) {
        sgl_request req{};
        req.scene_id = id, req.view = view_of(1000, 1000);
        req.view.dof.enabled = k > 0, req.view.dof.max_radius = 8.0f;
        uint64_t lo = 0, hi = 1ull << 32; // refused, admitted
        auto serve = [&](uint64_t bytes, long long *over) {
            const sgl_serve_opts opts{bytes, 4, 1, 0};
            sgl_server *srv = nullptr;
            uint64_t ticket = 0;
            sgl_request_result res{};
            if (sgl_server_create(ctx, &opts, &srv) != SGL_OK)
                exit(2);
            const size_t before = fake::peak = fake::live;
            const bool in = sgl_server_submit(srv, &req, &ticket) == SGL_OK;
            if (in && over) {
                if (sgl_server_wait(srv, ticket, 60.0, &res) != SGL_OK || res.status != SGL_OK)
                    exit(2);
                *over = (long long)(fake::peak - before) - (long long)bytes;
            }
            sgl_server_destroy(srv);
            return in;
        };
        while (hi - lo > 1) {
            const uint64_t mid = lo + (hi - lo) / 2;
            (serve(mid, nullptr) ? hi : lo) = mid;
        }
        long long over = 0;
        serve(k == 2 ? 2 * hi : (k == 3 ? 4 * hi : hi), &over);
        printf("%lld ", over);
    }
    printf("\n");
    return 0;
}

// Device allocations, copies and launches of an upload (a launch_* call counts
// once).
static int uploads()
{
    upload();
    const long before = fake::device_calls;
    upload();
    printf("%ld\n", fake::device_calls - before);
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
    else if (argc > 1 && !strcmp(argv[1], "failures"))
        r = failures();
    else if (argc > 1 && !strcmp(argv[1], "budget"))
        r = budget();
    else if (argc > 1 && !strcmp(argv[1], "uploads"))
        r = uploads();
    fake::auto_progress = true;
    sgl_destroy(ctx);
    return r;
}
