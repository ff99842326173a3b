"""The renderer's work as its users have it done, as timed cases.

Every case goes through the C ABI (include/sgl.h), with the descriptors packed
beforehand as a C or C++ program holds them: single frames into device or host
buffers, batches of views, posed batches, the serving loop, frames with
transparency layers, the allocation-free call and the depth-of-field gather
alone.  Scenes are the repository's seeded ones (swegl_gb300/scenes.py) and a
heightfield of one large triangle list.

exact() rasterises the same triangles in 64 bits for the depth outputs;
colours are whole bytes.
"""
import ctypes as C
import math

import numpy as np
import torch

from swegl_gb300 import abi
from swegl_gb300 import scenes as S
from swegl_gb300.runtime import Renderer, Server, host_buffer

FAR = float(np.array(0x7F7F7F7F, np.uint32).view(np.float32))  # cleared depth
NEAR = 0.001


def listed():
    return [
        # the smallest frame: a textured cube in a small window, where launches and latency count
        {"name": "cube_640x480", "kind": "cube", "w": 640, "h": 480},
        # a viewer that does without per-pixel lighting: flat light, bilinear texture, odd window, 50k triangles
        {"name": "flat_1283x719", "kind": "frame", "spheres": 13, "w": 1283, "h": 719, "shader": 2, "dof": False},
        # the ordinary frame: 819,200 triangles, 8 textures, sun and 4 point lights, Phong and bilinear, 1080p
        {"name": "spheres_1080p", "kind": "frame", "spheres": 200, "w": 1920, "h": 1080, "shader": 0, "dof": False},
        # the large frame: the same scene at 4K with depth of field
        {"name": "spheres_4k_dof", "kind": "frame", "spheres": 200, "w": 3840, "h": 2160, "shader": 0, "dof": True},
        # one large triangle list seen by a camera standing on it: a terrain, crossing the near plane
        {"name": "terrain_1080p", "kind": "terrain", "cells": 512, "w": 1920, "h": 1080},
        # translucent objects: 4 transparency layers over block-alpha textures
        {"name": "layers_1080p", "kind": "layers", "spheres": 200, "layers": 4, "w": 1920, "h": 1080},
        # many cameras on one scene in one call: 64 views of uneven size
        {"name": "batch_64_views", "kind": "batch", "spheres": 200, "views": 64, "w": 1920, "h": 1080, "posed": False},
        # an animated scene at many times in one call: every view with its own pose
        {"name": "posed_16_views", "kind": "batch", "spheres": 50, "views": 16, "w": 640, "h": 640, "posed": True},
        # a render service: requests of several scenes and sizes, half with depth of field, frames to the host
        {"name": "serve_48_requests", "kind": "serve", "requests": 48, "w": 3840, "h": 2160},
        # a frame callback that may not allocate
        {"name": "noalloc_960x540", "kind": "noalloc", "spheres": 25, "w": 960, "h": 540},
        # the drop-in render call: two viewports side by side on one host surface
        {"name": "splitscreen_host_720p", "kind": "host", "spheres": 25, "w": 1280, "h": 720},
        # the post pass alone on a frame the program already has, with a wide circle of confusion
        {"name": "dof_pass_1440p", "kind": "dof", "w": 2560, "h": 1440, "radius": 24.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cube", "frame", "frame", "frame", "terrain", "layers", "batch", "batch", "serve", "noalloc",
                       "host", "dof"])
    if kind == "cube":
        return {"kind": kind, "w": _log(rng, 64, 2560), "h": _log(rng, 64, 1440)}
    if kind == "frame":
        dof = rng.random() < 0.5
        return {"kind": kind, "spheres": _log(rng, 2, 200), "w": _log(rng, 64, 3840), "h": _log(rng, 64, 2160),
                "shader": rng.choice([0, 0, 0, 0, 1, 2, 3, 4, 5, 6, 7, 8]), "dof": dof}
    if kind == "terrain":
        return {"kind": kind, "cells": _log(rng, 24, 512), "w": _log(rng, 128, 1920), "h": _log(rng, 128, 1080)}
    if kind == "layers":
        return {"kind": kind, "spheres": _log(rng, 4, 200), "layers": rng.randint(1, 8), "w": _log(rng, 128, 1920),
                "h": _log(rng, 128, 1080)}
    if kind == "batch":
        posed = rng.random() < 0.5
        return {"kind": kind, "spheres": _log(rng, 2, 50 if posed else 200), "views": _log(rng, 2, 16 if posed else 64),
                "w": _log(rng, 160, 640 if posed else 1920), "h": _log(rng, 160, 640 if posed else 1080),
                "posed": posed}
    if kind == "serve":
        return {"kind": kind, "requests": _log(rng, 2, 48), "w": _log(rng, 256, 3840), "h": _log(rng, 256, 2160)}
    if kind == "noalloc":
        return {"kind": kind, "spheres": _log(rng, 2, 25), "w": _log(rng, 64, 960), "h": _log(rng, 64, 540)}
    if kind == "host":
        return {"kind": kind, "spheres": _log(rng, 2, 25), "w": 2 * _log(rng, 64, 640), "h": _log(rng, 64, 720)}
    return {"kind": kind, "w": _log(rng, 64, 2560), "h": _log(rng, 64, 1440),
            "radius": float(rng.choice([4.0, 8.5, 16.0, 24.0, 31.5, 48.0]))}


# ---------------------------------------------------------------- scenes --

SERVED = (3, 25, 123, 293)  # spheres of the serving scenes: 12k, 102k, 504k and 1.2M triangles
DEVICE = torch.device("cuda", 0)
_program = {}  # what one program holds once: the renderer and its stream


def _renderer():
    if "r" not in _program:
        _program["r"] = Renderer(0)
        _program["stream"] = torch.cuda.Stream(DEVICE)
    return _program["r"]


def _textures(seed, n=8, size=1024, alpha=False):
    """Tileable value noise in four octaves, per channel (or random texels with alpha constant over 8 x 8 squares)."""
    g = torch.Generator().manual_seed(seed)
    out = []
    for _ in range(n):
        if alpha:
            rgb = torch.randint(0, 256, (3, size, size), generator=g)
            cell = torch.randint(0, 8, (size // 8, size // 8), generator=g)
            a = torch.where(cell == 0, 0, torch.where(cell <= 3, 255, torch.randint(1, 255, cell.shape, generator=g)))
            a = a.repeat_interleave(8, 0).repeat_interleave(8, 1)
        else:
            total, amp = torch.zeros(3, size, size, device=DEVICE), 0.0
            for o in range(4):
                cells = 4 << o
                lat = torch.rand(1, 3, cells, cells, generator=g).to(DEVICE)
                lat = torch.cat([lat, lat[..., :1]], -1)
                lat = torch.cat([lat, lat[..., :1, :]], -2)
                step = size // cells
                up = torch.nn.functional.interpolate(lat, size=(size + step, size + step), mode="bilinear",
                                                     align_corners=False)
                total += 0.5 ** o * up[0, :, step // 2:step // 2 + size, step // 2:step // 2 + size]
                amp += 0.5 ** o
            rgb = (total / amp * 256.0).clamp_(0, 255).to(torch.int64).cpu()
            a = torch.full((size, size), 255)
        texel = (a.to(torch.int64) << 24) | (rgb[0] << 16) | (rgb[1] << 8) | rgb[2]
        out.append(texel.numpy().astype(np.uint32))
    return out


def _spheres(n, seed, textures):
    return S.spheres_scene(n_spheres=n, seed=seed, textures=textures)


def _terrain(cells, seed):
    """A heightfield of cells x cells quads as one triangle list, 40 units wide, camera height 0.4 above its middle."""
    rng = np.random.RandomState(seed % (1 << 31))
    g = np.linspace(-20.0, 20.0, cells + 1)
    x, z = np.meshgrid(g, g)
    ph, fr = rng.uniform(0, 6.28, (6, 2)), rng.uniform(0.2, 1.2, (6, 2))
    y = sum(0.25 * np.sin(fr[k, 0] * x + ph[k, 0]) * np.cos(fr[k, 1] * z + ph[k, 1]) for k in range(6))
    gy, gx = np.gradient(y, g, g)
    s = S.Scene()
    s.textures.extend(_textures(seed, 1, 512))
    s.materials.append((0xFFFFFFFF, 0, 0, 32))
    node = s.add_node()
    a = (np.arange(cells)[:, None] * (cells + 1) + np.arange(cells)[None, :]).reshape(-1)
    quad = np.stack([a, a + cells + 1, a + 1, a + 1, a + cells + 1, a + cells + 2], -1)
    pos = np.stack([x, y, z], -1).reshape(-1, 3)
    nrm = S.normalize_f32(np.stack([-gx, np.ones_like(gx), -gy], -1).reshape(-1, 3).astype(np.float32))
    uv = np.stack([(x + 20.0) / 40.0, (z + 20.0) / 40.0], -1).reshape(-1, 2)
    s.add_primitive(node, S.TRIANGLES, 0, pos, nrm, uv, quad.reshape(-1))
    s.point_lights = [(float(v[0]), 3.0, float(v[1]), 6.0) for v in rng.uniform(-8, 8, (2, 2))]
    yaw = rng.uniform(0, 6.28)
    eye = np.array([0.0, float(y[cells // 2, cells // 2]) + 0.4, 0.0])
    m, c = S.look_at(eye, eye + np.array([math.cos(yaw), -0.12, math.sin(yaw)]))
    return s.finalize(), m, c


def _camera(rng, radius=35.0):
    d = rng.normal(size=3)
    return S.look_at_origin(radius * d / np.linalg.norm(d))


def _pose(scene, rng):
    """Every node turned about its own y axis and moved a little."""
    nodes = abi.SceneDescHolder(scene).nodes
    for nd in nodes:
        nd.rotation[:] = [float(v) for v in S.rot_y(float(rng.uniform(0, 6.28))).astype(np.float32).reshape(-1)]
        nd.translation[:] = [float(np.float32(t + rng.uniform(-1, 1))) for t in nd.translation]
    return nodes


def _sizes(n, lo, w, h):
    """n window sizes between lo x lo and w x h, even over their logarithms; the same for every seed."""
    u = np.random.RandomState(n * 7919 + w + h).uniform(size=(n, 2))
    return [(max(1, min(w, int(lo * (w / lo) ** a))), max(1, min(h, int(lo * (h / lo) ** b)))) for a, b in u]


def _scenes(case, seed):
    """The case's scenes and views from the seed alone: [scene], [(scene index, View, nodes or None)]."""
    kind, w, h = case["kind"], case["w"], case["h"]
    rng = np.random.RandomState(seed % (1 << 31))
    if kind == "cube":
        m, c = _camera(rng, 5.0)
        return [S.cube_scene(seed=seed % (1 << 20))], [(0, S.view_for(w, h, m, c), None)]
    if kind == "terrain":
        s, m, c = _terrain(case["cells"], seed)
        return [s], [(0, S.view_for(w, h, m, c), None)]
    tex = _textures(seed, 8, 1024, alpha=kind == "layers")
    counts = SERVED if kind == "serve" else (case["spheres"],)
    scenes = [_spheres(n, (seed + k) % (1 << 20), tex) for k, n in enumerate(counts)]
    if kind == "host":  # two viewports on one surface
        views = []
        for k in range(2):
            m, c = _camera(rng)
            views.append((0, S.view_for(w // 2, h, m, c, x=k * (w // 2)), None))
        return scenes, views
    if kind == "batch":
        views = []
        for vw, vh in _sizes(case["views"], 128, w, h):
            m, c = _camera(rng)
            v = S.view_for(vw, vh, m, c)
            views.append((0, v, _pose(scenes[0], rng) if case["posed"] else None))
        return scenes, views
    if kind == "serve":
        views = []
        for vw, vh in _sizes(case["requests"], 64, w, h):
            m, c = _camera(rng)
            v = S.view_for(vw, vh, m, c)
            v.dof = bool(rng.uniform() < 0.5)
            views.append((int(rng.randint(len(scenes))), v, None))
        return scenes, views
    m, c = _camera(rng)
    v = S.view_for(w, h, m, c)
    v.shader, v.dof, v.layers = case.get("shader", 0), bool(case.get("dof", False)), case.get("layers", 0)
    return scenes, [(0, v, None)]


class _State:
    """Resident scenes, packed descriptors and output buffers of a program; released with it."""

    def __init__(self):
        self.r = _renderer()
        self.lib, self.ctx = self.r.lib, self.r.ctx
        self.stream = C.c_void_p(_program["stream"].cuda_stream)
        self.ids, self.server = [], None

    def __del__(self):
        try:
            torch.cuda.synchronize()
            if self.server is not None:
                self.server.close()
            for i in self.ids:
                self.r.release(i)
        except Exception:
            pass


def _target(pixels, depth, w, h):
    return abi.Target(pixels, 4 * w, w, h, C.cast(C.c_void_p(depth), C.POINTER(C.c_float)))


def prepare(case, seed):
    st = _State()
    st.kind = kind = case["kind"]
    w, h = case["w"], case["h"]
    if kind == "dof":
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        st.pixels = torch.randint(0, 1 << 24, (h, w), generator=g, device=DEVICE, dtype=torch.int32) | (255 << 24)
        # depth of a frame: patches at distances 2 to 80, a third of them empty
        z = 2.0 * 40.0 ** torch.rand(h // 24 + 1, w // 24 + 1, generator=g, device=DEVICE)
        z = z.repeat_interleave(24, 0).repeat_interleave(24, 1)[:h, :w]
        z = z * (1.0 + 0.05 * torch.rand(h, w, generator=g, device=DEVICE))
        p = S.projection(w, h)
        st.depth = torch.where(z > 25.0, torch.full_like(z, FAR), float(p[2, 2]) * z + float(p[2, 3])).contiguous()
        st.out = torch.zeros_like(st.pixels)
        m, c = S.camera_at_z(35.0)
        v = S.view_for(w, h, m, c)
        v.dof, v.dof_max_radius, v.dof_aperture = True, case["radius"], 0.15
        st.view = abi.view_desc(v)
        st.src = _target(st.pixels.data_ptr(), st.depth.data_ptr(), w, h)
        st.dst = _target(st.out.data_ptr(), st.depth.data_ptr(), w, h)
        return st
    scenes, views = _scenes(case, seed)
    st.ids = [st.r.upload(s) for s in scenes]
    n = len(views)
    px = [v.w * v.h for _, v, _ in views]
    at = np.concatenate([[0], np.cumsum(px)])
    st.views = (abi.ViewDesc * n)(*[abi.view_desc(v) for _, v, _ in views])
    if kind == "host":
        st.pixels, st.depth = np.zeros((h, w), np.uint32), np.zeros(int(at[-1]), np.float32)
        st.targets = (abi.Target * n)(*[_target(st.pixels.ctypes.data, st.depth[at[k]:].ctypes.data, w, h)
                                        for k in range(n)])
        return st
    if kind == "serve":
        buf = host_buffer(2 * int(at[-1]))
        st.pixels, st.depth = buf[:at[-1]], buf[at[-1]:].view(np.float32)
        st.requests = Server.requests([(st.ids[s], v, st.pixels[at[k]:at[k + 1]], st.depth[at[k]:at[k + 1]])
                                       for k, (s, v, _) in enumerate(views)])
        st.server = st.r.server()
        return st
    st.pixels = torch.zeros(int(at[-1]), dtype=torch.int32, device=DEVICE)
    st.depth = torch.zeros(int(at[-1]), dtype=torch.float32, device=DEVICE)
    st.targets = (abi.Target * n)(*[_target(st.pixels.data_ptr() + 4 * int(at[k]), st.depth.data_ptr() + 4 * int(at[k]),
                                            v.w, v.h) for k, (_, v, _) in enumerate(views)])
    if kind == "batch":
        st.items = (abi.BatchItem * n)()
        st.nodes = [nodes for _, _, nodes in views]
        for k in range(n):
            st.items[k].scene_id, st.items[k].view, st.items[k].target = st.ids[0], st.views[k], st.targets[k]
            if st.nodes[k] is not None:
                st.items[k].nodes, st.items[k].n_nodes = C.cast(st.nodes[k], C.POINTER(abi.NodeDesc)), len(st.nodes[k])
        st.opts = abi.BatchOpts(0, 0, 1)
    return st


def run(st):
    kind = st.kind
    if kind == "dof":
        st.r._check(st.lib.sgl_dof(st.ctx, C.byref(st.view), C.byref(st.src), C.byref(st.dst), 1, st.stream))
        return {"pixels": st.out}
    if kind == "serve":
        st.server.wait_many(st.server.submit_many(st.requests))
        return {"pixels": st.pixels.view(np.int32), "depth": st.depth}
    if kind == "host":
        st.r._check(st.lib.sgl_render(st.ctx, st.ids[0], st.views, st.targets, len(st.views), 0, None, None))
        return {"pixels": st.pixels.view(np.int32), "depth": st.depth}
    if kind == "batch":
        e = st.lib.sgl_render_batch(st.ctx, st.items, len(st.items), C.byref(st.opts), st.stream, None)
    elif kind == "noalloc":
        e = st.lib.sgl_render_noalloc(st.ctx, st.ids[0], st.views, st.targets, st.stream)
    else:
        e = st.lib.sgl_render(st.ctx, st.ids[0], st.views, st.targets, 1, 1, st.stream, None)
    st.r._check(e)
    return {"pixels": st.pixels, "depth": st.depth}


# ------------------------------------------------------------------ work --


def work(case):
    """Bytes: every scene once (32 B a vertex, 4 B an index; of its texels no more than two a pixel), the colour and
    depth of each pixel written once, and with depth of field 12 B a pixel more (colour and depth read, colour
    written).  Operations: 36 a vertex
    and view, 250 a shaded pixel (a third of a view of spheres, half a terrain), 100 a gathered pixel."""
    kind, w, h = case["kind"], case["w"], case["h"]
    if kind == "dof":
        return {"bytes": 12 * w * h, "flops": 100 * w * h}
    views, lo, dof = 1, None, 1.0 if case.get("dof") else 0.0
    if kind == "batch":
        views, lo = case["views"], 128
    elif kind == "serve":
        views, lo, dof = case["requests"], 64, 0.5
    px = views * w * h if lo is None else sum(a * b for a, b in _sizes(views, lo, w, h))
    if kind == "cube":
        verts, index, texels = 24, 24, 65536
    elif kind == "terrain":
        verts, index, texels = (case["cells"] + 1) ** 2, 6 * case["cells"] ** 2, 512 * 512
    else:
        n = sum(SERVED) if kind == "serve" else case["spheres"]
        verts = index = 64 * 66 * n
        texels = 8 * 1024 * 1024
    per_view = verts / (len(SERVED) if kind == "serve" else 1) * (2 if kind == "host" else views)
    return {"bytes": 32 * verts + 4 * index + 4 * min(texels, 2 * px) + (8 + 12 * dof) * px,
            "flops": 36 * per_view + px * (250 / (2 if kind == "terrain" else 3) + 100 * dof)}


# ----------------------------------------------------------------- exact --


def _triangles(scene):
    """The triangles in draw order, every second of a strip turned."""
    out = []
    idx = scene.indices.astype(np.int64)
    for _, mode, _, v0, _, i0, n in scene.primitives:
        k = idx[i0:i0 + n] + v0
        if mode == S.TRIANGLES:
            t = k[:n // 3 * 3].reshape(-1, 3)
        elif mode == S.TRIANGLE_FAN:
            t = np.stack([np.full(n - 2, k[0]), k[1:-1], k[2:]], -1)
        else:
            t = np.stack([k[:-2], k[1:-1], k[2:]], -1)
            t[1::2] = t[1::2][:, [1, 0, 2]]
        out.append(t)
    return torch.from_numpy(np.concatenate(out)).to(DEVICE)


def _world(scene, nodes):
    rot = torch.tensor(np.stack(scene.node_rotation).astype(np.float64)[:, :3, :3], device=DEVICE)
    move = torch.tensor(np.stack(scene.node_translation).astype(np.float64), device=DEVICE)
    if nodes is not None:
        rot = torch.tensor([list(nd.rotation) for nd in nodes], dtype=torch.float64,
                           device=DEVICE).reshape(-1, 4, 4)[:, :3, :3]
        move = torch.tensor([list(nd.translation) for nd in nodes], dtype=torch.float64, device=DEVICE)
    of = np.repeat([p[0] for p in scene.primitives], [p[4] for p in scene.primitives])
    of = torch.from_numpy(of.astype(np.int64)).to(DEVICE)
    p = torch.from_numpy(scene.positions.astype(np.float64)).to(DEVICE)
    return torch.einsum("vij,vj->vi", rot[of], p) + move[of]


def _clipped(t):
    """Clip-space triangles (n, 3, 3) cut at z' = NEAR: those in front, and the pieces of those that cross it."""
    front = (t[..., 2] >= NEAR).sum(1)
    out = [t[front == 3]]
    cross = t[(front == 1) | (front == 2)]
    one = (cross[..., 2] >= NEAR).sum(1) == 1
    # the vertex that is alone on its side first, the order round the triangle kept
    alone = torch.where(one[:, None], cross[..., 2] >= NEAR, cross[..., 2] < NEAR).to(torch.int64).argmax(1)
    order = (alone[:, None] + torch.arange(3, device=t.device)) % 3
    c = cross.gather(1, order[..., None].expand(-1, -1, 3))
    cut = lambda a, b: a + (b - a) * ((NEAR - a[:, 2:]) / (b[:, 2:] - a[:, 2:]))  # noqa: E731
    ab, ac = cut(c[:, 0], c[:, 1]), cut(c[:, 0], c[:, 2])
    out.append(torch.stack([c[:, 0], ab, ac], 1)[one])
    out.append(torch.stack([ab, c[:, 1], c[:, 2]], 1)[~one])
    out.append(torch.stack([ab, c[:, 2], ac], 1)[~one])
    return torch.cat(out)


def _depth(world, tris, view):
    """The z-buffer of a view's triangles in 64 bits: spans half open in x and y at whole pixels, 1 / z' linear over
    the screen, the nearest kept.  A triangle is drawn when each of its vertices belongs to a visible one (in the
    view volume and facing the camera)."""
    w, h = view.w, view.h
    vm = torch.tensor(np.asarray(view.view, np.float64)[:3], device=DEVICE)
    pm = torch.tensor(np.asarray(view.proj, np.float64)[:3], device=DEVICE)
    p = (world @ vm[:, :3].T + vm[:, 3]) @ pm[:, :3].T + pm[:, 3]
    ndc = torch.cat([p[:, :2] / p[:, 2:].abs(), p[:, 2:]], 1)
    a, b, c = (ndc[tris[:, k]] for k in range(3))
    lo, hi = torch.minimum(torch.minimum(a, b), c), torch.maximum(torch.maximum(a, b), c)
    facing = (b - a)[:, 0] * (c - a)[:, 1] - (b - a)[:, 1] * (c - a)[:, 0] > 0
    seen = facing & (hi[:, 0] >= -1) & (hi[:, 1] >= -1) & (lo[:, 0] < 1) & (lo[:, 1] < 1) & (hi[:, 2] >= NEAR)
    flag = torch.zeros(len(world), dtype=torch.bool, device=DEVICE)
    flag[tris[seen].reshape(-1)] = True
    t = _clipped(p[tris[flag[tris].all(1)]])
    x = view.x + w / 2.0 * (1.0 + t[..., 0] / t[..., 2])
    y = view.y + h / 2.0 * (1.0 - t[..., 1] / t[..., 2])
    y, k = y.sort(1)
    x, iz = x.gather(1, k), (1.0 / t[..., 2]).gather(1, k)
    x0 = x.amin(1).ceil().clamp(view.x, view.x + w).to(torch.int64)
    x1 = x.amax(1).ceil().clamp(view.x, view.x + w).to(torch.int64)
    y0 = y[:, 0].ceil().clamp(view.y, view.y + h).to(torch.int64)
    y1 = y[:, 2].ceil().clamp(view.y, view.y + h).to(torch.int64)
    count = (x1 - x0) * (y1 - y0)
    zb = torch.full((w * h,), FAR, dtype=torch.float64, device=DEVICE)
    keep = (count > 0).nonzero()[:, 0]
    ends = count[keep].cumsum(0)
    total, done = int(ends[-1]) if len(keep) else 0, 0
    while done < total:
        upto = min(total, done + (1 << 23))
        j = torch.arange(done, upto, device=DEVICE)
        q = torch.searchsorted(ends, j, right=True)
        i = keep[q]
        j = j - (ends[q] - count[i])
        px, py = x0[i] + j % (x1 - x0)[i], y0[i] + j // (x1 - x0)[i]
        X, Y, Z = x[i], y[i], iz[i]
        fx, fy = px.double(), py.double()
        at = lambda m, n, V: V[:, m] + (V[:, n] - V[:, m]) * ((fy - Y[:, m]) / (Y[:, n] - Y[:, m]))  # noqa: E731
        low = fy >= Y[:, 1]
        xs, zs = (torch.where(low, at(1, 2, V), at(0, 1, V)) for V in (X, Z))
        xl, zl = at(0, 2, X), at(0, 2, Z)
        inside = (torch.minimum(xs, xl) <= fx) & (fx < torch.maximum(xs, xl))
        z = 1.0 / (zs + (zl - zs) * ((fx - xs) / (xl - xs)))
        inside &= z > NEAR
        zb.scatter_reduce_(0, ((py - view.y) * w + px - view.x)[inside], z[inside], "amin")
        done = upto
    return zb


def exact(case, seed):
    if case["kind"] in ("dof", "layers"):  # whole numbers alone; the depth of the first fragment whose texel is opaque
        return None
    scenes, views = _scenes(case, seed)
    tris = [_triangles(s) for s in scenes]
    worlds = [None if views[0][2] is not None else _world(s, None) for s in scenes]
    out = [_depth(worlds[s] if nodes is None else _world(scenes[s], nodes), tris[s], v) for s, v, nodes in views]
    return {"pixels": None, "depth": torch.cat(out)}
