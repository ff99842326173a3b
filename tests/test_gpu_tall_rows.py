"""Triangles around the walk's row limits on the GPU against the oracle: heights
of 15 to 18 rows (the limit between a lane's rows and a warp's triangle), of
31 to 34 and 63 to 66 rows (a warp walks 32 rows at a time) and of the whole
view, their middle vertex anywhere between, and cut by the view's top and
bottom; through the fused and the general geometry pass, alone, in a batch of
uneven views and layered.  Depth, drawn triangles and fragments are equal,
colours within the repository's bar (2 LSB, 1 LSB on 99.9 %)."""
import numpy as np
import pytest

import oracle
from swegl_gb300 import scenes as S

pytestmark = pytest.mark.gpu
W, H = 160, 120


@pytest.fixture(scope="module")
def renderer():
    from swegl_gb300.runtime import Renderer

    r = Renderer(0)
    yield r
    r.close()


def tall_scene(heights, per_primitive, seed):
    """Triangles of the given pixel heights in a 160 x 120 view from (0, 0, 5), `per_primitive` in one list."""
    rng = S.Rng(seed)
    s = S.Scene()
    s.textures.append(S.texture_uniform(seed, 32, 32))
    s.materials.append((0xFFFFFFFF, 0, 1, 32))
    node = s.add_node()
    unit = 2.0 * 5.0 / (S.projection(W, H)[1, 1] * H)  # world units per pixel at z = 0
    pos = []
    for k in range(6 * len(heights)):
        h = heights[k % len(heights)] + rng.uniform(-0.4, 0.4, 1)[0]
        x, y0 = rng.uniform(-70, 70, 1)[0], rng.uniform(-75, 60, 1)[0]
        mid = rng.integers(0, 4, 1)[0]
        ym = y0 + h * (0.0, 0.3, 0.5, 0.97, 1.0)[mid]
        dx = rng.uniform(-40, 40, 2)
        z = rng.uniform(-0.5, 0.5, 3)
        pos += [(x * unit, y0 * unit, z[0]), ((x + dx[0]) * unit, ym * unit, z[1]), ((x + dx[1]) * unit, (y0 + h) * unit, z[2])]
    pos = np.asarray(pos, np.float32)
    nrm = np.tile(np.array([0.0, 0.0, 1.0], np.float32), (len(pos), 1))
    uv = rng.uniform(0.0, 1.0, 2 * len(pos)).reshape(-1, 2).astype(np.float32)
    n = 3 * per_primitive
    for i in range(0, len(pos), n):
        k = len(pos[i:i + n])
        s.add_primitive(node, S.TRIANGLES, 0, pos[i:i + n], nrm[i:i + n], uv[i:i + n], np.arange(k))
    s.point_lights = [(0.5, 1.5, 2.5, 2.0)]
    return s.finalize()


def view(w=W, h=H, dx=0.0):
    m, c = S.look_at((dx, 0.0, 5.0), (dx, 0.0, 0.0))
    return S.view_for(w, h, m, c)


def check(f, e):
    assert np.array_equal(f.zbuffer.view(np.uint32), e.zbuffer.view(np.uint32))
    d = np.abs(f.pixels.view(np.uint8).astype(np.int16) - e.pixels.view(np.uint8).astype(np.int16)).reshape(-1, 4).max(1)
    assert int(d.max()) <= 2 and float((d <= 1).mean()) >= 0.999


@pytest.mark.parametrize("per_primitive", [4, 120])  # fused pass; general pass (over 256 vertices)
@pytest.mark.parametrize("heights", [(15, 16, 17, 18), (31, 32, 33, 34), (63, 64, 65, 66), (2, 119, 200)])
def test_heights(renderer, heights, per_primitive):
    sc = tall_scene(heights, per_primitive, seed=11 + heights[0])
    sid = renderer.upload(sc)
    views = [view(), view(W - 7, H // 2, 0.3), view(33, H + 21, -0.2)]
    frames, stats = renderer.render(sid, views, stats=True)
    ref = oracle.render(sc, views)
    for f, e in zip(frames, ref.frames):
        check(f, e)
    assert stats["drawn_triangles"] == sum(s[0] for s in ref.stats)
    assert stats["fragments"] == sum(s[1] for s in ref.stats)
    _, winner, _, _ = renderer.render_debug(sid, views[0])
    assert np.array_equal(winner, oracle.render(sc, views[:1], winner=True).winner)
    views[0].layers = 2
    check(renderer.render(sid, views[:1])[0][0], oracle.render(sc, views[:1]).frames[0])
    renderer.release(sid)


def test_batch_equals_single_frames(renderer):
    import ctypes as C

    import torch

    from swegl_gb300 import abi

    ids = [renderer.upload(tall_scene((3, 16, 17, 33, 90), n, seed=5)) for n in (4, 120)]
    items, bufs = [], []
    for k in range(6):
        v = view(40 + 30 * k, 120 - 15 * k, 0.1 * k)
        pix = torch.zeros((v.h, v.w), dtype=torch.int32, device="cuda")
        z = torch.zeros((v.h, v.w), dtype=torch.float32, device="cuda")
        t = abi.Target(pix.data_ptr(), 4 * v.w, v.w, v.h, C.cast(C.c_void_p(z.data_ptr()), C.POINTER(C.c_float)))
        items.append((ids[k % 2], v, t))
        bufs.append((pix, z))
    renderer.render_batch(items)
    torch.cuda.synchronize()
    for (sid, v, _), (pix, z) in zip(items, bufs):
        f = renderer.render(sid, [v])[0][0]
        assert np.array_equal(pix.cpu().numpy().view(np.uint32), f.pixels)
        assert np.array_equal(z.cpu().numpy().view(np.uint32), f.zbuffer.view(np.uint32))
    for i in ids:
        renderer.release(i)
