"""Both ways of resolving transparency layers (fragments shaded when they are
linked, or nearest first when their pixel is resolved) on the same visible
scene: more fragments than layers and than the resolve holds in registers,
fragments of equal depth (transparent ones, and opaque ones at a transparent
one's depth), near-clipped ones, alone and offset on a shared surface.  Which
way is taken follows from triangles out of view: many opaque ones for one,
many translucent ones for the other.  Both equal the oracle (depth bits,
counts, colours within 2 LSB, 1 LSB on 99.9 %) and each other exactly."""
import numpy as np
import pytest

import oracle
from swegl_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def renderer():
    from swegl_gb300.runtime import Renderer

    r = Renderer(0)
    yield r
    r.close()


def scene(translucent_rest):
    s = S.Scene()
    s.textures += [S.texture_uniform(31, 64, 64), S.texture_block_alpha(32, 64, 64, 8),
                   S.texture_block_alpha(33, 32, 32, 4)]
    s.materials += [(0xFFFFFFFF, 0, 0, 32), (0xFFFFFFFF, 1, 1, 32), (0xFFFFFFFF, 2, 1, 32), (0x80FFFFFF, -1, 1, 32)]
    cube = s.add_node(translation=(0.0, 0.0, -2.5), rotation=S.rot_y(0.6).astype(np.float32))
    for p, nm, t, i in S.cube_mesh(2.0):
        s.add_primitive(cube, S.TRIANGLE_FAN, 0, p, nm, t, i)
    q = np.array([[-3.0, -2.0, 0.0], [3.0, -2.0, 0.0], [3.0, 2.0, 0.0], [-3.0, 2.0, 0.0]], np.float32)
    nq = np.tile(np.array([0.0, 0.0, 1.0], np.float32), (4, 1))
    uq = np.array([[0.0, 0.0], [2.0, 0.0], [2.0, 1.5], [0.0, 1.5]], np.float32)
    fan = np.arange(4, dtype=np.uint32)
    for k in range(8):
        node = s.add_node(translation=(0.05 * k, -0.03 * k, -2.0 + 0.25 * k), rotation=S.rot_z(0.07 * k).astype(np.float32))
        s.add_primitive(node, S.TRIANGLE_FAN, 1 + k % 2, q, nq, uq, fan)
        if k % 3 != 1:  # the same sheet again: equal depths, another texture (opaque where the first is not, and so on)
            s.add_primitive(node, S.TRIANGLE_FAN, 2 - k % 2, q, nq, uq + np.float32(0.25), fan)
    floor = s.add_node(translation=(0.0, -0.6, 0.0))  # runs under the camera and behind it
    p = np.array([[-4.0, 0.0, 3.0], [4.0, 0.0, 3.0], [4.0, 0.0, -6.0], [-4.0, 0.0, -6.0]], np.float32)
    s.add_primitive(floor, S.TRIANGLE_FAN, 1, p, np.tile(np.array([0.0, 1.0, 0.0], np.float32), (4, 1)), uq, fan)
    rest = s.add_node(translation=(0.0, 0.0, 60.0))  # behind the camera
    tri = np.tile(np.array([[0.0, 0.0, 0.0], [0.1, 0.0, 0.0], [0.0, 0.1, 0.0]], np.float32), (80, 1))
    for _ in range(10):
        s.add_primitive(rest, S.TRIANGLES, 3 if translucent_rest else 0, tri, np.tile(nq[:1], (240, 1)),
                        np.zeros((240, 2), np.float32), np.arange(240, dtype=np.uint32))
    s.point_lights = [(0.0, 1.0, 2.0, 2.0)]
    return s.finalize()


def view(w, h, layers, shader=0, x=0, y=0):
    m, c = S.look_at((0.2, 0.1, 1.6), (0.0, 0.0, -2.0))
    v = S.view_for(w, h, m, c)
    v.layers, v.shader, v.x, v.y = layers, shader, x, y
    return v


def close(got, exp):
    d = np.abs(got.view(np.uint8).astype(np.int16) - exp.view(np.uint8).astype(np.int16)).reshape(-1, 4).max(1)
    assert int(d.max()) <= 2 and float((d <= 1).mean()) >= 0.999


@pytest.mark.parametrize("layers,shader", [(1, 0), (3, 0), (8, 0), (4, 5), (2, 1)])
def test_both_ways_equal_the_oracle(renderer, layers, shader):
    v = view(200, 150, layers, shader)
    frames = []
    for rest in (False, True):
        sc = scene(rest)
        sid = renderer.upload(sc)
        (f,), stats = renderer.render(sid, [v], stats=True)
        ref = oracle.render(sc, [v])
        assert stats["fragments"] > 10 * v.w * v.h
        assert (stats["drawn_triangles"], stats["fragments"]) == tuple(ref.stats[0][:2])
        assert np.array_equal(f.zbuffer.view(np.uint32), ref.zbuffer.view(np.uint32))
        close(f.pixels, ref.pixels)
        frames.append(f)
        renderer.release(sid)
    assert np.array_equal(frames[0].pixels, frames[1].pixels)


@pytest.mark.parametrize("shader", [0, 5])
def test_both_ways_offset_on_a_surface_with_content(renderer, shader):
    bg = np.random.default_rng(5).integers(0, 2 ** 32, size=(200, 300), dtype=np.uint64).astype(np.uint32)
    views = [view(160, 110, 3, shader, x=70, y=60), view(120, 90, 8, shader, x=10, y=20)]
    frames = []
    for rest in (False, True):
        sc = scene(rest)
        sid = renderer.upload(sc)
        got, _ = renderer.render(sid, views, shared_surface=(300, 200), background=bg)
        ref = oracle.render(sc, views, shared_surface=(300, 200), background=bg)
        for g, e in zip(got, ref.frames):
            assert np.array_equal(g.zbuffer.view(np.uint32), e.zbuffer.view(np.uint32))
        close(got[0].pixels, ref.frames[0].pixels)
        frames.append(got[0].pixels)
        renderer.release(sid)
    assert np.array_equal(frames[0], frames[1])


def test_one_translucent_texel_costs_an_opaque_scene_little(renderer):
    """A deep stack of opaque sheets, and the same with one texel of the
    texture translucent: about the same time in the layer passes (all of the
    hidden fragments were shaded in the second once)."""
    times = []
    for clear in (0, 1):
        s = S.Scene()
        t = S.texture_uniform(31, 256, 256) | np.uint32(0xFF000000)
        t[0, :clear] &= np.uint32(0x80FFFFFF)
        s.textures.append(t)
        s.materials.append((0xFFFFFFFF, 0, 1, 32))
        q = np.array([[-3.0, -2.0, 0.0], [3.0, -2.0, 0.0], [3.0, 2.0, 0.0], [-3.0, 2.0, 0.0]], np.float32)
        nq = np.tile(np.array([0.0, 0.0, 1.0], np.float32), (4, 1))
        uq = np.array([[0.01, 0.01], [0.96, 0.01], [0.96, 0.97], [0.01, 0.97]], np.float32)
        for k in range(100):
            node = s.add_node(translation=(0.0, 0.0, -2.0 + 0.01 * k))
            s.add_primitive(node, S.TRIANGLE_FAN, 0, q, nq, uq, np.arange(4, dtype=np.uint32))
        s.point_lights = [(0.0, 1.0, 2.0, 2.0)]
        sid = renderer.upload(s.finalize())
        v = view(320, 240, 2)
        best = 1e9
        for _ in range(6):
            renderer.profile(True)
            renderer.render(sid, [v])
            p = renderer.profile_read()
            best = min(best, p["k_frags"]["total_ms"] + p["k_layers"]["total_ms"])
        renderer.profile(False)
        times.append(best)
        renderer.release(sid)
    assert times[1] < 1.25 * times[0], times
