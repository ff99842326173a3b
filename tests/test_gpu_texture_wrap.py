"""Texture coordinates outside the texture on the GPU against the oracle: the
wrap of the bilinear fetch by range (inside, one period off, repeated over
power-of-two and other sizes, negative beyond one period, past 2^22 texels,
infinite).  The texture shaders use exact arithmetic: pixels are equal."""
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


def sheet(size, lo, hi):
    s = S.Scene()
    s.textures.append(S.texture_uniform(5, *size))
    s.materials.append((0xFFFFFFFF, 0, 1, 32))
    node = s.add_node()
    pos = [[-1.2, -0.9, 0.0], [1.2, -0.9, 0.2], [1.2, 0.9, -0.1], [-1.2, 0.9, 0.1]]
    uv = np.array([[lo, lo], [hi, lo], [hi, hi], [lo, hi]], np.float32)
    s.add_primitive(node, S.TRIANGLE_FAN, 0, pos, [[0.0, 0.0, 1.0]] * 4, uv, [0, 1, 2, 3])
    return s.finalize()


@pytest.mark.parametrize("size", [(64, 64), (48, 20), (1, 1), (2, 3)])
@pytest.mark.parametrize("lo, hi", [(0.0, 1.0), (-0.999, 0.4), (0.3, 7.6), (-5.2, 2.4), (-9.0, -3.1), (9e4, 3e5),
                                    (-1e6, 4e6), (0.5, 1e9), (0.0, 1e30), (0.0, np.inf)])
def test_wrap(renderer, size, lo, hi):
    sc = sheet(size, lo, hi)
    m, c = S.look_at((0.2, 0.1, 2.4), (0.0, 0.0, 0.0))
    views = [S.view_for(97, 75, m, c) for _ in range(2)]
    views[0].shader, views[1].shader = 5, 6  # bilinear, nearest
    sid = renderer.upload(sc)
    frames, _ = renderer.render(sid, views)
    renderer.release(sid)
    for f, e in zip(frames, oracle.render(sc, views).frames):
        assert np.array_equal(f.pixels, e.pixels)
        assert np.array_equal(f.zbuffer.view(np.uint32), e.zbuffer.view(np.uint32))
