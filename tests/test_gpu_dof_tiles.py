"""The depth-of-field gather by reach on the GPU against the oracle: tiles
staged ahead (up to 16 pixels), staged in turn (up to 32) and gathered from
memory, on views whose rows are and are not 16-byte aligned, smaller and
larger than a tile, with constant, smooth and unlike radii; and views of all
reaches in one batch.  The gather is exact: pixels are equal."""
import ctypes as C

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


@pytest.mark.parametrize("radius", [0.0, 3.2, 16.0, 16.5, 24.0, 32.0, 33.0, 150.0])
@pytest.mark.parametrize("w, h", [(1, 1), (7, 50), (33, 31), (64, 64), (130, 97), (256, 160)])
def test_reach(renderer, w, h, radius):
    rng = np.random.default_rng(int(radius * 10) + w)
    m, c = S.camera_at_z(35.0)
    v = S.view_for(w, h, m, c)
    v.dof, v.dof_aperture, v.dof_max_radius = True, 4.0 * max(radius, 1.0) / h, radius
    px = rng.integers(0, 1 << 32, (h, w), dtype=np.uint64).astype(np.uint32)
    px[:, : w // 2] = 0xFF102030  # half of it constant
    z = rng.uniform(2.0, 60.0, (h // 9 + 1, w // 13 + 1)).repeat(9, 0).repeat(13, 1)[:h, :w]
    z = (z * rng.uniform(1.0, 1.05, (h, w)) * v.proj[2, 2] + v.proj[2, 3]).astype(np.float32)
    z.view(np.uint32)[rng.uniform(size=(h // 20 + 1, w // 20 + 1)).repeat(20, 0).repeat(20, 1)[:h, :w] < 0.4] = 0x7F7F7F7F
    assert np.array_equal(renderer.dof(v, px, z), oracle.dof(v, px, z))


@pytest.mark.parametrize("radius", [16.0, 32.0, 60.0])
def test_offsets_near_ties(renderer, radius):
    """Four million pixels of unlike radii: a product of radius and tap within a unit in the last place of a half
    rounds as the product does, then to even (a fused product and rounding differs about once in a million)."""
    rng = np.random.default_rng(9)
    w, h = 2048, 2048
    m, c = S.camera_at_z(35.0)
    v = S.view_for(w, h, m, c)
    v.dof, v.dof_aperture, v.dof_max_radius, v.dof_focus = True, 0.2, radius, 20.0
    px = rng.integers(0, 1 << 32, (h, w), dtype=np.uint64).astype(np.uint32)
    z = (rng.uniform(16.0, 24.0, (h, w)) * v.proj[2, 2] + v.proj[2, 3]).astype(np.float32)
    assert np.array_equal(renderer.dof(v, px, z), oracle.dof(v, px, z))


def test_reaches_in_one_batch(renderer):
    import torch

    from swegl_gb300 import abi

    sid = renderer.upload(S.mixed_scene())
    items, bufs = [], []
    for k, radius in enumerate([16.0, 40.0, 24.0, 2.0, 16.0, 90.0, 32.0, 8.0, 20.0]):
        m, c = S.look_at((0.3 * k - 1.0, 0.6, 4.0), (0.0, 0.0, 0.0))
        v = S.view_for(90 + 23 * k, 70 + 11 * k, m, c)
        v.dof, v.dof_focus, v.dof_aperture, v.dof_max_radius = True, 3.5, 0.4, radius
        pix = torch.zeros((v.h, v.w), dtype=torch.int32, device="cuda")
        z = torch.zeros((v.h, v.w), dtype=torch.float32, device="cuda")
        t = abi.Target(pix.data_ptr(), 4 * v.w, v.w, v.h, C.cast(C.c_void_p(z.data_ptr()), C.POINTER(C.c_float)))
        items.append((sid, v, t))
        bufs.append(pix)
    renderer.render_batch(items)
    torch.cuda.synchronize()
    for (_, v, _), pix in zip(items, bufs):
        assert np.array_equal(pix.cpu().numpy().view(np.uint32), oracle.render(S.mixed_scene(), [v]).pixels)
    renderer.release(sid)
