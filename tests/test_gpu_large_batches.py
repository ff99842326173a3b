"""Batches of more views than any block's share of counters: every request's
fragments and frame equal the view's own, and the walk's time per view does
not grow with the number of views (its fragment counts once went to one
global counter per lane from the 65th view on: 4.8 times the time for twice
the views)."""
import ctypes as C

import numpy as np
import pytest

from swegl_gb300 import abi
from swegl_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def renderer():
    from swegl_gb300.runtime import Renderer

    r = Renderer(0)
    yield r
    r.close()


def cameras(n, w, h, seed=9):
    rng = S.Rng(seed)
    out = []
    for _ in range(n):
        m, c = S.camera_on_sphere(rng, 30.0)
        out.append(S.view_for(w, h, m, c))
    return out


@pytest.mark.parametrize("n", [64, 65, 130, 1024, 1030])
def test_counts_of_every_view(renderer, n):
    sid = renderer.upload(S.spheres_scene(n_spheres=6, seed=2, tex_size=32))
    views = cameras(7, 61, 45)
    single = [renderer.render(sid, [v], stats=True) for v in views]
    srv = renderer.server(max_batch=4096, streams=1)
    pix = np.zeros((n, 45, 61), np.uint32)
    z = np.zeros((n, 45, 61), np.float32)
    reqs = srv.requests([(sid, views[k % 7], pix[k], z[k]) for k in range(n)])
    res = srv.wait_many(srv.submit_many(reqs))
    assert srv.stats()["batches"] == 1
    for k in range(n):
        (f,), stats = single[k % 7]
        assert res[k].status == 0 and res[k].fragments == stats["fragments"], k
        assert np.array_equal(pix[k], f.pixels) and np.array_equal(z[k], f.zbuffer), k
    srv.close()
    renderer.release(sid)


def test_walk_time_per_view_does_not_grow(renderer):
    import torch

    sid = renderer.upload(S.spheres_scene(n_spheres=50, seed=2, tex_size=32))
    views = cameras(256, 256, 256)
    pix = torch.zeros((256, 256, 256), dtype=torch.int32, device="cuda")
    z = torch.zeros((256, 256, 256), dtype=torch.float32, device="cuda")
    items = [(sid, v, abi.Target(pix[k].data_ptr(), 1024, 256, 256,
                                 C.cast(C.c_void_p(z[k].data_ptr()), C.POINTER(C.c_float))))
             for k, v in enumerate(views)]

    def walk(n):
        best = 1e9
        for _ in range(6):
            renderer.profile(True)
            renderer.render_batch(items[:n], use_graph=False)
            torch.cuda.synchronize()
            best = min(best, renderer.profile_read()["k_walk"]["total_ms"])
        renderer.profile(False)
        return best

    one, two, four = walk(64), walk(128), walk(256)
    assert two < 3.0 * one and four < 6.0 * one, (one, two, four)
    renderer.release(sid)
