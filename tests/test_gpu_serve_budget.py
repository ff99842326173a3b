"""A served view with depth of field on the least budget that admits it (no
room for its winner list: shaded by tiles) and on a larger one: both equal the
view rendered alone."""
import numpy as np
import pytest

from swegl_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(97, 61), (640, 480)])
def test_frames_on_the_least_budget(w, h):
    from swegl_gb300.runtime import Renderer, SglError

    r = Renderer(0)
    sid = r.upload(S.spheres_scene(n_spheres=12, seed=5, tex_size=64))
    v = S.spheres_view(w, h, 20.0)
    v.dof = True
    pix, z = np.zeros((h, w), np.uint32), np.zeros((h, w), np.float32)

    def serve(budget):
        srv = r.server(budget_bytes=budget, max_batch=2, streams=1)
        try:
            res = srv.wait(srv.submit(sid, v, pix, z))
            assert res["status"] == 0
            return True
        except SglError as e:
            assert e.status == -5  # the request alone exceeds the budget
            return False
        finally:
            srv.close()

    expect = r.render(sid, [v])[0][0]
    lo, hi = 0, 1 << 28
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if serve(mid) else (mid, hi)
    for budget in (hi, 2 * hi):
        pix[:], z[:] = 0, 0
        assert serve(budget)
        assert np.array_equal(pix, expect.pixels)
        assert np.array_equal(z.view(np.uint32), expect.zbuffer.view(np.uint32))
    r.close()
