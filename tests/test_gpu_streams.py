"""Device calls of one context on alternating streams, enqueued without a wait
between them: every frame equals the one rendered alone."""
import ctypes as C

import numpy as np
import pytest

from swegl_gb300 import abi
from swegl_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batched", [False, True])
def test_alternating_streams_equal_single_frames(batched):
    import torch

    from swegl_gb300.runtime import Renderer

    r = Renderer(0)
    ids = [r.upload(S.spheres_scene(n_spheres=40, seed=k, tex_size=64)) for k in (3, 4)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.default_stream()]
    rng = S.Rng(7)
    calls = []
    for k in range(24):
        m, c = S.camera_on_sphere(rng, 30.0)
        v = S.view_for(480 - 16 * (k % 5), 320 + 8 * (k % 3), m, c)
        pix = torch.zeros((v.h, v.w), dtype=torch.int32, device="cuda")
        z = torch.zeros((v.h, v.w), dtype=torch.float32, device="cuda")
        t = abi.Target(pix.data_ptr(), 4 * v.w, v.w, v.h, C.cast(C.c_void_p(z.data_ptr()), C.POINTER(C.c_float)))
        calls.append((ids[k % 2], v, t, pix, z))
    torch.cuda.synchronize()
    for k, (sid, v, t, _, _) in enumerate(calls):
        st = streams[k % 3].cuda_stream
        if batched:
            r.render_batch([(sid, v, t)], stream=st)
        else:
            r.render_device(sid, [v], [t], stream=st)
    torch.cuda.synchronize()
    for sid, v, _, pix, z in calls:
        f = r.render(sid, [v])[0][0]
        assert np.array_equal(pix.cpu().numpy().view(np.uint32), f.pixels)
        assert np.array_equal(z.cpu().numpy().view(np.uint32), f.zbuffer.view(np.uint32))
    r.close()


@pytest.mark.parametrize("posed", [False, True])
def test_calls_after_a_captured_batch(posed):
    """A batch captured into a caller's graph (direct launches) between calls
    on other streams: those go on as before, however many, and the replay
    draws the frame, also after them."""
    import torch

    from swegl_gb300.runtime import Renderer

    r = Renderer(0)
    scene = S.cube_scene()
    sid = r.upload(scene)
    v, other = S.cube_view(320, 240), S.cube_view(320, 240)
    m, c = S.look_at((2.0, 1.5, 3.0), (0.0, 0.0, 0.0))
    other.view, other.camera_pos = m, c
    nodes = abi.SceneDescHolder(scene).nodes if posed else None
    pix = torch.zeros((240, 320), dtype=torch.int32, device="cuda")
    z = torch.zeros((240, 320), dtype=torch.float32, device="cuda")
    t = abi.Target(pix.data_ptr(), 1280, 320, 240, C.cast(C.c_void_p(z.data_ptr()), C.POINTER(C.c_float)))
    a, b = torch.cuda.Stream(), torch.cuda.Stream()

    def frame(view, stream):
        pix.zero_()
        torch.cuda.synchronize()
        r.render_batch([(sid, view, t, nodes)], use_graph=False, stream=stream.cuda_stream)
        torch.cuda.synchronize()
        return pix.clone()

    expect, expect_other = frame(v, a), frame(other, a)
    graph = torch.cuda.CUDAGraph()
    # (a slot's first poses allocate their staging)
    with torch.cuda.graph(graph, stream=b, capture_error_mode="relaxed" if posed else "thread_local"):
        r.render_batch([(sid, v, t, nodes)], use_graph=False, stream=b.cuda_stream)
    for k in range(10):
        pix.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(pix, expect), k
        assert torch.equal(frame(other, (a, b)[k % 2]), expect_other), k
    r.close()
