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


def test_calls_after_a_captured_batch():
    """A batch captured into a caller's graph (direct launches) between calls
    on other streams: those go on as before, and the replay draws the frame."""
    import torch

    from swegl_gb300.runtime import Renderer

    r = Renderer(0)
    sid = r.upload(S.cube_scene())
    v = S.cube_view(320, 240)
    pix = torch.zeros((240, 320), dtype=torch.int32, device="cuda")
    z = torch.zeros((240, 320), dtype=torch.float32, device="cuda")
    t = abi.Target(pix.data_ptr(), 1280, 320, 240, C.cast(C.c_void_p(z.data_ptr()), C.POINTER(C.c_float)))
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    r.render_batch([(sid, v, t)], use_graph=False, stream=a.cuda_stream)
    torch.cuda.synchronize()
    expect = pix.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=b, capture_error_mode="thread_local"):
        r.render_batch([(sid, v, t)], use_graph=False, stream=b.cuda_stream)
    pix.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(pix, expect)
    for stream in (a, b):
        pix.zero_()
        torch.cuda.synchronize()
        r.render_batch([(sid, v, t)], use_graph=False, stream=stream.cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(pix, expect)
    r.close()
