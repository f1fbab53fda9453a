"""A cancelled call leaves nothing queued: its stream is idle when it returns,
and a call on another stream right after it gives the film of an undisturbed
context (gpu).  Rounds of one sample per pixel end in a launch that no later
wait of the call covers, so a cancel between rounds finds one running."""
import ctypes as C
import threading

import numpy as np
import pytest

from radiantium_gb300 import native as N
from radiantium_gb300 import procedural
from radiantium_gb300.device import Device

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _cancelled(dev, call, delay):
    """call() in this thread, cancelled from another after `delay` seconds."""
    t = threading.Timer(delay, dev.cancel)
    t.start()
    try:
        with pytest.raises(N.RTError) as e:
            call()
    finally:
        t.join()
    assert e.value.code == N.RT_ERR_CANCELLED


@pytest.mark.parametrize("kind", ["path", "volume", "particles", "batch"])
def test_cancel_on_one_stream_then_render_on_another(kind):
    w = h = 256
    s, st = procedural.volume_box(w, h) if kind == "volume" else procedural.cornell_box(w, h)
    if kind == "particles":
        st = st.replace(integrator=N.INTEGRATOR_PARTICLE, max_depth=-1, min_depth=5)
    out = torch.zeros((w, h, 3), dtype=torch.float32, device="cuda")
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with Device(0) as dev:
        dev.upload(s)
        assert dev.lib.rt_debug_set_limits(C.c_void_p(dev.h.value), C.c_int64(w * h), 0) == N.RT_OK
        dev.set_renderer(N.RENDERER_WAVEFRONT)

        def render(n, stream):
            if kind == "particles":
                dev.render_particles_device(st, n * w * h, out.data_ptr(), stream=stream.cuda_stream)
            elif kind == "batch":
                dev.render_batch_device([(dev, st.replace(spp=n))], [out.data_ptr()], stream=stream.cuda_stream)
            else:
                dev.render_device(st.replace(spp=n), out.data_ptr(), stream=stream.cuda_stream)

        torch.cuda.synchronize()
        render(2, a)
        want = out.cpu().numpy()
        for k in range(8):
            _cancelled(dev, lambda: render(1 << 14, a), 0.02 + 0.0013 * k)
            assert a.query(), "work of the cancelled call is still queued"
            render(2, b)
            got = out.cpu().numpy()
            if kind == "particles":
                assert np.allclose(got, want, rtol=1e-5, atol=1e-6 * want.max()), k
            else:
                assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), k
