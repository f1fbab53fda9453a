"""The kernel that ends a wavefront round (rt_debug_set_finish): films are the
oracle's bit for bit (the light tracer's within summation order) whether the
loop runs to its end, hands over somewhere on the way, or never starts, with
few slots refilled many times, and at path counts that leave warps partly
empty."""
import ctypes as C

import numpy as np
import pytest

from radiantium_gb300 import native as N
from radiantium_gb300 import procedural
from radiantium_gb300.device import Device
from oracle.oracle import OracleScene

pytestmark = pytest.mark.gpu


def _case(name):
    if name == "volume":
        s, st = procedural.volume_box(23, 17)
        return s, st.replace(spp=3)
    if name == "zoo_all":
        s, st = procedural.material_zoo(21, 19)
        return s, st.replace(spp=3, strategy=N.STRATEGY_ALL)
    if name == "zoo_nee":
        s, st = procedural.material_zoo(21, 19)
        return s, st.replace(spp=3, method=N.METHOD_NEE)
    s, st = procedural.cornell_box(33, 31)
    if name == "particles":
        return s, st.replace(integrator=N.INTEGRATOR_PARTICLE, max_depth=-1, min_depth=7)
    return s, st.replace(spp=5)


@pytest.mark.parametrize("slots", [0, 97])
@pytest.mark.parametrize("name", ["cornell", "zoo_all", "zoo_nee", "volume", "particles"])
def test_films_do_not_depend_on_where_a_round_is_handed_over(name, slots):
    s, st = _case(name)
    particles = name == "particles"
    orc = OracleScene(s)
    try:
        want = orc.render_particles(st, 3001) if particles else orc.render(st)
    finally:
        orc.close()
    with Device(0) as dev:
        dev.upload(s)
        if slots:
            assert dev.lib.rt_debug_set_limits(C.c_void_p(dev.h.value), C.c_int64(0), slots) == N.RT_OK
        for finish in (0, 1, 33, 500, 1 << 20, -1):
            assert dev.lib.rt_debug_set_finish(C.c_void_p(dev.h.value), finish) == N.RT_OK
            for mode in (N.RENDERER_WAVEFRONT, N.RENDERER_WAVEFRONT_GRAPH):
                dev.set_renderer(mode)
                if particles:
                    got = dev.render_particles(st, 3001)
                    assert np.allclose(got, want, rtol=1e-5, atol=1e-6 * want.max()), (finish, mode)
                else:
                    got = dev.render(st)
                    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (finish, mode)
