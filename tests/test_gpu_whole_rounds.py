"""Path rounds that run in one launch (gpu): up to one sample for each resident
lane of the kernel that ends a round, 77,824 on a GB300 of 152 SMs, a one-type
scene has no loop.  Films on both sides of that line are the loop's bits, and
the oracle's; the launches of a call show which side it took."""
import ctypes as C

import numpy as np
import pytest

from radiantium_gb300 import native as N
from radiantium_gb300 import procedural
from oracle.oracle import OracleScene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp", [(256, 256, 1), (303, 256, 1), (304, 256, 1), (275, 283, 1), (320, 256, 1), (64, 76, 16),
                                     (64, 77, 16)])
def test_films_around_the_line(dev, w, h, spp):
    s, st = procedural.cornell_box(w, h)
    st = st.replace(spp=spp)
    orc = OracleScene(s)
    try:
        want = orc.render(st)
    finally:
        orc.close()
    dev.upload(s)
    launches, films = {}, {}
    try:
        for finish in (0, -1):
            assert dev.lib.rt_debug_set_finish(C.c_void_p(dev.h.value), finish) == N.RT_OK
            for wide in (False, True):
                dev.set_traversal(N.TRAVERSAL_WIDE if wide else N.TRAVERSAL_EXACT)
                films[finish, wide] = dev.render(st).view(np.uint32)
                launches[finish, wide] = dev.stats()["kernel_launches"]
    finally:
        dev.set_traversal(N.TRAVERSAL_EXACT)
        dev.lib.rt_debug_set_finish(C.c_void_p(dev.h.value), -1)
    for finish in (0, -1):
        assert np.array_equal(films[finish, False], want.view(np.uint32)), finish
    assert np.array_equal(films[0, True], films[-1, True])
    assert launches[0, False] > 20            # the loop's iterations
    if w * h * spp <= 65536:
        assert launches[-1, False] < 12       # start, trace, finish, film: no loop
    if w * h * spp > 80000:
        assert launches[-1, False] > 20
