"""The megakernel's traversal (one ray per thread) in its short form, and in its
general form while counting and for a scene with an inverted box: films equal
the oracle's bit for bit, counted node, primitive and instance visits equal the
wavefront's."""
import numpy as np
import pytest

from radiantium_gb300 import native as N
from radiantium_gb300 import procedural
from oracle.oracle import OracleScene
from tests.test_gpu_node_visits import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["cornell", "inverted", "zoo", "instanced"])
def test_megakernel_films_and_counts(dev, name):
    s = _scene(name)
    st = procedural.cornell_box(32, 32)[1].replace(spp=3, max_depth=6)
    orc = OracleScene(s)
    try:
        want = orc.render(st)
    finally:
        orc.close()
    dev.upload(s)
    counts = {}
    try:
        for counting in (False, True):
            dev.set_counting(counting)
            for mode in (N.RENDERER_MEGAKERNEL, N.RENDERER_WAVEFRONT):
                dev.set_renderer(mode)
                got = dev.render(st)
                assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (counting, mode)
                v = dev.stats()
                counts[counting, mode] = [v[k] for k in ("node_visits", "prim_tests", "instance_visits")]
    finally:
        dev.set_counting(False)
        dev.set_renderer(N.RENDERER_AUTO)
    assert counts[True, N.RENDERER_MEGAKERNEL] == counts[True, N.RENDERER_WAVEFRONT]
    assert counts[True, N.RENDERER_MEGAKERNEL][0] > 0
