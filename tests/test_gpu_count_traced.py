"""What a counting run counts (gpu): the reference's rays by default, with
count_traced the rays that a run without counting traces.  They differ in the
MIS rays of infinite lights alone, and films are the same bits in all runs."""
import numpy as np
import pytest

from radiantium_gb300 import native as N
from tests.test_gpu_node_visits import _scene
from radiantium_gb300 import procedural

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [N.RENDERER_WAVEFRONT, N.RENDERER_WAVEFRONT_GRAPH])
@pytest.mark.parametrize("name", ["cornell", "instanced"])
def test_counts_of_the_traced_rays(dev, name, mode):
    s = _scene(name)
    st = procedural.cornell_box(32, 32)[1].replace(spp=4, max_depth=6)
    dev.upload(s)
    dev.set_renderer(mode)
    try:
        plain = dev.render(st)
        dev.set_counting(True)
        counts, films = [], []
        for traced in (False, True, False):
            dev.count_traced(traced)
            films.append(dev.render(st))
            counts.append(dev.stats())
    finally:
        dev.count_traced(False)
        dev.set_counting(False)
        dev.set_renderer(N.RENDERER_AUTO)
    for f in films:
        assert np.array_equal(f.view(np.uint32), plain.view(np.uint32))
    ref, got, again = counts
    keys = ("rays_closest", "rays_shadow", "node_visits", "prim_tests", "instance_visits")
    assert [ref[k] for k in keys] == [again[k] for k in keys]
    if name == "cornell":                    # no infinite light: the same rays
        assert [ref[k] for k in keys] == [got[k] for k in keys]
    else:
        moved = ref["rays_closest"] - got["rays_closest"]
        added = got["rays_shadow"] - ref["rays_shadow"]
        assert moved > 0 and 0 < added <= moved
        assert got["node_visits"] < ref["node_visits"] and got["instance_visits"] < ref["instance_visits"]
