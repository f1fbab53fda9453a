"""The short node visit (no counting, trees without inverted boxes) against the
general one (counting) and the oracle: hits, distances, barycentrics and tie
flags bit for bit, for rays that hit boxes exactly on their planes (NaN plane
distances), degenerate rays, and a scene whose tree must keep the general form
(a sphere of negative radius has a box with min > max)."""
import numpy as np
import pytest

from radiantium_gb300 import native as N
from radiantium_gb300 import procedural
from radiantium_gb300.scene import Group, Sphere
from oracle.oracle import OracleScene
from tests.test_gpu_edge import _degenerate_rays
from tests.test_gpu_parity import assert_hits_equal, random_rays
from tests.test_gpu_wide_traversal import _axis_rays

pytestmark = pytest.mark.gpu


def _scene(name):
    if name == "zoo":
        return procedural.material_zoo(32, 32)[0]
    if name == "instanced":
        return procedural.instanced_spheres(32, 32, sphere_n=12, grid=4, env_w=32, env_h=16)[0]
    s, _ = procedural.cornell_box(32, 32)
    if name == "inverted":
        s.spheres.append(Sphere((0.5, 0.5, 0.5), -0.2))
        s.groups.append(Group(N.GROUP_SPHERE, 0, material=s.groups[0].material))
    return s


def _plane_rays(n, seed):
    """Rays along an axis or in a coordinate plane that start exactly on planes
    of the Cornell box's bounding boxes (coordinates 0, 1, 0.4, 0.6)."""
    rng = np.random.default_rng(seed)
    rays = np.zeros(n, dtype=N.ray_dtype())
    rays["o"] = rng.choice(np.array([0.0, 1.0, 0.4, 0.6, 0.999], np.float32), (n, 3))
    d = rng.choice(np.array([-1.0, 0.0, 1.0, -0.0, 0.5], np.float32), (n, 3))
    d[np.abs(d).sum(1) == 0, 0] = 1.0
    rays["d"] = d
    rays["min_t"], rays["max_t"] = 1e-4, 3.4028234663852886e38
    return rays


@pytest.mark.parametrize("name", ["cornell", "inverted", "zoo", "instanced"])
def test_short_and_general_visits_equal_the_oracle(dev, name):
    s = _scene(name)
    box = ((-3, 0, -3), (3, 3, 3)) if name in ("zoo", "instanced") else ((0, 0, 0), (1, 1, 1))
    rays = np.concatenate([random_rays(box, 20011, 3), random_rays(box, 20011, 4, inside=True),
                           _axis_rays(s, 20000, 5), _plane_rays(20000, 6), _degenerate_rays()])
    dev.upload(s)
    orc = OracleScene(s)
    try:
        want_h, want_a = orc.trace_closest(rays), orc.trace_any(rays)
    finally:
        orc.close()
    for counting in (False, True):
        dev.set_counting(counting)
        try:
            assert_hits_equal(dev.trace_closest(rays), want_h)
            assert np.array_equal(dev.trace_any(rays).astype(np.uint8), want_a.astype(np.uint8))
        finally:
            dev.set_counting(False)
    assert (want_h["prim"] >= 0).sum() > rays.size // 10
