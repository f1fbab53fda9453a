"""Closest hits of rays with a finite max_t over instances.  An instance's
candidate is a world distance, so a first hit can lie beyond the ray's own max_t
(directions longer than 1; unit directions by rounding) and MaxT grows when the
prototype is left: boxes that lay beyond it before are visited after all.  The
short node visit against the oracle and the counting (general) one, bit for bit."""
import numpy as np
import pytest

from radiantium_gb300 import native as N
from radiantium_gb300 import procedural
from radiantium_gb300.scene import Camera, Group, Mat4, Mesh, SceneDesc, Sphere
from oracle.oracle import OracleScene
from tests.test_gpu_parity import assert_hits_equal, random_rays

FMAX = 3.4028234663852886e38


def _wall(x):
    return Mesh(np.array([[x, -1, -1], [x, 1, -1], [x, 0, 1]], np.float32), np.array([[0, 1, 2]], np.int32))


def _two_walls():
    """An instanced triangle at x = 0 before a plain one at x = 4."""
    s = SceneDesc(camera=Camera.look_at(8, 8, 40.0, (-5.0, 0.0, 0.0), (0.0, 0.0, 0.0)), name="two walls")
    m = procedural.cornell_box(8, 8)[0].materials[0]
    m.tex_r = s.add_const(0.5)
    mat = s.add_material(m)
    s.blas.append([Group(N.GROUP_MESH, s.add_mesh(_wall(0.0)))])
    s.groups.append(Group(N.GROUP_INSTANCE, 0, material=mat))
    s.groups.append(Group(N.GROUP_MESH, s.add_mesh(_wall(4.0)), material=mat))
    return s


def _instances():
    s = procedural.instanced_spheres(32, 32, sphere_n=12, grid=4, env_w=32, env_h=16)[0]
    mat = s.groups[0].material
    for c in ((0.0, 0.9, 0.0), (2.6, 2.4, 2.6), (-2.6, 0.3, 1.3)):          # spheres among the instances
        s.spheres.append(Sphere(c, 0.6))
        s.groups.append(Group(N.GROUP_SPHERE, len(s.spheres) - 1, material=mat))
    tilt = Mat4.scale((0.5, 2.0, 1.0)) * Mat4.translation((0.0, 3.0, 0.0))
    s.groups.append(Group(N.GROUP_INSTANCE, 0, material=mat, model_to_world=tilt))
    return s


def _finite_rays(n, seed, want):
    """Rays of any direction length whose max_t lies around what they can hit:
    drawn, and at the oracle's own hit distance and its neighbours (`want`:
    rays -> the oracle's hits)."""
    rng = np.random.default_rng(seed)
    rays = random_rays(((-6, 0, -6), (6, 4, 6)), n, seed)
    rays["d"] *= np.exp2(rng.integers(-3, 4, n)).astype(np.float32)[:, None]
    rays["max_t"] = (rng.random(n) * 12).astype(np.float32)
    unit = random_rays(((-6, 0, -6), (6, 4, 6)), n, seed + 1)
    unit["max_t"] = FMAX
    t = want(unit)["t"]
    for k in range(3):
        r = unit[k::3]
        r["max_t"] = t[k::3]
        if k:
            r["max_t"] = np.nextafter(r["max_t"], np.float32(0 if k == 1 else FMAX))
    return np.concatenate([rays, unit])


def test_a_first_hit_in_an_instance_lets_max_t_grow():
    orc = OracleScene(_two_walls())
    try:
        rays = np.zeros(1, dtype=N.ray_dtype())
        rays["o"], rays["d"], rays["min_t"], rays["max_t"] = (-5, 0, 0), (2, 0, 0), 1e-4, 4.0
        h = orc.trace_closest(rays)
        assert h["prim"][0] == 1 and h["t"][0] == 4.5       # the plain wall, beyond max_t
    finally:
        orc.close()


@pytest.mark.gpu
@pytest.mark.parametrize("scene", [_two_walls, _instances])
def test_finite_rays_over_instances(dev, scene):
    s = scene()
    orc = OracleScene(s)
    try:
        rays = _finite_rays(20003, 5, orc.trace_closest)
        far = np.zeros(64, dtype=N.ray_dtype())
        far["o"], far["min_t"], far["max_t"] = (-5, 0, 0), 1e-4, 4.0
        far["d"][:, 0] = np.linspace(0.5, 4.0, 64)
        rays = np.concatenate([rays, far])
        want_h, want_a = orc.trace_closest(rays), orc.trace_any(rays)
    finally:
        orc.close()
    assert ((want_h["prim"] >= 0) & (want_h["t"] > rays["max_t"])).sum() > 10
    dev.upload(s)
    for counting in (False, True):
        dev.set_counting(counting)
        try:
            assert_hits_equal(dev.trace_closest(rays), want_h)
            assert np.array_equal(dev.trace_any(rays).astype(np.uint8), want_a.astype(np.uint8))
        finally:
            dev.set_counting(False)


class _Moved(Mat4):
    """A model-to-world matrix whose world-to-model counterpart is the identity:
    the scene description takes any two."""
    def invert(self):
        return Mat4.identity()


def _far_plane_scene():
    """A camera whose far plane lies 6 away.  The instance is hit in model space
    at 5, but its point lands at 13; a lit wall at 9, beyond the far plane, is
    then nearer."""
    s = SceneDesc(camera=Camera.look_at(16, 12, 30.0, (-5.0, 0.0, 0.0), (0.0, 0.0, 0.0), far=6.0), name="far plane")
    m = procedural.cornell_box(8, 8)[0].materials[0]
    m.tex_r = s.add_const(0.5)
    mat = s.add_material(m)
    low = Mesh(np.array([[-12, -9, -1], [-12, -8, -1], [-12, -8.5, 1]], np.float32), np.array([[0, 1, 2]], np.int32))
    s.blas.append([Group(N.GROUP_MESH, s.add_mesh(_wall(0.0))), Group(N.GROUP_MESH, s.add_mesh(low))])
    s.groups.append(Group(N.GROUP_INSTANCE, 0, material=mat, model_to_world=_Moved(Mat4.translation((8.0, 0.0, 0.0)).m)))
    lit = Mesh(_wall(4.0).positions, np.array([[0, 2, 1]], np.int32))        # faces the camera
    s.groups.append(Group(N.GROUP_MESH, s.add_mesh(lit), material=mat, emissive=True, le=(3.0, 2.0, 1.0)))
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("integrator", [N.INTEGRATOR_PATH, N.INTEGRATOR_VOL_PATH])
def test_camera_rays_whose_max_t_grows(dev, integrator):
    s = _far_plane_scene()
    st = procedural.cornell_box(8, 8)[1].replace(spp=3, max_depth=3, integrator=integrator)
    orc = OracleScene(s)
    try:
        want = orc.render(st)
    finally:
        orc.close()
    assert (want.sum(2) > 1.0).sum() > 10               # pixels that see the lit wall
    dev.upload(s)
    try:
        for finish in (0, -1):
            assert dev.lib.rt_debug_set_finish(dev.h, finish) == N.RT_OK
            for mode in (N.RENDERER_WAVEFRONT, N.RENDERER_WAVEFRONT_GRAPH, N.RENDERER_MEGAKERNEL):
                dev.set_renderer(mode)
                assert np.array_equal(dev.render(st).view(np.uint32), want.view(np.uint32)), (finish, mode)
    finally:
        dev.lib.rt_debug_set_finish(dev.h, -1)
        dev.set_renderer(N.RENDERER_AUTO)


@pytest.mark.gpu
def test_transmittance_walks_over_instances(dev):
    """vol_path's walks to a light are closest-hit rays that end at it."""
    s, st = procedural.volume_sphere(24, 20, sphere_n=6)
    s.blas.append([Group(N.GROUP_MESH, s.groups[0].ref)])
    mat = s.groups[1].material
    for i in range(5):
        s.groups.append(Group(N.GROUP_INSTANCE, 0, material=mat if i % 2 else -1, medium_inside=s.groups[0].medium_inside,
                              model_to_world=Mat4.scale((0.4, 0.3, 0.5)) * Mat4.translation((i - 2.0, 1.5 + 0.3 * i, 0.4))))
    st = st.replace(spp=4, max_depth=8)
    orc = OracleScene(s)
    try:
        want = orc.render(st)
    finally:
        orc.close()
    dev.upload(s)
    try:
        for mode in (N.RENDERER_WAVEFRONT, N.RENDERER_WAVEFRONT_GRAPH, N.RENDERER_MEGAKERNEL):
            dev.set_renderer(mode)
            assert np.array_equal(dev.render(st).view(np.uint32), want.view(np.uint32)), mode
    finally:
        dev.set_renderer(N.RENDERER_AUTO)
