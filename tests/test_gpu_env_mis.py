"""MIS rays of infinite lights as any-hit rays (the wavefront, counting off):
films equal the oracle's bit for bit with one and two infinite lights beside
area lights, with a map that is black over half of its texels, and for every
material (specular ones take the ray's weight without a light pdf)."""
import numpy as np
import pytest

from radiantium_gb300 import native as N
from radiantium_gb300 import procedural
from radiantium_gb300.scene import Group, Mat4, Texture
from oracle.oracle import OracleScene

pytestmark = pytest.mark.gpu


def _half_black(seed):
    img = np.random.default_rng(seed).uniform(0.0, 2.0, (16, 32, 3)).astype(np.float32)
    img[:, ::2] = 0.0
    return Texture.from_image_hw3(img)


@pytest.mark.parametrize("strategy", [N.STRATEGY_UNIFORM, N.STRATEGY_ALL])
@pytest.mark.parametrize("maps", [1, 2])
def test_infinite_light_mis_rays(dev, maps, strategy):
    s, st = procedural.material_zoo(40, 28)
    env = [g for g in s.groups if g.kind == N.GROUP_INFINITE_LIGHT][0]
    env.ref = s.add_texture(_half_black(1))
    if maps == 2:
        s.groups.append(Group(N.GROUP_INFINITE_LIGHT, s.add_texture(_half_black(2)),
                              model_to_world=Mat4.from_axis_angle((1, 0, 0), 0.6)))
    st = st.replace(spp=6, strategy=strategy)
    dev.upload(s)
    orc = OracleScene(s)
    try:
        want = orc.render(st)
    finally:
        orc.close()
    try:
        for mode in (N.RENDERER_WAVEFRONT, N.RENDERER_WAVEFRONT_GRAPH):
            dev.set_renderer(mode)
            assert np.array_equal(dev.render(st).view(np.uint32), want.view(np.uint32)), mode
    finally:
        dev.set_renderer(N.RENDERER_AUTO)
