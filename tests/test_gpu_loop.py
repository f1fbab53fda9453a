"""The bounce loop itself (gpu).  Rounds of few paths end in one launch
(rt_finish.cu), and the films of most tests are that small, so tests of what
only the loop does - queue positions and the sort under bounds checks, its
iteration and bounce caps, slot reuse by several jobs, several rounds - run here
once more with the hand-over off (rt_debug_set_finish 0) in every context."""
import ctypes as C

import pytest

from radiantium_gb300 import native as N
from radiantium_gb300.device import Device
from tests import test_gpu_debug_bounds, test_gpu_failure
from tests.test_gpu_batch import (scenes, test_batch_all_light_strategy,  # noqa: F401
                                  test_batch_matches_single_renders, test_batch_of_volumes_matches_single_renders,
                                  test_batch_repeats_and_single_graph_render)
from tests.test_gpu_failure import test_wavefront_iteration_cap  # noqa: F401
from tests.test_gpu_particles import (test_tall_tree_wavefront_matches_megakernel,  # noqa: F401
                                      test_wavefront_rounds, test_wavefront_small_slot_pool)

pytestmark = pytest.mark.gpu

# the same in a child process: every context that it makes keeps the loop
PRELUDE = r'''
from radiantium_gb300.device import Device as _Device
_init = _Device.__init__
def _loop_only(self, *a, **k):
    _init(self, *a, **k)
    assert self.lib.rt_debug_set_finish(self.h, 0) == 0
_Device.__init__ = _loop_only
'''


def _loop(dev, paths=0):
    assert dev.lib.rt_debug_set_finish(C.c_void_p(dev.h.value), paths) == N.RT_OK


@pytest.fixture(scope="module", autouse=True)
def loop_only(dev):
    init = Device.__init__

    def made(self, *a, **k):
        init(self, *a, **k)
        _loop(self)

    with pytest.MonkeyPatch.context() as m:
        m.setattr(Device, "__init__", made)
        _loop(dev)
        yield
    _loop(dev, -1)


def test_debug_bounds_of_the_loop(tmp_path, monkeypatch):
    monkeypatch.setattr(test_gpu_debug_bounds, "CHILD", PRELUDE + test_gpu_debug_bounds.CHILD)
    test_gpu_debug_bounds.test_debug_bounds_build(tmp_path)


def test_caps_of_the_loop(tmp_path, monkeypatch):
    monkeypatch.setattr(test_gpu_failure, "CHILD", PRELUDE + test_gpu_failure.CHILD)
    test_gpu_failure.test_device_loop_caps(tmp_path)
