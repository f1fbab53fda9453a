"""The wide tree of boxes that reach to infinity (a sphere whose centre plus
radius overflows, a vertex at infinity): a quantised child box still covers
every finite coordinate of its exact box, and the finite boxes beside it."""
import numpy as np
import pytest

from tests.test_cpu_oracle import _lib_bvh, _lib_wide

FMAX = float(np.finfo(np.float32).max)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("count", [1, 3])
def test_quantised_boxes_cover_unbounded_ones(axis, count):
    rng = np.random.default_rng(10 * axis + count)
    lo = rng.random((60, 3)).astype(np.float32) * 10 - 5
    boxes = np.concatenate([lo, lo + 0.5], axis=1)
    boxes[7:7 + count, 3 + axis] = np.inf
    b, w = _lib_bvh(boxes), _lib_wide(boxes)
    unbounded = 0
    for i in range(w["nchild"].size):
        s = np.ldexp(1.0, w["e"][i].astype(np.int64) - 127)
        for c in range(int(w["nchild"][i])):
            bn = w["child"][i, c]
            qlo = w["p"][i].astype(np.float64) + w["qlo"][i, :, c] * s
            qhi = w["p"][i].astype(np.float64) + w["qhi"][i, :, c] * s
            ex_hi = b["bounds"][bn, 3:].astype(np.float64)
            unbounded += int(np.isinf(ex_hi).any())
            assert (qlo <= b["bounds"][bn, :3]).all(), (i, c)
            assert (qhi >= np.minimum(ex_hi, FMAX)).all(), (i, c, qhi, ex_hi)
    assert unbounded >= count
