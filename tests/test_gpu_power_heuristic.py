"""The device's PowerHeuristic (binary32 pairs, binary64 where they cannot
decide) against the reference's binary64 expression: the same bits everywhere,
at the ends of the short form's range, near ties and powers of two, and for
zeros, infinities and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs(kind):
    rng = np.random.default_rng(len(kind))
    n = 1_000_003
    if kind == "wide":                       # over and beyond the short form's range
        f, g = np.exp2(rng.uniform(-40, 40, (2, n)))
    elif kind == "near_range_end":
        f = np.exp2(rng.choice([-30.0, 30.0], n)) * (1 + rng.integers(-4, 5, n) * 2.0 ** -24)
        g = np.exp2(rng.uniform(-31, 31, n))
    elif kind == "small_ratios":             # quotients with few bits: ties between binary32 values
        f, g = rng.integers(1, 1025, (2, n)) / 64.0
    elif kind == "towards_one":              # f >> g and g >> f
        f, g = np.exp2(rng.uniform(0, 1, n)), np.exp2(rng.uniform(-16, 16, n))
    else:
        v = np.array([0.0, -0.0, 1.0, 2.0 ** -30, 2.0 ** 30, 1e-45, 1e-38, 3.4e38, np.inf, np.nan, 0.5, 1e-20, 1e20])
        f, g = (a.reshape(-1) for a in np.meshgrid(v, v))
    return f.astype(np.float32), g.astype(np.float32)


@pytest.mark.parametrize("kind", ["wide", "near_range_end", "small_ratios", "towards_one", "special"])
def test_power_heuristic_equals_binary64(dev, kind):
    f, g = _pairs(kind)
    got = dev.detmath(8, f, g)
    f64, g64 = f.astype(np.float64), g.astype(np.float64)
    with np.errstate(all="ignore"):
        want = ((f64 * f64) / (f64 * f64 + g64 * g64)).astype(np.float32)
    same = (got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want))
    assert same.all(), (f[~same][:4], g[~same][:4], got[~same][:4], want[~same][:4])
