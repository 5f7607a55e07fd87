"""Box pairs where the FP32 copies of the sweep cannot decide: bounds that are equal or one FP64 step apart, magnitudes
from FP64's subnormals to 1e300, infinite and NaN bounds.  The pairs are those of the closed FP64 interval test."""
import numpy as np
import pytest

from woo_gb300 import abi

pytestmark = pytest.mark.gpu


def _boxes(n, scale, rng):
    """Boxes whose bounds lie on a few values and their neighbours in FP64, so that many touch exactly, just overlap
    or just miss."""
    grid = scale * np.array([-2.0, -1.0, 0.0, 0.3, 1.0, 1.7, 3.0])
    k = rng.integers(0, 6, (n, 3))
    step = rng.integers(-1, 2, (2, n, 3))
    b = [np.where(s < 0, np.nextafter(g, -np.inf), np.where(s > 0, np.nextafter(g, np.inf), g))
         for s, g in zip(step, (grid[k], grid[k + 1]))]
    return b[0], b[1]


def _check(lo, hi):
    n = len(lo)
    got = abi.Handle(n).collide_boxes(lo, hi, np.full(n, 5, np.uint32), 2)
    with np.errstate(invalid="ignore"):
        ok = ((lo[:, None] <= hi[None]) & (hi[:, None] >= lo[None])).all(2)
    i, j = np.nonzero(np.triu(ok, 1))
    assert np.array_equal(got, np.stack([i, j], axis=1))
    return len(i)


@pytest.mark.parametrize("scale", [5e-324, 1e-310, 1e-50, 2e-45, 1e-44, 1e-40, 1.2e-38, 1e-37, 1e-30, 1e-3, 1.0, 1e30, 3e38, 1e39, 1e150, 1e299])
def test_touching_boxes(wdem_lib, scale):
    assert _check(*_boxes(400, scale, np.random.default_rng(3))) > 400


@pytest.mark.parametrize("scale", [1e-50, 1e-44, 1.0, 3e38, 1e39, 1e299])
def test_large_boxes(wdem_lib, scale):
    """Boxes with some infinite or NaN bounds against boxes that touch their finite ones."""
    rng = np.random.default_rng(4)
    lo, hi = _boxes(400, scale, rng)
    big = rng.random(400) < 0.1
    kind = rng.integers(0, 5, (400, 3))
    lo[big[:, None] & ((kind == 0) | (kind == 2))] = -np.inf
    hi[big[:, None] & ((kind == 1) | (kind == 2))] = np.inf
    nan = np.nonzero(big)[0][:3]
    lo[nan[:2], 0] = np.nan
    hi[nan[1:], 2] = np.nan
    assert _check(lo, hi) > 400
