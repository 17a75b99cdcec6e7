"""Sheltering with one exponential for both directions of a pair (the factor
of the direction against the wind is exactly 1): the forms that decide which
way the factors are computed - wind along, across and against the pair, no
wind, no current, pairs that just touch (a quotient of zero by zero), floes of
equal and different freeboard, in contact and apart - against the FP64 oracle,
which computes every factor by itself, bit for bit."""
import numpy as np
import pytest

from godar_b200.lib import Stepper
from godar_b200.params import BC_OPEN_BOTTOM, BC_OPEN_LEFT, BC_OPEN_RIGHT, BC_OPEN_TOP, PREC_FP64, make_params
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

OPEN = BC_OPEN_LEFT | BC_OPEN_RIGHT | BC_OPEN_BOTTOM | BC_OPEN_TOP


def _field(gap, wind, current, seed):
    """A row of disks `gap` apart along x, with one above it."""
    rng = np.random.default_rng(seed)
    r = np.array([500.0, 500.0, 300.0, 700.0, 500.0])
    x = np.empty(5)
    x[0] = 2000.0
    for k in range(1, 5):
        x[k] = x[k - 1] + r[k - 1] + r[k] + gap
    y = np.full(5, 4000.0)
    y[4] += 900.0
    h = np.array([1.0, 1.0, 0.4, 2.5, 1.0])
    p = make_params(2e4, 1e4, cohesion=0, shelter=1, ridging=0, dt=0.01, rtree=4000.0, boundary=OPEN,
                    ua=wind[0], va=wind[1], uw=current[0], vw=current[1])
    return p, x, y, r, h, rng.uniform(-0.1, 0.1, 5), rng.uniform(-0.1, 0.1, 5)


@pytest.mark.parametrize("wind,current", [((10.0, 0.0), (0.0, 0.0)), ((-10.0, 0.0), (0.2, 0.0)),
                                          ((0.0, 10.0), (0.0, -0.2)), ((0.0, 0.0), (-0.1, 0.1)),
                                          ((7.0, -3.0), (0.1, 0.05))])
@pytest.mark.parametrize("gap", [0.0, -0.5, 30.0])
def test_both_directions_equal_the_oracle(gap, wind, current):
    p, x, y, r, h, u, v = _field(gap, wind, current, 3)
    z = np.zeros(5)
    o = po.Oracle(p, x, y, r, h, z, z, u, v)
    s = Stepper(p, 5, PREC_FP64)
    s.upload(x, y, r, h, z, z, u, v)
    for k in (1, 6):
        o.step(k)
        s.step(1, 0, k)
        ref = o.floes()
        for name in ("x", "y", "u", "v", "omega", "tfx", "tfy", "m"):
            got = s.field(name)
            assert np.array_equal(np.isnan(got), np.isnan(ref[name])), name
            fine = ~np.isnan(got)
            assert np.array_equal(got[fine].view(np.int64), ref[name][fine].view(np.int64)), (name, k)
    o.close()
    s.close()
