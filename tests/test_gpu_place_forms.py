"""Placement over the forms that decide how its cell lists are built and
walked: one disk, axes periodic or not, domains a few cells wide (wrapped
neighbours repeat), disks that cover thousands of the smallest class's cells,
negative and positive gaps.  Every placed disk lies in the domain without
overlap, and a call is a function of its inputs alone."""
import numpy as np
import pytest

from godar_b200.lib import place_disks

pytestmark = pytest.mark.gpu


def _check(x, y, r, Lx, Ly, px, py, gap):
    ok = np.isfinite(x)
    x, y, s = x[ok], y[ok], r[ok] + 0.5 * gap
    for a, L, per in ((x, Lx, px), (y, Ly, py)):
        if per:
            assert np.all((a >= 0) & (a <= L))
        else:
            assert np.all(a >= s - 1e-9 * L) and np.all(a <= L - s + 1e-9 * L)
    dx, dy = x[:, None] - x[None, :], y[:, None] - y[None, :]
    if px:
        dx -= Lx * np.round(dx / Lx)
    if py:
        dy -= Ly * np.round(dy / Ly)
    over = np.hypot(dx, dy) < (s[:, None] + s[None, :]) * (1 - 1e-12)
    np.fill_diagonal(over, False)
    assert not over.any()


@pytest.mark.parametrize("px,py", [(True, True), (True, False), (False, False)])
@pytest.mark.parametrize("name,r,Lx,Ly,gap", [
    ("one", [300.0], 1000.0, 900.0, 0.0),
    ("narrow", [100.0] * 12, 450.0, 2600.0, 0.0),
    ("mixed sizes", list(np.geomspace(900.0, 4.0, 300)), 7000.0, 6000.0, 0.0),
    ("tiny beside large", [400.0, 1.0, 1.0, 0.05, 0.01], 1300.0, 1200.0, 0.0),
    ("gap", list(np.linspace(20.0, 40.0, 200)), 1400.0, 1500.0, 3.0),
    ("overlap", list(np.linspace(20.0, 40.0, 200)), 1300.0, 1300.0, -4.0)])
def test_forms(name, r, Lx, Ly, gap, px, py):
    r = np.array(r)
    x, y, placed = place_disks(r, Lx, Ly, px, py, seed=11, max_rounds=64, gap=gap)
    assert placed == int(np.sum(np.isfinite(x))) > 0
    _check(x, y, r, Lx, Ly, px, py, gap)
    x2, y2, p2 = place_disks(r, Lx, Ly, px, py, seed=11, max_rounds=64, gap=gap)
    assert p2 == placed and x.tobytes() == x2.tobytes() and y.tobytes() == y2.tobytes()
