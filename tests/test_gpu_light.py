"""The step kernels of batches without ridging, sheltering and walls (shapes
not written, rebuild positions read only near the skin), on fast floes that
expire the rows many times, with and without a contact list, and when a field
with ridging joins and leaves: against the merged steps of small batches,
which write and read everything, bit for bit."""
import numpy as np
import pytest

from godar_b200.lib import Batch
from godar_b200.params import BC_PERIODIC_X, BC_PERIODIC_Y, PREC_FP64, PREC_MIXED, make_params

pytestmark = pytest.mark.gpu

NAMES = ("x", "y", "u", "v", "omega", "r", "h")


def _grid(n, gap, speed, drift, ridging, seed):
    """Floes on a jittered grid, `gap` of their spacing apart, with a common
    and random velocities; a periodic domain."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(np.sqrt(n)))
    d = 250.0
    at = np.arange(n)
    x = (at % m + 0.5) * d + rng.uniform(-0.02, 0.02, n) * d
    y = (at // m + 0.5) * d + rng.uniform(-0.02, 0.02, n) * d
    r = rng.uniform(0.45, 0.5, n) * d * (1.0 - gap)
    p = make_params(m * d, m * d, cohesion=0, shelter=0, ridging=ridging, dt=0.05, rtree=400.0,
                    boundary=BC_PERIODIC_X | BC_PERIODIC_Y)
    return p, x, y, r, rng.uniform(0.5, 2.0, n), drift + rng.uniform(-speed, speed, (2, n))


def _run(precision, n, gap, speed, drift, fused, monkeypatch):
    monkeypatch.setenv("GODAR_FUSED", fused)
    b = Batch(precision)

    def add(ridging, seed):
        p, x, y, r, h, (u, v) = _grid(n, gap, speed, drift, ridging, seed)
        return b.add(p, x, y, r, h, u=u, v=v)

    out, hs = [], [add(0, 1), add(0, 2)]

    def go():
        b.step(1)                       # a diagnostic step among plain ones
        b.set_diagnostics(False)
        b.step(37)
        for _ in range(5):
            b.step_async(1)
        b.set_diagnostics(True)
        b.step(3)
        out.extend(b.field(k, name) for k in hs for name in NAMES)

    go()
    hs.append(add(1, 3))
    go()
    b.remove(hs.pop())
    go()
    out.append(np.array(b.stats()["rebuilds"]))
    b.close()
    return out


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,gap,speed,drift", [(300, 0.04, 8.0, 0.0), (1300, 0.04, 40.0, 0.0), (500, 0.4, 1.0, 60.0)])
def test_light_steps(precision, n, gap, speed, drift, monkeypatch):
    a, b = (_run(precision, n, gap, speed, drift, fused, monkeypatch) for fused in ("1", "0"))
    assert all(np.isfinite(v).all() for v in a)
    assert a[-1] > 4
    for k, (p, q) in enumerate(zip(a, b)):
        assert p.tobytes() == q.tobytes(), k
