"""The calls of a monitored batch: summaries of fields at the edges of the
reduction's rounds, forcing set for more fields than one block sets, and
queued single steps against chunked ones."""
import numpy as np
import pytest

from godar_b200 import generators as gen
from godar_b200.lib import Batch
from godar_b200.params import BC_PERIODIC_X, BC_PERIODIC_Y, PREC_FP64, PREC_MIXED, make_params

pytestmark = pytest.mark.gpu


def _apart(n, seed, **kw):
    rng = np.random.default_rng(seed)
    m = max(6, int(np.ceil(np.sqrt(n))))
    at = np.arange(n)
    p = make_params(m * 400.0, m * 400.0, cohesion=0, shelter=0, ridging=0, dt=0.1, rtree=500.0,
                    boundary=BC_PERIODIC_X | BC_PERIODIC_Y, **kw)
    return p, (at % m + 0.5) * 400.0, (at // m + 0.5) * 400.0, rng.uniform(60.0, 150.0, n), rng.uniform(0.5, 3.0, n), \
        rng.uniform(-2.0, 2.0, (3, n))


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_summary_sizes(precision):
    sizes = [1, 2, 255, 256, 257, 1023, 1024, 1025, 2049, 5000]
    b = Batch(precision)
    hs, ps = [], []
    for k, n in enumerate(sizes):
        p, x, y, r, h, (u, v, om) = _apart(n, k)
        hs.append(b.add(p, x, y, r, h, u=u, v=v, omega=1e-3 * om))
        ps.append(p)
    b.step(2)
    got = b.summary()
    for k, (hid, n, p) in enumerate(zip(hs, sizes, ps)):
        r, h, u, v, om = (b.field(hid, q) for q in ("r", "h", "u", "v", "omega"))
        m = p.rhoice * np.pi * h * r * r
        terms = m * u, m * v, 0.5 * m * (u * u + v * v) + 0.25 * m * r * r * om * om
        for t, s in zip(terms, got[k]):
            # n sums of n terms, in another order
            assert abs(t.sum() - s) <= 4 * (n + 16) * 2.0 ** -53 * np.abs(t).sum(), (n, k)
        assert abs(got[k][3] - np.sqrt(u * u + v * v).max()) <= 2.0 ** -51 * got[k][3]
    b.close()


@pytest.mark.parametrize("fields", [1, 255, 257, 600])
def test_forcing_of_many_fields(fields):
    rng = np.random.default_rng(fields)
    uvw = rng.uniform(-10.0, 10.0, (fields, 4))
    out = []
    for late in (False, True):
        b = Batch(PREC_MIXED)
        hs = []
        for k in range(fields):
            f = {} if late else dict(zip(("ua", "va", "uw", "vw"), uvw[k]))
            p, x, y, r, h, (u, v, om) = _apart(3, 7, **f)
            hs.append(b.add(p, x, y, r, h, u=u, v=v))
        b.set_diagnostics(False)
        if late:
            b.set_uniform_forcing(uvw)
        for _ in range(5):
            b.step_async(1)
        b.wait()
        out.append([b.field(k, q).tobytes() for k in hs for q in ("x", "u", "v", "omega")])
        b.close()
    assert out[0] == out[1]


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_queued_steps_of_separate_kernels(precision, monkeypatch):
    monkeypatch.setenv("GODAR_FUSED", "0")
    f = gen.bonded_field(n=1500, seed=8)
    out = []
    for calls in ([40], [1] * 40, [3, 1, 1, 16, 1, 2, 16]):
        b = Batch(precision)
        hid = b.add_field(f)
        b.step(12)
        for k in calls:
            b.step_async(k)
        b.wait()
        out.append([b.field(hid, q).tobytes() for q in ("x", "y", "u", "omega", "tfx")])
        b.close()
    assert out[0] == out[1] == out[2]
