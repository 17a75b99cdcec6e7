"""Steps of small batches as one or two launches against the five step
kernels, bit for bit: sizes at the edges of the rules that choose between one
cluster, two launches with the sums by groups of lanes (one to eight rounds a
block) and two launches with one thread per floe, and rows that overflow a
group's list.  The five kernels are compared with the oracle elsewhere."""
import numpy as np
import pytest

from godar_b200 import generators as gen
from godar_b200.lib import FLOE_FIELDS, P_BONDS, P_CONTACTS, Stepper
from godar_b200.params import BC_PERIODIC_Y, PREC_FP64, PREC_MIXED, make_params

pytestmark = pytest.mark.gpu


def _ring(shelter):
    """Large floes, each in a ring of small ones that touch or nearly touch
    it: about 60 pairs a large floe that add to its sums."""
    rng = np.random.default_rng(4)
    R, r0, m = 3000.0, 140.0, 60
    x, y, r = [], [], []
    for cx, cy in ((9000.0, 9000.0), (18000.0, 9500.0)):
        x.append(cx), y.append(cy), r.append(R)
        for k in range(m):
            a = 2.0 * np.pi * k / m
            d = R + r0 + rng.uniform(-0.01, 2.0)
            x.append(cx + d * np.cos(a)), y.append(cy + d * np.sin(a)), r.append(r0)
    n = len(x)
    # small floes of lower and of higher id than their large one
    order = rng.permutation(n)
    p = make_params(3e4, 2.4e4, cohesion=1, shelter=shelter, ridging=shelter, dt=1e-3, rtree=3000.0, bond_lim=0.0,
                    bond_lim_rel=0.05, bond_frac=0.7, bond_seed=3, ua=12.0, va=-5.0, uw=0.1, vw=0.0,
                    boundary=BC_PERIODIC_Y)
    h = rng.uniform(0.5, 2.0, n)
    return gen.Field("ring", p, np.array(x)[order], np.array(y)[order], np.array(r)[order], h, 10,
                     u=rng.uniform(-0.2, 0.2, n), v=rng.uniform(-0.2, 0.2, n))


def _run(f, precision, fused, monkeypatch):
    monkeypatch.setenv("GODAR_FUSED", fused)
    s = Stepper(f.params, f.n, precision)
    s.upload(f.x, f.y, f.r, f.h, f.theta, f.omega, f.u, f.v)
    if f.forcing is not None:
        s.set_field(f.forcing)
    s.step(1, 0, 3)
    s.set_diagnostics(False)
    s.step(4, 0, 11)
    s.step_async(15)
    s.step_async(16)
    s.set_diagnostics(True)
    s.step_async(17)
    out, contacts = s.download(which=P_CONTACTS)
    out["stats"] = np.array(list(s.stats()[1].values()))
    for k, lists in (("contact", contacts), ("bond", s.pairs(P_BONDS))):
        for q, a in enumerate(lists):
            out[f"{k}{q}"] = a
    s.close()
    return out


def _same(f, precision, monkeypatch):
    a, b = (_run(f, precision, fused, monkeypatch) for fused in ("1", "0"))
    assert np.isfinite(a["x"]).all()
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k
    assert set(FLOE_FIELDS) <= set(a)


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [64, 390, 420, 970, 1010, 9472, 9473, 65536, 65537, 102400, 102401, 122880, 122881])
def test_bonded_fields(n, precision, monkeypatch):
    _same(gen.bonded_field(n=n, seed=n, device="gpu" if n > 9000 else "cpu"), precision, monkeypatch)


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [300, 9473, 18945, 37889])
def test_sheltering_fields(n, precision, monkeypatch):
    _same(gen.polydisperse_field(n=n, seed=2, phi=0.6, dt=1e-3), precision, monkeypatch)


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("shelter", [0, 1])
def test_rows_longer_than_a_group_lists(shelter, precision, monkeypatch):
    _same(_ring(shelter), precision, monkeypatch)
