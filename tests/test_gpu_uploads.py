"""Fields admitted together: their arrays leave through the pinned slots
gathered into long copies, whatever sizes meet (a slot's edge, one floe, more
than two slots, restart lists of bonds), and read back as they were given."""
import numpy as np
import pytest

from godar_b200.lib import Batch
from godar_b200.params import BC_PERIODIC_X, BC_PERIODIC_Y, PREC_FP64, PREC_MIXED, make_params

pytestmark = pytest.mark.gpu

STATE = ["x", "y", "u", "v", "r", "h", "theta", "omega"]


def _field(n, seed, restart):
    rng = np.random.default_rng(seed)
    m = int(np.ceil(np.sqrt(n)))
    sp = 120.0
    L = max(m * sp, 4000.0)
    p = make_params(L, L, cohesion=1, shelter=0, ridging=0, dt=1e-3, rtree=150.0, bond_lim=1.0, ua=5.0,
                    boundary=BC_PERIODIC_X | BC_PERIODIC_Y)
    k = np.arange(n)
    s = {"x": (k % m + 0.5) * sp, "y": (k // m + 0.5) * sp, "r": rng.uniform(59.0, 59.9, n),
         "h": rng.uniform(0.5, 2.0, n)}
    for name in ("theta", "omega", "u", "v"):
        s[name] = rng.uniform(-1e-3, 1e-3, n)
    bonds = None
    if restart:
        b = np.stack([k[:-1], k[1:]], 1)
        bonds = b[(b[:, 1] % m) != 0]
    return p, s, bonds


def _add(b, f):
    p, s, bonds = f
    return b.add(p, s["x"], s["y"], s["r"], s["h"], s["theta"], s["omega"], s["u"], s["v"], bonds=bonds,
                 restart=0 if bonds is None else 1)


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_fields_admitted_together(precision):
    # 16,384 doubles fill a slot, 32,768 both, 32,769 go directly
    sizes = [1, 16383, 16384, 16385, 2, 32768, 32769, 40000, 3] + [7] * 60 + [500, 16381, 1]
    fields = [_field(n, 100 + k, k % 3 == 1) for k, n in enumerate(sizes)]
    b = Batch(precision)
    first = [_add(b, f) for f in fields[:5]]
    b.step(1)
    ids = first + [_add(b, f) for f in fields[5:]]
    for hid, (_, s, _) in list(zip(ids, fields))[5:]:
        for name in STATE:
            assert b.field(hid, name).tobytes() == s[name].tobytes(), (len(s["x"]), name)
    b.step(3)
    for k, hid in enumerate(ids):
        if sizes[k] == 7 and k % 9:
            continue
        one = Batch(precision)
        i = _add(one, fields[k])
        one.step(4 if k < 5 else 3)
        for name in STATE:
            assert b.field(hid, name).tobytes() == one.field(i, name).tobytes(), (sizes[k], name)
        one.close()
    b.close()


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("fields", [1, 2, 3, 4, 8, 15, 16, 24, 32, 48, 64])
def test_parameters_and_forcing_grids_of_many_fields(fields, precision):
    # one copy must not cross from one buffer into the next, which for some
    # numbers of fields begins where the first ends
    rng = np.random.default_rng(fields)
    made = []
    for k in range(fields):
        p, s, _ = _field(6 + k % 3, k, False)
        p.field_nx, p.field_ny = 4, 4
        made.append((p, s, rng.uniform(-1.0, 1.0, 64)))

    def add(b, f):
        p, s, grid = f
        return b.add(p, s["x"], s["y"], s["r"], s["h"], s["theta"], s["omega"], s["u"], s["v"], field=grid)

    for _ in range(2):
        b = Batch(precision)
        ids = [add(b, f) for f in made]
        b.step(3)
        for k in {0, fields // 2, fields - 1}:
            one = Batch(precision)
            i = add(one, made[k])
            one.step(3)
            for name in STATE:
                assert b.field(ids[k], name).tobytes() == one.field(i, name).tobytes(), (k, name)
            one.close()
        b.close()
