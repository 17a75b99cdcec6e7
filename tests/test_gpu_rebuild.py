"""The neighbour search over the forms its cell walk, rows and lists meet:
boundaries of every kind, domains a few cells wide, floes outside a wall-less
domain, rows longer than a group keeps in shared memory (on either side of the
limit), fields of one floe, many small fields beside a large one.  Candidates
and bonds are compared with a restatement of their rules over all pairs."""
import numpy as np
import pytest

from godar_b200.lib import P_BONDS, P_CANDIDATES, Batch, Stepper
from godar_b200.params import (BC_OPEN_BOTTOM, BC_OPEN_LEFT, BC_OPEN_RIGHT, BC_OPEN_TOP, BC_PERIODIC_X,
                               BC_PERIODIC_Y, PREC_FP64, PREC_MIXED, make_params)

pytestmark = pytest.mark.gpu

OPEN = BC_OPEN_LEFT | BC_OPEN_RIGHT | BC_OPEN_BOTTOM | BC_OPEN_TOP


def _points(n, Lx, Ly, r, seed, spill=0.0):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-spill * Lx, (1 + spill) * Lx, n)
    y = rng.uniform(-spill * Ly, (1 + spill) * Ly, n)
    return x, y, rng.uniform(0.5 * r, r, n), rng.uniform(0.5, 2.0, n)


def _grid(n, Lx, Ly, r, seed):
    """Floes that do not overlap: on a jittered grid."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(np.sqrt(max(n, 36))))
    at = rng.permutation(m * m)[:n]
    sx, sy = Lx / m, Ly / m
    x = (at % m + 0.5) * sx + rng.uniform(-0.02, 0.02, n) * sx
    y = (at // m + 0.5) * sy + rng.uniform(-0.02, 0.02, n) * sy
    return x, y, rng.uniform(0.6, 1.0, n) * min(r, 0.47 * sy), rng.uniform(0.5, 2.0, n)


def _all_pairs(p, x, y, r):
    dx, dy = x[:, None] - x[None, :], y[:, None] - y[None, :]
    for d, L, per in ((dx, p.nx, p.boundary & BC_PERIODIC_X), (dy, p.ny, p.boundary & BC_PERIODIC_Y)):
        if per:
            d[d > 0.5 * L] -= L
            d[d < -0.5 * L] += L
    dist = np.sqrt(dx * dx + dy * dy)
    i, j = np.nonzero((dist <= r[:, None] + p.rtree) & (np.arange(len(x))[:, None] < np.arange(len(x))[None, :]))
    gap = (r[i] + r[j]) - dist[i, j]
    lim = p.bond_lim + p.bond_lim_rel * (r[i] + r[j])
    return list(zip(i, j)), list(zip(i[gap >= -lim], j[gap >= -lim]))


# a floe between two chosen counts of partners: all within the search radius
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("boundary", [0, OPEN, BC_PERIODIC_X | BC_PERIODIC_Y, BC_PERIODIC_X, BC_PERIODIC_Y | BC_OPEN_LEFT])
@pytest.mark.parametrize("n,Lx,Ly,rtree,spill", [(1, 900.0, 900.0, 100.0, 0.0), (40, 900.0, 5000.0, 120.0, 0.0),
                                                 (113, 800.0, 800.0, 350.0, 0.0), (112, 800.0, 800.0, 350.0, 0.0),
                                                 (300, 900.0, 1000.0, 300.0, 0.0), (700, 9000.0, 7000.0, 400.0, 0.2)])
def test_candidates_and_bonds_of_the_first_step(n, Lx, Ly, rtree, spill, boundary, precision):
    if spill and boundary & (BC_PERIODIC_X | BC_PERIODIC_Y) or spill and boundary == 0:
        spill = 0.0          # only an open domain has floes outside it
    p = make_params(Lx, Ly, cohesion=1, shelter=0, ridging=0, dt=1e-9, rtree=rtree, bond_lim=0.0, bond_lim_rel=0.4,
                    boundary=boundary)
    x, y, r, h = _points(n, Lx, Ly, 6.0, n, spill)
    want_c, want_b = _all_pairs(p, x, y, r)
    s = Stepper(p, n, precision)
    s.upload(x, y, r, h)
    s.step(1, 0, 1)
    ci, cj, _ = s.pairs(P_CANDIDATES)
    bi, bj, _ = s.pairs(P_BONDS)
    assert list(zip(ci, cj)) == want_c
    assert list(zip(bi, bj)) == want_b
    s.close()


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_fields_of_many_sizes_step_as_alone(precision):
    sizes = [1, 2, 700, 3, 1, 45, 260, 1]
    fields = []
    for k, n in enumerate(sizes):
        p = make_params(4000.0, 3000.0, cohesion=1, shelter=0, ridging=0, dt=1e-3, rtree=150.0, bond_lim_rel=0.3,
                        ua=5.0 + k, boundary=OPEN if k % 2 else BC_PERIODIC_X | BC_PERIODIC_Y)
        fields.append((p, *_grid(n, 4000.0, 3000.0, 40.0, 50 + k)))
    b = Batch(precision)
    ids = []
    for f in fields:              # admitted one by one between steps, then some leave
        ids.append(b.add(*f))
        b.step(2)
    for k in (1, 2, 5):
        b.remove(ids[k])
    b.step(3)
    for k, f in enumerate(fields):
        if k in (1, 2, 5):
            continue
        one = Batch(precision)
        i = one.add(*f)
        one.step(2 * (len(fields) - k) + 3)
        for name in ("x", "y", "u", "v", "omega"):
            assert b.field(ids[k], name).tobytes() == one.field(i, name).tobytes(), (k, name)
        one.close()
    b.close()
