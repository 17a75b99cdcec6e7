"""Neighbour rows and bond rows longer than a group of lanes keeps in shared
memory (112 partners, 64 bonds) and than the tiles they are ranked in (128):
the candidates and bonds against all pairs, and the FP64 steps that sum along
these rows against the oracle bit for bit, with rebuilds on the way."""
import numpy as np
import pytest

from godar_b200 import generators as gen
from godar_b200.lib import P_BONDS, P_CANDIDATES
from godar_b200.params import (BC_OPEN_BOTTOM, BC_OPEN_LEFT, BC_OPEN_RIGHT, BC_OPEN_TOP, PREC_FP64, PREC_MIXED,
                               make_params)

from .helpers import DIAG, STATE, check_mixed_positions, gpu_for, run_both

pytestmark = pytest.mark.gpu

OPEN = BC_OPEN_LEFT | BC_OPEN_RIGHT | BC_OPEN_BOTTOM | BC_OPEN_TOP


def _params(L, **kw):
    return make_params(L, L, **{**dict(cohesion=1, shelter=0, ridging=0, dt=1e-3, rtree=2000.0, bond_lim=0.0,
                                       bond_lim_rel=0.06, ua=12.0, va=-6.0, boundary=OPEN), **kw})


def _packed(n):
    """n floes that are all candidates of one another, many of them bonded."""
    rng = np.random.default_rng(n)
    m = int(np.ceil(np.sqrt(n)))
    at = rng.permutation(m * m)[:n]
    sp = 60.0
    x = 1000.0 + (at % m) * sp + rng.uniform(-1.0, 1.0, n)
    y = 1000.0 + (at // m) * sp + rng.uniform(-1.0, 1.0, n)
    r = rng.uniform(28.0, 28.9, n)
    return gen.Field("packed", _params(4000.0), x, y, r, rng.uniform(0.5, 2.0, n), 10,
                     u=10.0 + rng.uniform(-0.5, 0.5, n), v=rng.uniform(-0.5, 0.5, n))


def _ring(k, at):
    """A large floe of id `at` in a ring of k small ones that all bond to it."""
    rng = np.random.default_rng(k)
    r0 = 30.0
    R = r0 * (k + 2) / np.pi
    a = 2.0 * np.pi * np.arange(k) / k
    d = R + r0 + rng.uniform(0.0, 1.0, k)
    o = rng.permutation(k)
    L = 4.0 * R + 4000.0
    x = np.insert((d * np.cos(a))[o], at, 0.0) + 0.5 * L
    y = np.insert((d * np.sin(a))[o], at, 0.0) + 0.5 * L
    r = np.insert(np.full(k, r0), at, R)
    n = k + 1
    return gen.Field("ring", _params(L, bond_lim_rel=0.0, bond_lim=2.0), x, y, r, rng.uniform(0.5, 2.0, n), 10,
                     u=10.0 + 0.01 * R + rng.uniform(-0.2, 0.2, n), v=rng.uniform(-0.2, 0.2, n))


def _all_pairs(f):
    p = f.params
    dx, dy = f.x[:, None] - f.x[None, :], f.y[:, None] - f.y[None, :]
    d = np.sqrt(dx * dx + dy * dy)
    i, j = np.nonzero((d <= f.r[:, None] + p.rtree) & (np.arange(f.n)[:, None] < np.arange(f.n)[None, :]))
    gap = (f.r[i] + f.r[j]) - d[i, j]
    lim = p.bond_lim + p.bond_lim_rel * (f.r[i] + f.r[j])
    return list(zip(i, j)), list(zip(i[gap >= -lim], j[gap >= -lim]))


def _check(f):
    cands, bonds = _all_pairs(f)
    for precision in (PREC_FP64, PREC_MIXED):
        g = gpu_for(f, precision)
        g.step(1, 0, 1)
        if f.name == "packed":          # (the first step may part a ring's candidate by a rounding)
            assert list(zip(*g.pairs(P_CANDIDATES)[:2])) == cands
        assert list(zip(*g.pairs(P_BONDS)[:2])) == bonds
        g.close()
    # a common drift past half the skin (0.5 % of the largest radius and rtree)
    o, g = run_both(f, 1500, chunks=3)
    moved = np.hypot(g.field("x") - f.x, g.field("y") - f.y).max()
    assert moved > 0.005 * (f.r.max() + f.params.rtree)
    want = o.floes()
    for k in STATE + DIAG:
        assert g.field(k).tobytes() == want[k].tobytes(), k
    m = gpu_for(f, PREC_MIXED)
    m.step(1, 0, 1500)
    check_mixed_positions(f, m, g, onsets=True)
    for s in (g, m):
        s.close()
    return cands, bonds


@pytest.mark.parametrize("n", [113, 114, 129, 130, 300])
def test_rows_of_every_floe(n):
    cands, _ = _check(_packed(n))
    assert len(cands) == n * (n - 1) // 2          # n - 1 partners a floe


@pytest.mark.parametrize("k", [63, 64, 65, 66, 200])
def test_a_large_floes_bonds(k):
    for at in (0, k // 2, k):
        _, bonds = _check(_ring(k, at))
        assert sum(at in b for b in bonds) == k
