"""Pair lists of rows of every length: rows that a group keeps in shared memory,
rows ranked by a whole block (a large floe among small ones, of lowest, middle
and highest id), one block and several, against the lists of all pairs."""
import ctypes

import numpy as np
import pytest

from godar_b200 import lib as gl
from godar_b200.params import BC_OPEN_BOTTOM, BC_OPEN_LEFT, BC_OPEN_RIGHT, BC_OPEN_TOP, PREC_FP64, PREC_MIXED, make_params

pytestmark = pytest.mark.gpu

OPEN = BC_OPEN_LEFT | BC_OPEN_RIGHT | BC_OPEN_BOTTOM | BC_OPEN_TOP


def _field(n, large, at):
    """n - 1 small floes on a jittered grid around a large one of id `at`,
    which `large` of them are near to."""
    rng = np.random.default_rng(n + at)
    R, r = 3000.0, 20.0
    ring = max(large, 1)
    a = 2 * np.pi * np.arange(ring) / ring
    d = R + 30.0 + (np.arange(ring) % 12) * 55.0
    x, y = d * np.cos(a), d * np.sin(a)
    rest = n - 1 - large
    m = int(np.ceil(np.sqrt(max(rest, 1))))
    q = np.arange(rest)
    x = np.r_[x[:large], 6000.0 + (q % m) * 60.0]
    y = np.r_[y[:large], (q // m) * 60.0]
    o = rng.permutation(n - 1)
    x = np.insert(x[o], at, 0.0) + 20000.0
    y = np.insert(y[o], at, 0.0) + 20000.0
    rr = np.insert(np.full(n - 1, r) * rng.uniform(0.9, 1.0, n - 1), at, R)
    return x, y, rr, np.ones(n)


def _want(x, y, r, rtree):
    out = []
    for i in range(len(x)):
        d = np.sqrt((x[i] - x[i + 1:]) * (x[i] - x[i + 1:]) + (y[i] - y[i + 1:]) * (y[i] - y[i + 1:]))
        out += [(i, i + 1 + j) for j in np.nonzero(d <= r[i] + rtree)[0]]
    return out


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,large", [(2, 1), (30, 20), (30, 21), (80, 64), (80, 65), (500, 129), (1500, 900),
                                     (2048, 0), (2049, 700), (4000, 1400)])
def test_candidates_in_order(n, large, precision):
    for at in sorted({0, n // 2, n - 1}):
        x, y, r, h = _field(n, large, at)
        p = make_params(40000.0, 40000.0, cohesion=0, shelter=0, ridging=0, dt=1e-9, rtree=800.0, boundary=OPEN)
        s = gl.Stepper(p, n, precision)
        s.upload(x, y, r, h)
        s.step(1, 0, 1)
        i, j, v = s.pairs(gl.P_CANDIDATES)
        assert list(zip(i, j)) == _want(x, y, r, 800.0)
        if at == 0 and large:
            assert np.sum(i == 0) >= large          # the large floe's row
        m = len(i)
        for cap in {1, m // 3, m - 1, m + 5} - {0, -1}:
            cnt = ctypes.c_int(-1)
            pi, pj = np.full(cap, -7, np.int32), np.full(cap, -7, np.int32)
            pv = np.full(cap, np.nan)
            gl._check(gl.load().godar_gpu_get_pairs(s._h, gl.P_CANDIDATES, gl._ptr(pi, gl._ip), gl._ptr(pj, gl._ip),
                                                    gl._ptr(pv), cap, ctypes.byref(cnt)))
            k = min(cap, m)
            assert cnt.value == m
            assert np.array_equal(pi[:k], i[:k]) and np.array_equal(pj[:k], j[:k]) and np.array_equal(pv[:k], v[:k])
        ti, tj, tv = s.pairs(gl.P_CONTACTS)
        assert np.array_equal(i[v > 0], ti) and np.array_equal(j[v > 0], tj)
        s.close()
