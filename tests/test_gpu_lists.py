"""Read-backs: pair lists come in ascending (i, j) whatever their length and
the caller's capacity (one block, and count - scan - fill above 8,192 floes;
through the staging buffer and past it), and one download of every field
equals the fields read one by one."""
import ctypes

import numpy as np
import pytest

from godar_b200 import generators as gen
from godar_b200 import lib as gl
from godar_b200.params import PREC_FP64, PREC_MIXED

pytestmark = pytest.mark.gpu


def _pairs(s, which, cap):
    """The first cap pairs and the length the call reports."""
    cnt = ctypes.c_int(-1)
    pi, pj = np.full(cap, -7, np.int32), np.full(cap, -7, np.int32)
    val = np.full(cap, np.nan)
    gl._check(gl.load().godar_gpu_get_pairs(s._h, which, gl._ptr(pi, gl._ip), gl._ptr(pj, gl._ip), gl._ptr(val), cap,
                                            ctypes.byref(cnt)))
    return pi, pj, val, cnt.value


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [64, 1000, 8192, 8193, 20000])
def test_lists_are_sorted_and_cut_at_the_capacity(n, precision):
    f = gen.bonded_field(n=n, seed=3)
    s = gl.Stepper(f.params, n, precision)
    s.upload(f.x, f.y, f.r, f.h)
    s.set_field(f.forcing)
    s.step(1, 0, 2)
    for which in (gl.P_CANDIDATES, gl.P_CONTACTS, gl.P_BONDS):
        i, j, v = s.pairs(which)
        m = len(i)
        # few floes may have no contact yet
        assert (m > 0 or which == gl.P_CONTACTS) and np.all(i < j)
        key = i.astype(np.int64) * n + j
        assert np.all(key[1:] > key[:-1])
        if which == gl.P_CONTACTS:
            assert np.all(v > 0)
        for cap in (1, m // 2, m - 1, m, m + 9, 4 * m + 100):
            if cap <= 0:
                continue
            pi, pj, pv, total = _pairs(s, which, cap)
            k = min(cap, m)
            assert total == m
            assert np.array_equal(pi[:k], i[:k]) and np.array_equal(pj[:k], j[:k]) and np.array_equal(pv[:k], v[:k])
    # the contacts are the candidates that overlap
    ci, cj, cv = s.pairs(gl.P_CANDIDATES)
    ti, tj, tv = s.pairs(gl.P_CONTACTS)
    assert np.array_equal(ci[cv > 0], ti) and np.array_equal(cj[cv > 0], tj) and np.array_equal(cv[cv > 0], tv)
    every = s.download()[0]
    for name in gl.FLOE_FIELDS:
        assert np.array_equal(every[name], s.field(name)), name
    s.close()
