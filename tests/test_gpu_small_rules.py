"""The rules that choose a small batch's form, on either side of each line:
one block or a cluster, the diagnostic step with its chunk or apart from it, the
floes' sums by groups of lanes or by a thread each.  Every form gives the
separate kernels' bits."""
import numpy as np
import pytest

from godar_b200 import generators as gen
from godar_b200.params import BC_OPEN_BOTTOM, BC_OPEN_LEFT, BC_OPEN_RIGHT, BC_OPEN_TOP, PREC_FP64, PREC_MIXED, make_params

from .test_gpu_long_rows import _packed, _ring
from .test_gpu_merged import _same

pytestmark = pytest.mark.gpu

OPEN = BC_OPEN_LEFT | BC_OPEN_RIGHT | BC_OPEN_BOTTOM | BC_OPEN_TOP


def _free(n, rtree=200.0, sp=400.0, **kw):
    """Floes on a jittered grid, out of touch."""
    rng = np.random.default_rng(n)
    m = int(np.ceil(np.sqrt(n)))
    at = rng.permutation(m * m)[:n]
    x = (at % m + 0.5) * sp + rng.uniform(-9.0, 9.0, n)
    y = (at // m + 0.5) * sp + rng.uniform(-9.0, 9.0, n)
    p = make_params(m * sp, m * sp, **{**dict(cohesion=0, shelter=0, ridging=0, dt=1e-2, rtree=rtree, ua=9.0, va=-4.0,
                                              boundary=OPEN), **kw})
    return gen.Field("free", p, x, y, rng.uniform(15.0, 20.0, n), rng.uniform(0.5, 2.0, n), 10,
                     u=rng.uniform(-1.0, 1.0, n), v=rng.uniform(-1.0, 1.0, n))


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 512, 513, 1024, 1025])
def test_one_block_of_free_floes(n, precision, monkeypatch):
    _same(_free(n), precision, monkeypatch)


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [200, 215, 230, 256, 257, 285])
def test_one_block_of_bonded_floes(n, precision, monkeypatch):
    _same(gen.bonded_field(n=n, seed=1), precision, monkeypatch)


# every floe a candidate of every other: 990 and 1,035 entries for a block's
# four rounds, and far more than a cluster's
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [45, 46, 130, 300, 600])
def test_diagnostic_steps_of_many_candidates(n, precision, monkeypatch):
    _same(_free(n, rtree=50000.0, sp=60.0, cohesion=1, bond_lim_rel=0.7, dt=1e-3), precision, monkeypatch)


# pairs in touch for fewer and for more than a quarter of the floes
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,pairs", [(4200, 0), (4200, 1), (5000, 1240), (5000, 1260), (9472, 40), (9473, 40)])
def test_sums_of_few_pairs(n, pairs, precision, monkeypatch):
    f = _free(n, rtree=60.0, cohesion=1, bond_lim=2.0, dt=1e-3)
    # the last floes join earlier ones, near enough for a bond
    for k in range(pairs):
        i, j = k, n - 1 - k
        a = 0.7 * k
        f.x[j] = f.x[i] + np.cos(a) * (f.r[i] + f.r[j] + 0.5)
        f.y[j] = f.y[i] + np.sin(a) * (f.r[i] + f.r[j] + 0.5)
    _same(f, precision, monkeypatch)


# rows of hundreds of entries of which few, or all, add to a floe's sums
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("shelter", [0, 1])
def test_sums_along_long_rows(shelter, precision, monkeypatch):
    fields = [_packed(300), _ring(200, 0), _ring(200, 100), _ring(1500, 700)]
    # one small floe in five touches the large one
    k = fields[3]
    big = int(np.argmax(k.r))
    dx, dy = k.x - k.x[big], k.y - k.y[big]
    d = np.hypot(dx, dy)
    d[big] = 1.0
    to = np.where(np.arange(k.n) % 5 == 0, k.r[big] + k.r - 0.01, d)
    to[big] = 0.0
    k.x, k.y = k.x[big] + dx / d * to, k.y[big] + dy / d * to
    for f in fields:
        f.params.shelter = f.params.ridging = shelter
        _same(f, precision, monkeypatch)


# diagnostic steps with the sums in the update's kernel and apart
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [32768, 32769])
@pytest.mark.parametrize("kind", ["bonded", "poly", "walls"])
def test_diagnostic_sums(kind, n, precision, monkeypatch):
    if kind == "poly":
        f = gen.polydisperse_field(n=n, seed=2, phi=0.6, dt=1e-3)
    else:
        f = gen.bonded_field(n=n, seed=2, device="gpu")
        f.params.ridging = 1
        if kind == "walls":
            f.params.boundary = 0
    _same(f, precision, monkeypatch)


# FP64: by the entries too, 327,680 of them beyond 8,192 floes
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,rtree", [(8192, 360.0), (8300, 300.0), (8300, 360.0)])
def test_diagnostic_sums_of_many_entries(n, rtree, precision, monkeypatch):
    _same(_free(n, rtree=rtree, sp=60.0, cohesion=1, bond_lim_rel=0.7, dt=1e-3), precision, monkeypatch)


# one block, FP64: 128 floes keep a diagnostic step of all pairs, 129 do not
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [128, 129])
def test_diagnostic_steps_on_one_block(n, precision, monkeypatch):
    _same(_free(n, rtree=50000.0, sp=60.0, dt=1e-3), precision, monkeypatch)


# mixed: a large floe whose row is far longer than the others', and none
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("large", [0, 1])
def test_diagnostic_sums_of_one_long_row(large, precision, monkeypatch):
    n = 33000
    f = _free(n, rtree=100.0, sp=60.0, cohesion=1, bond_lim_rel=0.7, dt=1e-3)
    if large:
        f.params.nx += 5000.0
        f.x[17], f.y[17], f.r[17] = f.x.max() + 2040.0, 0.5 * f.y.max(), 2000.0
    _same(f, precision, monkeypatch)
