"""Sheltering and other fields in one batch, over the sizes at which the floes'
sums change kernels (one wave of groups of lanes, a kernel of their own, the
separate kernels of larger batches): every field as when it steps alone, bit
for bit."""
import pytest

from godar_b200 import generators as gen
from godar_b200.lib import Batch
from godar_b200.params import PREC_FP64, PREC_MIXED

pytestmark = pytest.mark.gpu

NAMES = ("x", "y", "u", "v", "omega", "r", "h", "tfx", "fcx", "fbx")


def _run(fields, precision):
    b = Batch(precision)
    hs = [b.add_field(f) for f in fields]
    b.step(2)
    b.set_diagnostics(False)
    b.step(9)
    for _ in range(4):
        b.step_async(1)
    b.set_diagnostics(True)
    b.step(2)
    out = [[b.field(k, q).tobytes() for q in NAMES] for k in hs]
    b.close()
    return out


@pytest.mark.parametrize("fused", ["1", "0"])
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [300, 6600, 9000])
def test_each_field_as_alone(n, precision, fused, monkeypatch):
    fields = [gen.bonded_field(n=700, seed=1), gen.polydisperse_field(n=n, seed=2, phi=0.6, dt=1e-3),
              gen.bonded_field(n=1801, seed=3), gen.polydisperse_field(n=310, seed=4, phi=0.6, dt=1e-3)]
    alone = [_run([f], precision)[0] for f in fields]
    monkeypatch.setenv("GODAR_FUSED", fused)
    for k, (a, b) in enumerate(zip(alone, _run(fields, precision))):
        assert a == b, k
