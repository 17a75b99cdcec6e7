"""Diagnostics that no step has computed yet read as zero, whatever a context
destroyed before left in the memory that the new one reuses."""
import numpy as np
import pytest

from godar_b200 import generators as gen
from godar_b200.lib import FLOE_FIELDS, Stepper
from godar_b200.params import PREC_FP64, PREC_MIXED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_diagnostics_before_the_first_diagnostic_step(precision):
    f = gen.bonded_field(n=2000, seed=3)
    diag = FLOE_FIELDS[8:]
    for on in (True, False):
        s = Stepper(f.params, f.n, precision)
        s.upload(f.x, f.y, f.r, f.h)
        s.set_field(f.forcing)
        s.set_diagnostics(on)
        s.step(1, 0, 3)
        out = s.floes(diag)
        assert all(np.any(out[k] != 0.0) == on for k in diag if on is False or k in ("tfx", "fbx", "tp")), on
        s.close()
