"""A batch whose fields have more than 2^30 cells together: sparse fields in
wide domains have the most cells a field can have (4,096 by 4,096), and the
scan over the batch's cells indexes past half the range of an int."""
import numpy as np
import pytest

from godar_b200.lib import Batch
from godar_b200.params import BC_PERIODIC_X, BC_PERIODIC_Y, PREC_FP64, PREC_MIXED, make_params

pytestmark = pytest.mark.gpu

L = 42000.0
FIELDS = 65                       # 65 * 4096^2 cells: 1.09e9, 8.7 GB of cell lists


def _field(k):
    """A pair in contact and two floes apart, at the ends of the domain."""
    p = make_params(L, L, cohesion=1, shelter=0, ridging=0, dt=1e-3, rtree=9.0, ua=4.0 + k, va=3.0,
                    boundary=BC_PERIODIC_X | BC_PERIODIC_Y)
    x = np.array([20.0, 39.9, L - 5.0, L - 500.0])
    y = np.array([L - 20.0, L - 20.0, 7.0, 0.5 * L + k])
    return p, x, y, np.full(4, 10.0), np.full(4, 1.0 + 0.01 * k)


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_batch_of_sparse_fields(precision):
    b = Batch(precision)
    ids = [b.add(*_field(k)) for k in range(FIELDS)]
    b.step(3)
    for k in (0, 1, FIELDS // 2, FIELDS - 1):
        one = Batch(precision)
        i = one.add(*_field(k))
        one.step(3)
        for name in ("x", "y", "u", "v", "omega"):
            assert b.field(ids[k], name).tobytes() == one.field(i, name).tobytes(), (k, name)
        one.close()
    b.close()
