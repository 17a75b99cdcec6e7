"""The arrays of a read-back are the caller's own, one by one: a caller that
keeps one field keeps no other one alive, except between the sizes at which
the fields together and one alone get huge pages."""
import pytest

from godar_b200 import generators as gen
from godar_b200.lib import FLOE_FIELDS, P_BONDS, SHARED, Stepper

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [256, 20000])
def test_every_field_owns_its_memory(n):
    f = gen.bonded_field(n=n, seed=1, device="gpu")
    s = Stepper(f.params, f.n)
    s.upload(f.x, f.y, f.r, f.h)
    s.set_field(f.forcing)
    s.step(1, 0, 1)
    for out in (s.floes(), s.floes(["x", "u"]), s.download()[0], s.download(which=P_BONDS)[0]):
        assert all(a.flags.owndata and a.base is None for a in out.values())
    assert set(s.floes()) == set(FLOE_FIELDS)
    s.close()


def test_fields_of_one_block_are_only_those_asked_for():
    f = gen.bonded_field(n=70000, seed=1, device="gpu")
    s = Stepper(f.params, f.n)
    s.upload(f.x, f.y, f.r, f.h)
    s.set_field(f.forcing)
    s.step(1, 0, 1)
    assert all(a.flags.owndata for a in s.floes(["x", "u", "tp"]).values())
    every = s.floes()
    assert every["x"].base.nbytes == len(FLOE_FIELDS) * f.n * 8 >= SHARED > f.n * 8
    for k in FLOE_FIELDS:
        assert every[k].tobytes() == s.field(k).tobytes(), k
    s.close()
