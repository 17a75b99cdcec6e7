"""The device memory that destroyed contexts leave for later ones: bounded,
given back on request, and given back to the library's own allocations when
the device has no other memory left."""
import pytest

from godar_b200 import generators as gen
from godar_b200 import lib as gl
from godar_b200.lib import Stepper
from godar_b200.params import PREC_MIXED

pytestmark = pytest.mark.gpu

N = 450000
MB = 1 << 20
KEPT, KEPT_BYTES = 4, 256 * MB


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _open(f, steps=2):
    s = Stepper(f.params, N, PREC_MIXED)
    s.upload(f.x, f.y, f.r, f.h)
    s.set_field(f.forcing)
    s.step(1, 0, steps)
    return s


@pytest.fixture(scope="module")
def field():
    f = gen.bonded_field(n=N, seed=6, device="gpu")
    _open(f).close()               # the device code is loaded
    gl.release_kept()
    return f


def test_what_is_kept_is_bounded_and_released(field):
    free0 = _free()
    alive = [_open(field) for _ in range(6)]
    used = free0 - _free()
    # pools that were not cut, or all six sets, would be beyond the bound
    assert min(used // 6, KEPT_BYTES * 6) > KEPT_BYTES and used * KEPT // 6 > KEPT * KEPT_BYTES + 512 * MB
    for s in alive:
        s.close()
    held = free0 - _free()
    assert 0 < held <= KEPT * KEPT_BYTES + 64 * MB
    gl.release_kept()
    assert free0 - _free() <= 64 * MB


def test_a_new_context_gets_what_others_left(field):
    import torch
    gl.release_kept()
    torch.cuda.empty_cache()
    free0 = _free()
    s = _open(field)
    need = free0 - _free()
    want = s.field("x").tobytes()
    s.close()
    assert need > 768 * MB
    alive = [_open(field) for _ in range(KEPT)]
    for s in alive:
        s.close()
    # too little for a set's own pool and the free memory, enough with the
    # pools of the other sets
    block = torch.empty(_free() - (need - 512 * MB), dtype=torch.uint8, device="cuda")
    try:
        s = _open(field)
        assert s.field("x").tobytes() == want
        s.close()
    finally:
        del block
        torch.cuda.empty_cache()
        gl.release_kept()
