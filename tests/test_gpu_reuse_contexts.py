"""Fields stepped in two CUDA contexts of one process by turns: what destroyed
ones leave for later ones stays with its context, and nothing of it is lost."""
import ctypes

import numpy as np
import pytest

from godar_b200 import generators as gen
from godar_b200.lib import Stepper
from godar_b200.params import PREC_MIXED

pytestmark = pytest.mark.gpu

N = 60000


@pytest.fixture
def second_context():
    """A second context on the first device, made current by push()."""
    import torch
    torch.cuda.init()
    torch.zeros(1, device="cuda")           # the primary context exists and is current
    cu = ctypes.CDLL("libcuda.so.1")
    ctx = ctypes.c_void_p()
    assert cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, 0) == 0

    class Second:
        def __enter__(self):
            assert cu.cuCtxPushCurrent_v2(ctx) == 0

        def __exit__(self, *_):
            assert cu.cuCtxPopCurrent_v2(ctypes.byref(ctypes.c_void_p())) == 0

    assert cu.cuCtxPopCurrent_v2(ctypes.byref(ctypes.c_void_p())) == 0
    yield Second()
    assert cu.cuCtxDestroy_v2(ctx) == 0


def _run(f):
    s = Stepper(f.params, N, PREC_MIXED)
    s.upload(f.x, f.y, f.r, f.h)
    s.set_field(f.forcing)
    s.step(1, 0, 3)
    out = s.field("x").tobytes()
    s.close()
    return out


def test_two_contexts_by_turns(second_context):
    import torch
    f = gen.bonded_field(n=N, seed=5, device="gpu")
    want = _run(f)
    with second_context:
        assert _run(f) == want
    torch.cuda.synchronize()
    free0, _ = torch.cuda.mem_get_info()
    # a set left behind at every turn would be some 100 MB and more each
    for _ in range(6):
        assert _run(f) == want
        with second_context:
            assert _run(f) == want
    torch.cuda.synchronize()
    free1, _ = torch.cuda.mem_get_info()
    assert free0 - free1 <= 64 << 20
