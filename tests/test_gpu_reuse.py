"""Contexts that come and go: a destroyed context's streams, events, pinned
memory and memory pool serve a later one, from any thread, with more contexts
alive than are kept, and every run equals a first one bit for bit; the device
memory held afterwards is bounded."""
import threading

import numpy as np
import pytest

from godar_b200 import generators as gen
from godar_b200.lib import P_BONDS, Stepper
from godar_b200.params import PREC_FP64, PREC_MIXED

pytestmark = pytest.mark.gpu


def _run(n, precision, steps):
    f = gen.bonded_field(n=n, seed=n)
    s = Stepper(f.params, n, precision)
    s.upload(f.x, f.y, f.r, f.h)
    s.set_field(f.forcing)
    for k in range(steps):
        s.step_async(k + 1)
    out = [s.download()[0][k] for k in ("x", "u", "omega", "fbx")] + list(s.pairs(P_BONDS))
    return s, [a.tobytes() for a in out]


def test_contexts_in_turn_and_at_once():
    import torch
    want = {}
    for n, p in ((300, PREC_FP64), (1500, PREC_MIXED), (9000, PREC_FP64)):
        s, want[n, p] = _run(n, p, 20)
        s.close()
    for _ in range(3):
        for (n, p), ref in want.items():
            s, got = _run(n, p, 20)
            s.close()
            assert got == ref, (n, p)
    # seven at once
    alive = []
    for k in range(7):
        (n, p), ref = list(want.items())[k % 3]
        s, got = _run(n, p, 20)
        assert got == ref
        alive.append(s)
    for s in alive:
        s.close()
    torch.cuda.synchronize()
    free0, _ = torch.cuda.mem_get_info()
    s, got = _run(60000, PREC_MIXED, 3)
    s.close()
    torch.cuda.synchronize()
    free1, _ = torch.cuda.mem_get_info()
    assert free0 - free1 <= 5 * (256 << 20)


def test_contexts_on_several_threads():
    ref = {}
    for n in (200, 700, 2500):
        s, ref[n] = _run(n, PREC_MIXED, 12)
        s.close()
    bad = []

    def work(n):
        for _ in range(6):
            s, got = _run(n, PREC_MIXED, 12)
            s.close()
            if got != ref[n]:
                bad.append(n)

    ts = [threading.Thread(target=work, args=(n,)) for n in (200, 700, 2500, 200, 700, 2500)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
