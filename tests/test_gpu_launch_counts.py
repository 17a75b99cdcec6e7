"""The count of step kernels in godar_batch_phase_stats: every kernel a step
launches, whether the batch runs merged steps (one launch a chunk, or two to
five a step) or the separate kernels (four, FP64 three of sheltering fields;
mixed one more on diagnostic steps)."""
import pytest

from godar_b200 import generators as gen
from godar_b200.lib import Batch
from godar_b200.params import PREC_FP64, PREC_MIXED

pytestmark = pytest.mark.gpu


def _launched(f, precision, calls, monkeypatch, fused="1"):
    """Kernels of each of `calls`: (steps, diagnostics, queued)."""
    monkeypatch.setenv("GODAR_FUSED", fused)
    monkeypatch.setenv("GODAR_TUNE", "0")
    b = Batch(precision)
    b.add_field(f)
    b.step(1)
    out = []
    for steps, diag, queued in calls:
        b.set_diagnostics(diag)
        s0 = b.stats()
        (b.step_async if queued else b.step)(steps)
        s1 = b.stats()
        assert s1["launches"] - s0["launches"] == steps and s1["rebuilds"] == s0["rebuilds"]
        out.append(s1["kernel_launches"] - s0["kernel_launches"])
    b.close()
    return out


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_merged_steps(precision, monkeypatch):
    # one block: a launch for each of the chunks of a call (the chunks' lengths double: 1, 2, 4 ..)
    one = _launched(gen.bonded_field(n=64, seed=1), precision, [(1, False, False), (1, True, True), (16, False, False)],
                    monkeypatch)
    assert one[:2] == [1, 1] and 1 <= one[2] < 16
    # two launches a step, with diagnostics too
    calls = [(1, False, False), (6, False, False), (6, True, False), (5, False, True)]
    assert _launched(gen.bonded_field(n=5000, seed=2), precision, calls, monkeypatch) == [2, 12, 12, 10]


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_merged_steps_of_sheltering_fields(precision, monkeypatch):
    # sums in a kernel of their own beyond 9,472 floes on plain steps; mixed,
    # the bonds of a field with ridging follow the pairs in their own kernel
    f = gen.polydisperse_field(n=12000, seed=2, phi=0.6, dt=1e-3)
    bonds = 1 if precision == PREC_MIXED and f.params.cohesion and f.params.ridging else 0
    got = _launched(f, precision, [(4, False, False), (4, True, False)], monkeypatch)
    assert got == [4 * (3 + bonds), 3 * (3 + bonds) + 2 + bonds]


def test_diagnostic_steps_of_larger_merged_batches(monkeypatch):
    # beyond 32,768 floes with enough candidates a diagnostic step's sums have a
    # kernel of their own, FP64 behind two kernels of pairs
    calls = [(4, False, False), (4, True, False)]
    for n, diag in ((32768, 2), (32769, 4)):
        f = gen.bonded_field(n=n, seed=2, device="gpu")
        assert _launched(f, PREC_FP64, calls, monkeypatch) == [8, 6 + diag]
        assert _launched(f, PREC_MIXED, calls, monkeypatch) == [8, 8]


def test_separate_kernels(monkeypatch):
    calls = [(4, False, False), (4, True, False)]
    bonded = gen.bonded_field(n=3000, seed=2)
    assert _launched(bonded, PREC_FP64, calls, monkeypatch, "0") == [16, 16]
    assert _launched(bonded, PREC_MIXED, calls, monkeypatch, "0") == [16, 17]
    poly = gen.polydisperse_field(n=3000, seed=2, phi=0.6, dt=1e-3)
    assert _launched(poly, PREC_FP64, calls, monkeypatch, "0") == [12, 12]
