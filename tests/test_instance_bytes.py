"""The estimate a batch admits its fields by counts the FP64 path's working
copies of the bonds (state, geometry, order: 92 bytes each) where they make the
difference, and is what it was for fields of the usual number of bonds."""
from godar_b200.lib import Batch

SETS = 2 * (4 + 80 + 48)          # a bond in the two sets: higher id, static, dynamic record


def test_usual_fields_are_admitted_as_before():
    for n in (1, 400, 65536, 2_000_000):
        for bonds in (0, n, 4 * n, 8 * n):
            assert Batch.instance_bytes(n, bonds) == n * (672 + 64 + 12 * 398 + 144) + bonds * (SETS + 8) + 4096


def test_bond_rich_fields_count_the_working_copies():
    n = 1000
    per = (Batch.instance_bytes(n, 40 * n) - Batch.instance_bytes(n, 20 * n)) / (20 * n)
    assert per == SETS + 48 + 40 + 4
    assert Batch.instance_bytes(n, 20 * n) > n * 5656 + 20 * n * (SETS + 8) + 4096
    # monotone where the rule changes
    b = [Batch.instance_bytes(n, k * n // 10) for k in range(200)]
    assert all(y > x for x, y in zip(b, b[1:]))
