"""The clock of a wall over the steps of a fused run: one addition a step, in bounded memory.  No GPU."""

import tracemalloc

import pytest


@pytest.mark.parametrize("steps", [0, 1, 65535, 65536, 65537, 300_000])
def test_one_addition_a_step(steps):
    from taichimps_gb300 import FixWallGran
    f = FixWallGran.__new__(FixWallGran)
    f.elapsed = want = 0.125
    f.passed(steps, 1e-4)
    for _ in range(steps):
        want += 1e-4
    assert f.elapsed == want


def test_memory_of_a_long_run():
    from taichimps_gb300 import FixWallGran
    f = FixWallGran.__new__(FixWallGran)
    f.elapsed = 0.0
    tracemalloc.start()
    f.passed(5_000_000, 1e-4)
    peak = tracemalloc.get_traced_memory()[1]
    tracemalloc.stop()
    assert peak < 4_000_000, peak
