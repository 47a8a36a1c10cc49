"""Tile widths that run as the same kernel are timed once (no GPU)."""
from unbiased_differentiable_splatting_gb300 import autotune


def test_widths_that_run_as_eight():
    calls = []

    def timer(tx, spread, leaf):  # every call a little faster than the one before
        calls.append((tx, spread, leaf))
        return 10.0 - 0.01 * len(calls) + (5.0 if tx == 4 else 0.0)

    best, times = autotune._sweep(autotune.once_per_kernel(timer), autotune.CANDIDATES, autotune.SPREADS, None)
    assert sorted(calls) == [(4, 0, 0), (4, 1, 0), (8, 0, 0), (8, 1, 0)]
    assert best["tile_x"] == 8 and times["8/1"] == times["16/1"] == times["32/1"]
