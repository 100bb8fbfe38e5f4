"""How many gather slot values a 2D program buffers."""

from __future__ import annotations

from beamz_b200 import runtime as R


def test_slot_samples_are_bounded():
    assert R.slot_samples_fit(1, 1, 1_000_000) and not R.slot_samples_fit(1, 1, 4_000_000)
    assert R.slot_samples_fit(1, 4, 40_000) and not R.slot_samples_fit(1, 4, 160_000)
    assert not R.slot_samples_fit(1, 1, 10, batch=1)
