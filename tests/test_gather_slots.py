"""Gather slots sorted by the cell they read (FdtdDft.slot_order): every sampled
slot once, in the row and 16-column block of its cell, and no other."""

from __future__ import annotations

import types

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from beamz_b200 import plan as P  # noqa: E402
from beamz_b200 import runtime as R  # noqa: E402


@pytest.mark.parametrize("seed", range(8))
def test_dft_slots_lie_in_their_blocks(seed):
    rng = np.random.default_rng(seed)
    Y, X = int(rng.integers(1, 40)), int(rng.integers(1, 70))
    pol = ("tm", "te")[seed % 2]
    shapes = [P.component_shape(c, (Y, X), pol) for c in P.COMPONENTS]
    comps = [P.COMPONENT_INDEX[c] for c in P.active_components(2, pol)]
    M, K, n = (int(v) for v in rng.integers(1, (4, 4, 60)))
    weights = (rng.random((M, 6, K, n)) < 0.7).astype(np.float32)
    for m in range(M):  # a packed plan holds zeros beyond a monitor's own points
        weights[m, :, :, int(rng.integers(0, n + 1)):] = 0.0
    arena = types.SimpleNamespace(
        indices=torch.as_tensor(rng.integers(-3, Y * X + 5, (M, 6, K, n)).astype(np.int32)),
        weights=torch.as_tensor(weights), masks=torch.as_tensor((rng.random((M, 6)) < 0.7).astype(np.float32)))
    order, first = R._dft_slots(arena, comps, shapes, (Y + 1, X + 1))
    blocks = -(-(X + 1) // 16)
    assert order.dtype == first.dtype == torch.int32 and first.numel() == 3 * (Y + 1) * blocks + 1
    got = []
    for a, c in enumerate(comps):
        for j in range(Y + 1):
            for b in range(blocks):
                at = (a * (Y + 1) + j) * blocks + b
                for e in range(int(first[at]), int(first[at + 1])):
                    m, cc, k, p = np.unravel_index(int(order[e]), (M, 6, K, n))
                    y, x = divmod(int(arena.indices[m, cc, k, p]), shapes[c][1])
                    assert (cc, y, x // 16) == (c, j, b)
                    got.append((m, cc, k, p))
    want = set()
    for m, c, p in np.ndindex(M, 6, n):
        if c not in comps or arena.masks[m, c] == 0:
            continue
        for k in range(K):
            if arena.weights[m, c, k, p] == 0:
                break
            if 0 <= int(arena.indices[m, c, k, p]) < int(np.prod(shapes[c])):
                want.add((m, c, k, p))
    assert len(got) == len(set(got)) and set(got) == want


def test_recorder_values_without_a_cell_come_last():
    shape = (5, 20)
    idx = torch.tensor([[99, -1, 3, 17, 100, 40, 3]], dtype=torch.int32)
    w = torch.tensor([[1.0, 1.0, 2.0, 0.0, 1.0, -1.0, 0.5]])
    order, first = R._recorder_slots(idx, w, shape, (6, 21))
    live = int(first[-1])
    assert sorted(order[:live].tolist()) == [0, 2, 5, 6] and sorted(order[live:].tolist()) == [1, 3, 4]


def test_slot_samples_are_bounded():
    assert R.slot_samples_fit(1, 1, 1_000_000) and not R.slot_samples_fit(1, 1, 4_000_000)
    assert R.slot_samples_fit(1, 4, 40_000) and not R.slot_samples_fit(1, 4, 160_000)
    assert not R.slot_samples_fit(1, 1, 10, batch=1)
