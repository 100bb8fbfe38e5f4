"""Gather slots sorted by the cell they read (fdtd_slot_order): every sampled
slot once, in the row and 16-column block of its cell, and the others after
them."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from beamz_b200 import abi  # noqa: E402
from beamz_b200 import plan as P  # noqa: E402
from beamz_b200 import runtime as R  # noqa: E402

pytestmark = pytest.mark.gpu


def _sorted(idx, w, masks, comps, shapes, lattice):
    dev = lambda a: None if a is None else torch.as_tensor(a, device="cuda")  # noqa: E731
    stream = R.ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    order, first = R._slots_by_cell(abi.load_library(), stream, dev(idx), dev(w), dev(masks), comps, shapes, lattice)
    return order.cpu().numpy(), first.cpu().numpy()


# Grids whose blocks fit one round of the scan, fill it exactly, and take several.
@pytest.mark.parametrize("seed,grid", [(0, (1, 1)), (1, (5, 7)), (2, (31, 40)), (3, (12, 69)), (4, (90, 130)), (5, (1023, 127)),
                                       (6, (400, 401)), (7, (63, 5))])
def test_slots_lie_in_their_blocks(seed, grid):
    rng = np.random.default_rng(seed)
    Y, X = grid
    pol = ("tm", "te")[seed % 2]
    names = P.active_components(2, pol)
    comps = [P.COMPONENT_INDEX[c] for c in names]
    shapes = [P.component_shape(c, grid, pol) for c in names]
    M, K, n = int(rng.integers(1, 4)), int(rng.integers(1, 4)), int(rng.integers(1, 600))
    idx = rng.integers(-3, Y * X + 5, (M, 6, K, n)).astype(np.int32)
    w = (rng.random((M, 6, K, n)) < 0.7).astype(np.float32)
    masks = (rng.random((M, 6)) < 0.7).astype(np.float32)
    order, first = _sorted(idx, w, masks, comps, shapes, (Y + 1, X + 1))
    blocks = -(-(X + 1) // 16)
    assert order.size == M * 3 * K * n and first.size == 3 * (Y + 1) * blocks + 1
    assert first[0] == 0 and np.all(np.diff(first) >= 0)
    m, c, k, p = np.unravel_index(order, idx.shape)
    live = np.arange(order.size) < first[-1]
    a = np.searchsorted(comps, c)
    y, x = np.divmod(idx.reshape(-1)[order], np.array([s[1] for s in shapes])[a])
    at = (a * (Y + 1) + y) * blocks + x // 16
    np.testing.assert_array_equal(at[live], np.searchsorted(first, np.flatnonzero(live), side="right") - 1)
    sampled = np.cumprod(w != 0, axis=2)[m, c, k, p] & (masks[m, c] != 0)
    sampled &= (idx.reshape(-1)[order] >= 0) & (idx.reshape(-1)[order] < np.array([s[0] * s[1] for s in shapes])[a])
    np.testing.assert_array_equal(sampled.astype(bool), live)
    assert np.unique(order).size == order.size and np.all(np.isin(c, comps))


def test_recorder_values_without_a_cell_come_last():
    idx = np.array([99, -1, 3, 17, 100, 40, 3], np.int32).reshape(1, 1, 1, -1)
    w = np.array([1.0, 1.0, 2.0, 0.0, 1.0, -1.0, 0.5], np.float32).reshape(1, 1, 1, -1)
    order, first = _sorted(idx, w, None, [0], [(5, 20)], (6, 21))
    assert sorted(order[: first[-1]]) == [0, 2, 5, 6] and sorted(order[first[-1]:]) == [1, 3, 4]


def test_slot_tables_of_other_sizes_are_refused():
    idx, w = np.zeros((1, 6, 1, 4), np.int32), np.ones((1, 6, 1, 4), np.float32)
    with pytest.raises(abi.FdtdError):
        _sorted(idx, w, None, [2, 3, 4], [(9, 9)] * 3, (8, 9))  # taller than the lattice
    with pytest.raises(abi.FdtdError):
        _sorted(idx, w, None, [2, 3, 6], [(8, 9)] * 3, (8, 9))
    with pytest.raises(abi.FdtdError):
        _sorted(idx, w[..., :3].copy(), None, [2, 3, 4], [(8, 9)] * 3, (8, 9))
