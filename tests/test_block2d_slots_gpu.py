"""Several 2D steps per launch with more gather slots than a tile's list holds:
whole-plane monitors of one and of three slots per point and recorders of
shuffled lists, bit for bit against the phase schedule; and the time of such a
program against its samples taken one step at a time."""

from __future__ import annotations

import dataclasses
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from beamz_b200 import plan as P  # noqa: E402
from beamz_b200 import runtime as R  # noqa: E402
from tests.scenarios import random_initial_fields, scenario_2d  # noqa: E402

pytestmark = pytest.mark.gpu


def _plane_monitor(grid, pol, slots, seed=0, nfreq=2):
    """Every cell of every active component (the last point repeated for the
    smaller ones), `slots` cells per point, some of zero weight."""
    rng = np.random.default_rng(seed)
    act = P.active_components(2, pol)
    n = (grid[0] + 1) * (grid[1] + 1)
    idx, w = [], []
    for c in P.COMPONENTS:
        size = int(np.prod(P.component_shape(c, grid, pol)))
        idx.append(np.minimum(np.arange(n)[:, None] + np.arange(slots) * 7, size - 1).astype(np.int32))
        weight = rng.standard_normal((n, slots)).astype(np.float32)
        w.append(weight if slots == 1 else weight * (rng.random((n, slots)) < 0.7))
    mask = np.array([1.0 if c in act else 0.0 for c in P.COMPONENTS], np.float32)
    freqs = np.linspace(0.9, 1.1, nfreq).astype(np.float32) * np.float32(P.LIGHT_SPEED / 1.55e-6)
    return P.DftMonitorPlan(freqs, idx, [np.asarray(v, np.float32) for v in w], mask)


def _list_recorder(grid, pol, interval, n, seed=1):
    """Four fifths of the cells of every active component in shuffled order, an
    eighth of them with weight zero."""
    rng = np.random.default_rng(seed)
    act = P.active_components(2, pol)
    sizes = [int(np.prod(P.component_shape(c, grid, pol))) for c in act]
    flat = [rng.permutation(s)[: max(1, 4 * s // 5)].astype(np.int32)[:, None] for s in sizes]
    w = [np.where(rng.random(f.shape) < 0.125, 0.0, 1.25).astype(np.float32) for f in flat]
    return P.RecorderPlan(tuple(act), interval, n, flat, w, shapes=tuple((f.size,) for f in flat), signs=(1.0, -1.0, 1.0))


@pytest.mark.parametrize("grid,pol,slots,steps,record", [
    ((20, 30), "tm", 1, 9, True),       # one tile
    ((20, 30), "te", 3, 8, True),
    ((90, 130), "tm", 3, 11, True),     # lists that overflow in most tiles
    ((97, 111), "te", 1, 7, True),
    ((330, 340), "tm", 1, 10, False),   # tiles of more than 32 rows
    ((700, 500), "te", 1, 8, False),    # more than one wave
])
def test_full_lists_match_the_phase_schedule(grid, pol, slots, steps, record):
    spec = scenario_2d(grid=grid, polarization=pol, seed=steps, pml_cells=4, nsteps=40, metallic=("left",))
    spec = dataclasses.replace(spec, monitors=[*spec.monitors, _plane_monitor(grid, pol, slots)])
    if record:
        spec = dataclasses.replace(spec, recorders=[_list_recorder(grid, pol, 1, 12), _list_recorder(grid, pol, 3, 2, 4)])
    fields = random_initial_fields(spec, seed=2)
    got = []
    for schedule in ("fused", "phases"):
        prog = R.compile_program(spec, schedule=schedule)
        assert prog.slot_samples == (schedule == "fused")
        st = R.initial_state(prog, fields=fields)
        R.run_steps(st, prog, steps)
        R.run_steps(st, prog, 4)
        got.append((st.numpy(), [R.recorded(st, prog, r) for r in range(len(spec.recorders))]))
    (a, ra), (b, rb) = got
    for c in P.active_components(2, pol):
        np.testing.assert_array_equal(a[c], b[c], err_msg=c)
    for k in ("dft_re", "dft_im", "dft_w"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    for x, y in zip(ra, rb):
        assert x.keys() == y.keys()
        for k in x:
            np.testing.assert_array_equal(x[k], y[k], err_msg=k)


def test_samples_beyond_the_buffer_step_one_by_one():
    """Too many slot values to buffer: interpolated samples, single steps, the
    same bits."""
    grid = (300, 310)
    spec = scenario_2d(grid=grid, seed=3, pml_cells=4, nsteps=40)
    spec = dataclasses.replace(spec, monitors=[_plane_monitor(grid, "tm", 4)])
    fields = random_initial_fields(spec, seed=2)
    progs = [R.compile_program(spec, schedule=s) for s in ("fused", "phases")]
    assert not progs[0].slot_samples
    out = [R.run_steps(R.run_steps(R.initial_state(p, fields=fields), p, 5), p, 4).numpy() for p in progs]
    for k in ("Ez", "Hx", "Hy", "dft_re", "dft_im", "dft_w"):
        np.testing.assert_array_equal(out[0][k], out[1][k], err_msg=k)
    for k in ("psi_h", "psi_e"):
        for x, y in zip(out[0][k], out[1][k]):
            np.testing.assert_array_equal(x, y, err_msg=k)


def test_a_whole_plane_monitor_is_no_slower_than_single_steps():
    """A tile looks at its own slots only.  Looking through all of them took ten
    times the single steps' time here; twice is the bound, for noise."""
    grid = (400, 400)
    spec = scenario_2d(grid=grid, seed=3, pml_cells=8, nsteps=200)
    spec = dataclasses.replace(spec, monitors=[_plane_monitor(grid, "tm", 1)])
    best = []
    for batch in (16, 1):  # batch 1: one launch per step and sample
        prog = R.compile_program(spec, dft_batch=batch)
        st = R.initial_state(prog, fields=random_initial_fields(spec, seed=2))
        times = []
        for _ in range(4):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            R.run_steps(st, prog, 48)
            torch.cuda.synchronize()
            times.append(time.perf_counter() - t0)
        best.append(min(times))
    assert best[0] <= 2.0 * best[1], best


def test_slot_tables_of_other_sizes_are_rejected():
    spec = scenario_2d(grid=(20, 30), nsteps=4)
    prog = R.compile_program(spec)
    st = R.initial_state(prog)
    import ctypes

    s = prog.fill(st, 1)
    assert prog.lib.fdtd_validate(ctypes.byref(s)) == 0
    s.dft.slot_first.dims[0] -= 1
    assert prog.lib.fdtd_validate(ctypes.byref(s)) == 1
    s = prog.fill(st, 1)
    s.dft.slot_order.data = None
    assert prog.lib.fdtd_validate(ctypes.byref(s)) == 1
