"""Several 2D steps per launch (csrc/block2d.cu) against the phase schedule,
which advances one half step per kernel: every bit of the fields, CPML
memories, DFT arena and records, at the edges of the tiling (own columns 48 at
eight steps per launch), odd step counts and every kind of input."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from beamz_b200 import plan as P  # noqa: E402
from beamz_b200 import runtime as R  # noqa: E402
from tests.scenarios import random_initial_fields, scenario_2d, with_metrics  # noqa: E402

pytestmark = pytest.mark.gpu


def _rich(grid, pol, pml, seed, metallic=(), metric=None, conductive=False, recorders=True, cpml=True):
    """A scene with sources at every timing, monitors of one and of several
    gather slots, and recorders of single cells and of whole components."""
    rng = np.random.default_rng(seed)
    n = 40
    spec = scenario_2d(grid=grid, polarization=pol, seed=seed, pml_cells=pml, metallic=metallic, nsteps=n, cpml=cpml)
    act = P.active_components(2, pol)
    shapes = {c: P.component_shape(c, grid, pol) for c in P.COMPONENTS}
    ecomp = "Ez" if pol == "tm" else "Ex"
    sy, sx = shapes[ecomp]
    wave = (rng.standard_normal(n) * 1e-2).astype(np.float32)
    line = rng.standard_normal((sy, 1)).astype(np.float32)
    srcs = [*spec.sources, P.SourcePlan(ecomp, "e", (0, sx // 2), line, wave),
            P.SourcePlan(ecomp, "pre_e", (sy // 2, 0), rng.standard_normal((1, sx)).astype(np.float32), wave)]
    # A monitor of up to three slots per point anywhere on the grid, zero weights among them.
    idx, w = [], []
    for c in P.COMPONENTS:
        size = int(np.prod(shapes[c]))
        idx.append(rng.integers(0, size, (37, 3)).astype(np.int32))
        w.append((rng.standard_normal((37, 3)) * (rng.random((37, 3)) < 0.7)).astype(np.float32))
    mask = np.array([1.0 if c in act else 0.0 for c in P.COMPONENTS], np.float32)
    mons = [*spec.monitors, P.DftMonitorPlan(spec.monitors[0].freqs[:2], idx, w, mask, window_code=1, t_start=2 * spec.dt,
                                             t_end=30 * spec.dt, interval=2)]
    spec = dataclasses.replace(spec, sources=srcs, monitors=mons)
    if recorders:
        flat = [rng.integers(0, int(np.prod(shapes[c])), (50, 1)).astype(np.int32) for c in act]
        ones = [np.where(np.arange(50) % 7 == 3, 0.0, 1.5).astype(np.float32)[:, None] for _ in act]
        spec = dataclasses.replace(spec, recorders=[
            P.RecorderPlan(tuple(act), 3, 9, flat, ones, shapes=((50,),) * 3, signs=(1.0, -1.0, 1.0)),
            P.domain_recorder(grid, act[:2], interval=2, num_steps=n, polarization=pol), _box_recorder(shapes[act[1]], act[1], n)])
    if conductive:
        eps = np.full(grid, 2.085, np.float32)
        eps[grid[0] // 3:] = 12.11
        e_site, h_site, e_eps = P.lossy_site_coefficients_2d(eps, np.where(eps > 3, np.float32(4e4), np.float32(0)),
                                                             spec.dt, pol)
        spec = dataclasses.replace(spec, e_site=e_site, h_site=h_site, e_site_eps=e_eps)
    return with_metrics(spec, metric, seed=seed) if metric else spec


def _box_recorder(shape, comp, n):
    """Every step of a box of one component (the form the adjoint records)."""
    y0, x0 = shape[0] // 4, shape[1] // 5
    ny, nx = max(1, shape[0] // 2), max(1, shape[1] // 2)
    flat = ((y0 + np.arange(ny))[:, None] * shape[1] + x0 + np.arange(nx)[None, :]).reshape(-1, 1).astype(np.int32)
    return P.RecorderPlan((comp,), 1, n, [flat], [np.ones(flat.shape, np.float32)], shapes=((ny, nx),), signs=(-1.0,))


CASES = [
    ((5, 7), "tm", 1, 1, {}), ((13, 15), "te", 3, 7, {}), ((47, 95), "tm", 6, 8, {}),
    ((48, 96), "te", 9, 9, dict(metallic=("left", "top"))), ((130, 49), "tm", 20, 16, dict(metallic=("right", "bottom"))),
    ((9, 200), "te", 4, 17, dict(conductive=True)), ((200, 31), "tm", 5, 23, dict(conductive=True, metallic=("left",))),
    ((61, 143), "tm", 8, 24, dict(metric="rectilinear")), ((143, 61), "te", 8, 33, dict(metric="axis_uniform")),
    ((70, 50), "tm", 0, 15, dict(cpml=False, metallic=("left", "right"))), ((64, 64), "te", 32, 18, {}),
    ((700, 400), "tm", 12, 11, dict(recorders=False)), ((1200, 900), "te", 10, 10, dict(recorders=False)),
]


@pytest.mark.parametrize("grid,pol,pml,steps,options", CASES)
def test_blocked_steps_match_the_phase_schedule(grid, pol, pml, steps, options):
    spec = _rich(grid, pol, pml, seed=steps, **options)
    fields = random_initial_fields(spec, seed=3)
    got = []
    for schedule in ("fused", "phases"):
        prog = R.compile_program(spec, schedule=schedule)
        st = R.initial_state(prog, fields=fields)
        R.run_steps(st, prog, steps)
        R.run_steps(st, prog, 5)  # from the bank where the first call ended
        got.append((st.numpy(), [R.recorded(st, prog, r) for r in range(len(spec.recorders))]))
    (a, ra), (b, rb) = got
    for c in P.active_components(2, pol):
        np.testing.assert_array_equal(a[c], b[c], err_msg=c)
    for k in ("psi_h", "psi_e"):
        for x, y in zip(a[k], b[k]):
            np.testing.assert_array_equal(x, y, err_msg=k)
    for k in ("dft_re", "dft_im", "dft_w"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    for x, y in zip(ra, rb):
        assert x.keys() == y.keys()
        for k in x:
            np.testing.assert_array_equal(x[k], y[k], err_msg=k)
