"""Phase-level calls on fused programs with one E coefficient per site, which
compile onto the pitched layout: half steps, sources, monitors, recorders and the
design-box curl as on the dense layout, bit for bit, alone and between runs of
whole steps."""

from __future__ import annotations

import ctypes
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from beamz_b200 import abi  # noqa: E402
from beamz_b200 import adjoint as A  # noqa: E402
from beamz_b200 import plan as P  # noqa: E402
from beamz_b200 import runtime as R  # noqa: E402
from tests.scenarios import random_initial_fields, scenario_3d  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,metallic,cpml", [
    ((9, 10, 37), (), True), ((12, 7, 128), ("front", "right", "top"), True), ((6, 9, 35), ("left", "back"), False),
])
def test_phase_calls_on_per_site_programs(grid, metallic, cpml):
    kw = dict(pml_cells=3) if cpml else dict(cpml_edges=())
    spec = scenario_3d(grid=grid, seed=5, metallic=metallic, nsteps=9, **kw)
    eps = torch.as_tensor(np.random.default_rng(5).uniform(2.0, 12.0, grid).astype(np.float32), device="cuda")
    coefs = A.eps_to_coefficients_3d(eps, spec.dt, P.EPS_0)
    spec = A.site_spec(spec, {c: v.cpu().numpy() for c, v in zip(("Ex", "Ey", "Ez"), coefs)})
    spec = dataclasses.replace(spec, recorders=[P.domain_recorder(grid, ("Hx", "Ez"), interval=2, num_steps=9)])
    fields = random_initial_fields(spec, seed=3)
    got = []
    for layout, schedule in (("auto", "fused"), ("dense", "phases")):
        prog = R.compile_program(spec, layout=layout, schedule=schedule)
        assert prog.per_site == (schedule == "fused")
        st = R.initial_state(prog, fields=fields)
        for _ in range(3):
            R.step_by_phases(st, prog)
        R.run_steps(st, prog, 3)
        R.step_by_phases(st, prog)
        out = st.numpy()
        lo, hi = (grid[0] // 2, grid[1] // 2, 8), (grid[0] // 2 + 1, grid[1] // 2 + 1, 20)
        curls = [torch.zeros(tuple(b - a for a, b in zip(lo, hi)), device="cuda") for _ in range(3)]
        a = abi.FdtdAdjointStep()
        a.abi_version = abi.FDTD_ABI_VERSION
        a.box_lo[:], a.box_hi[:] = list(lo), list(hi)
        for c in range(3):
            a.curl[c] = abi.buffer_of(curls[c])
        s = prog.fill(st, 0)
        abi.check(prog.lib.fdtd_adjoint_curl(R._stream(prog), ctypes.byref(s), ctypes.byref(a)), "curl")
        got.append((out, R.recorded(st, prog, 0), [c.cpu().numpy() for c in curls]))
    (a, ra, ca), (b, rb, cb) = got
    for c in P.COMPONENTS:
        np.testing.assert_array_equal(a[c], b[c], err_msg=c)
    for k in ("psi_h", "psi_e"):
        for x, y in zip(a[k], b[k]):
            np.testing.assert_array_equal(x, y, err_msg=k)
    for k in ("dft_re", "dft_im", "dft_w"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    for k in ra:
        np.testing.assert_array_equal(ra[k], rb[k], err_msg=k)
    for x, y in zip(ca, cb):
        assert np.abs(x).max() > 0
        np.testing.assert_array_equal(x, y)


def test_codebook_programs_still_refuse_phase_calls():
    prog = R.compile_program(scenario_3d(grid=(9, 10, 37), seed=1, nsteps=3))
    assert prog.layout == "pitched" and not prog.per_site
    with pytest.raises(abi.FdtdError):
        R.update_h(R.initial_state(prog), prog)
