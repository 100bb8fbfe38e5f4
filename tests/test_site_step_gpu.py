"""The class step with one E coefficient per site (pitched FDTD_MATERIAL_SITE)
against the phase schedule on the dense layout, bit for bit: full and partial
last tiles, metallic walls, sources at every timing, and the automatic choice
for materials with more coefficients than the codebook holds."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from beamz_b200 import adjoint as A  # noqa: E402
from beamz_b200 import plan as P  # noqa: E402
from beamz_b200 import runtime as R  # noqa: E402
from tests.scenarios import random_initial_fields, scenario_3d  # noqa: E402

pytestmark = pytest.mark.gpu


def _smooth(grid, seed, **kw):
    """``scenario_3d`` with a continuous permittivity."""
    spec = scenario_3d(grid=grid, seed=seed, **kw)
    eps = torch.as_tensor(np.random.default_rng(seed).uniform(2.0, 12.0, grid).astype(np.float32), device="cuda")
    coefs = A.eps_to_coefficients_3d(eps, spec.dt, P.EPS_0)
    return A.site_spec(spec, {c: v.cpu().numpy() for c, v in zip(("Ex", "Ey", "Ez"), coefs)})


@pytest.mark.parametrize("grid,pml,metallic,sources", [
    ((9, 10, 37), 3, (), True), ((12, 7, 128), 3, ("front", "right"), True), ((20, 31, 130), 4, ("top",), False),
    ((33, 24, 256), 12, ("back", "left", "bottom"), False), ((5, 16, 300), 0, ("front", "back"), False),
])
def test_site_step_matches_the_phase_schedule(grid, pml, metallic, sources):
    kw = dict(cpml_edges=()) if pml == 0 else dict(pml_cells=pml)
    spec = _smooth(grid, 5, metallic=metallic, sources=sources, **kw)
    if pml < 12:
        spec = dataclasses.replace(spec, recorders=[P.domain_recorder(grid, ("Hx", "Ez"), interval=2, num_steps=9)])
    fields = random_initial_fields(spec, seed=3)
    got = []
    for layout, schedule in (("auto", "fused"), ("dense", "phases")):
        prog = R.compile_program(spec, schedule=schedule, layout=layout)
        st = R.run_steps(R.initial_state(prog, fields=fields), prog, 9)
        if schedule == "fused":
            assert prog.layout == "pitched" and prog.step_kernel == ("site" if prog.per_site else "classes")
            assert prog.per_site == (np.unique(spec.e_site["Ex"][1]).size > 256)
        got.append((st.numpy(), [R.recorded(st, prog, r) for r in range(len(spec.recorders))],
                    R.field_diagnostics(st, prog)))
    (a, ra, da), (b, rb, db) = got
    for c in P.COMPONENTS:
        np.testing.assert_array_equal(a[c], b[c], err_msg=c)
    for k in ("psi_h", "psi_e"):
        for x, y in zip(a[k], b[k]):
            np.testing.assert_array_equal(x, y, err_msg=k)
    for k in ("dft_re", "dft_im", "dft_w"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    for x, y in zip(ra, rb):
        for k in x:
            np.testing.assert_array_equal(x[k], y[k], err_msg=k)
    assert da.nonfinite == db.nonfinite and da.max_field == db.max_field
    assert abs(da.energy - db.energy) <= 1e-6 * abs(db.energy)


def test_site_layout_takes_new_coefficients():
    """layout="site" on a two-material scene, coefficients replaced in place."""
    grid = (12, 14, 129)
    base = _smooth(grid, 7, pml_cells=3)
    two = dataclasses.replace(base, e_site={c: (np.float32(1), np.full_like(v[1], 1e-3)) for c, v in base.e_site.items()})
    fields = random_initial_fields(base, seed=1)
    prog = R.compile_program(two, layout="site")
    for c in ("Ex", "Ey", "Ez"):
        prog.e_source[c].copy_(torch.as_tensor(base.e_site[c][1], device="cuda"))
    out = R.run_steps(R.initial_state(prog, fields=fields), prog, 4).numpy()
    ref = R.compile_program(base, schedule="phases", layout="dense")
    want = R.run_steps(R.initial_state(ref, fields=fields), ref, 4).numpy()
    for c in P.COMPONENTS:
        np.testing.assert_array_equal(out[c], want[c], err_msg=c)
    with pytest.raises(ValueError):
        R.compile_program(two, layout="site", arithmetic="fast")
