"""The class step with per-site coefficients marching several z chunks per
column, the last one short, with H sources in it and across a chunk's edge: bit
for bit against the phase schedule."""

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


@pytest.mark.parametrize("z_chunk", [4, 8, 12])
@pytest.mark.parametrize("grid", [(29, 20, 256), (26, 17, 300)])
def test_site_step_with_short_last_chunks(grid, z_chunk):
    rng = np.random.default_rng(2)
    spec = scenario_3d(grid=grid, seed=2, pml_cells=4, metallic=("back",), nsteps=8)
    eps = torch.as_tensor(rng.uniform(2.0, 12.0, grid).astype(np.float32), device="cuda")
    coefs = A.eps_to_coefficients_3d(eps, spec.dt, P.EPS_0)
    spec = A.site_spec(spec, {c: v.cpu().numpy() for c, v in zip(("Ex", "Ey", "Ez"), coefs)})
    wave = (rng.standard_normal(8) * 1e-3).astype(np.float32)
    box = lambda *s: rng.standard_normal(s).astype(np.float32)  # noqa: E731
    spec = dataclasses.replace(spec, sources=[
        *spec.sources,
        P.SourcePlan("Hx", "h", (grid[0] - 2, 3, 120), box(2, 4, 20), wave),   # the last planes, two tiles
        P.SourcePlan("Hz", "h", (10, 6, grid[2] - 9), box(4, 3, 9), wave)])    # across the edge of a chunk
    fields = random_initial_fields(spec, seed=4)
    out = []
    for kw in (dict(z_chunk=z_chunk), dict(schedule="phases", layout="dense")):
        prog = R.compile_program(spec, **kw)
        assert prog.per_site == ("z_chunk" in kw)
        out.append(R.run_steps(R.initial_state(prog, fields=fields), prog, 7).numpy())
    for c in P.COMPONENTS:
        np.testing.assert_array_equal(out[0][c], out[1][c], err_msg=c)
    for k in ("psi_h", "psi_e"):
        for x, y in zip(out[0][k], out[1][k]):
            np.testing.assert_array_equal(x, y, err_msg=k)
