"""Several 2D steps per launch on every launch shape (tiles of one wave up to 32
rows and taller ones, grids of several waves) with conductive material and
derivative metrics, bit for bit against the phase schedule."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from beamz_b200 import plan as P  # noqa: E402
from beamz_b200 import runtime as R  # noqa: E402
from tests.scenarios import random_initial_fields  # noqa: E402
from tests.test_block2d_gpu import _rich  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(150, 170), (330, 340), (700, 500)])
@pytest.mark.parametrize("pol", ["tm", "te"])
@pytest.mark.parametrize("options", [dict(conductive=True), dict(metric="rectilinear"),
                                     dict(conductive=True, metric="axis_uniform"),
                                     dict(conductive=True, cpml=False), dict(metric="rectilinear", cpml=False)])
def test_blocked_steps_on_every_launch_shape(grid, pol, options):
    spec = _rich(grid, pol, 6, seed=11, metallic=("left", "bottom"), recorders=grid[0] < 700, **options)
    fields = random_initial_fields(spec, seed=3)
    got = []
    for schedule in ("fused", "phases"):
        prog = R.compile_program(spec, schedule=schedule)
        st = R.run_steps(R.initial_state(prog, fields=fields), prog, 11)
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
        for k in x:
            np.testing.assert_array_equal(x[k], y[k], err_msg=k)
