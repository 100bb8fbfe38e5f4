"""<v, A u> = <A^T v, u> for one step A over fields and CPML memories, with
E and H coefficients that decay (per site and uniform), TM, TE and 3D, CPML,
metallic walls and derivative metrics.  A is a step of the phase kernels, A^T
fdtd_adjoint_steps: nothing is shared between the two sides."""

from __future__ import annotations

import ctypes
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from beamz_b200 import abi  # noqa: E402
from beamz_b200 import plan as P  # noqa: E402
from beamz_b200 import runtime as R  # noqa: E402
from tests.scenarios import scenario_2d, scenario_3d, with_metrics  # noqa: E402

pytestmark = pytest.mark.gpu


def _spec(kind, material, metallic, metric, seed):
    """A scene in units of its cells, with E and H coefficients of order one."""
    rng = np.random.default_rng(seed)
    if kind == "3d":
        spec = scenario_3d(grid=(13, 18, 35), seed=seed, pml_cells=3, metallic=metallic, sources=False, monitors=False)
    else:
        spec = dataclasses.replace(scenario_2d(grid=(37, 70), polarization=kind, pml_cells=5, metallic=metallic),
                                   sources=[], monitors=[])
    act = P.active_components(spec.ndim, spec.polarization)
    pairs = {}
    for c in act:
        shape = P.component_shape(c, spec.grid_shape, spec.polarization) if material == "site" or c[0] == "E" else ()
        lossless = material == "lossless"
        decay = np.float32(1.0) if lossless else rng.uniform(0.6, 0.95, shape).astype(np.float32)
        pairs[c] = (decay, rng.uniform(0.2, 0.5, shape).astype(np.float32))
    spec = dataclasses.replace(spec, resolution=1.0, voxel_ids=None, eps_table=None, e_site_eps=None,
                               e_site={c: v for c, v in pairs.items() if c[0] == "E"},
                               h_site={c: v for c, v in pairs.items() if c[0] == "H"})
    return with_metrics(spec, metric, seed=seed) if metric else spec


def _randomize(st, rng):
    tensors = [f for f in st.fields if f.numel()] + list(st.psi_h) + list(st.psi_e)
    for t in tensors:
        t.copy_(torch.as_tensor(rng.standard_normal(tuple(t.shape)).astype(np.float32)))
    return tensors, [t.clone() for t in tensors]


def _dot(a, b, f=lambda t: t):
    return sum(float((f(x.double()) * f(y.double())).sum()) for x, y in zip(a, b))


@pytest.mark.parametrize("metallic,metric", [((), None), (("left", "top", "front"), None), (("right", "bottom"), "rectilinear")])
@pytest.mark.parametrize("material", ["lossless", "uniform", "site"])
@pytest.mark.parametrize("kind", ["tm", "te", "3d"])
def test_adjoint_step_transposes_the_phase_step(kind, material, metallic, metric):
    if kind != "3d":
        metallic = tuple(m for m in metallic if m != "front")
    spec = _spec(kind, material, metallic, metric, seed=3)
    prog = R.compile_program(spec, schedule="phases", layout="dense")
    rng = np.random.default_rng(7)
    st = R.initial_state(prog)
    u1, u0 = _randomize(st, rng)
    R.run_steps(st, prog, 1)
    lam = R.initial_state(prog)
    l0, l1 = _randomize(lam, rng)
    a = abi.FdtdAdjointStep()
    a.abi_version, a.step = abi.FDTD_ABI_VERSION, 0
    s = prog.fill(lam, 0)
    abi.check(prog.lib.fdtd_adjoint_steps(R._stream(prog), ctypes.byref(s), ctypes.byref(a), 1), "fdtd_adjoint_steps")
    # At most 16 float32 roundings lie between an input and an output, of terms
    # whose magnitudes the sums of |v| |A u| and |A^T v| |u| stand for.
    bound = 16 * 2.0**-24 * (_dot(l1, u1, torch.abs) + _dot(l0, u0, torch.abs))
    lhs, rhs = _dot(l1, u1), _dot(l0, u0)
    assert abs(lhs - rhs) <= bound, (lhs, rhs, bound)
