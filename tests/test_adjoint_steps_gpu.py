"""fdtd_adjoint_steps against the same steps one by one (fdtd_adjoint_step):
fields, memories and the gradient of a box whose curls differ from step to
step, bit for bit, in 2D TM and TE (which takes no box) and in 3D with CPML and a
metallic wall."""

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
from tests.scenarios import scenario_2d, scenario_3d  # noqa: E402

pytestmark = pytest.mark.gpu

_E_SRC, _H_SRC = (5, 4, 3, 5, 4, 3), (2, 1, 0, 2, 1, 0)


def _spec(kind):
    if kind != "3d":
        return dataclasses.replace(scenario_2d(grid=(31, 70), polarization=kind, pml_cells=4, metallic=("left",)),
                                   monitors=[])
    spec = scenario_3d(grid=(14, 17, 66), seed=2, pml_cells=3, metallic=("front",), sources=False, monitors=False)
    eps = torch.as_tensor(spec.eps_table[spec.voxel_ids].astype(np.float32), device="cuda")
    coefs = A.eps_to_coefficients_3d(eps, spec.dt, P.EPS_0)
    return A.site_spec(spec, {c: v.cpu().numpy() for c, v in zip(("Ex", "Ey", "Ez"), coefs)})


@pytest.mark.parametrize("kind", ["tm", "te", "3d"])
def test_a_run_of_adjoint_steps_equals_single_steps(kind):
    spec = _spec(kind)
    prog = R.compile_program(spec, schedule="phases", layout="dense")
    act = P.active_components(spec.ndim, spec.polarization)
    lo, hi = ((0, 8, 20), (1, 14, 40)) if spec.ndim == 2 else ((5, 6, 20), (8, 11, 31))
    box, count = tuple(b - a for a, b in zip(lo, hi)), 3
    rng = np.random.default_rng(5)
    dev = lambda *s: torch.as_tensor(rng.standard_normal(s).astype(np.float32), device="cuda")  # noqa: E731
    e_act = [i for i, c in enumerate(("Ex", "Ey", "Ez")) if c in act and kind != "te"]
    curls = {i: dev(count, *box) for i in e_act}
    first = R.initial_state(prog)
    tensors = lambda st: [f for f in st.fields if f.numel()] + list(st.psi_h) + list(st.psi_e)  # noqa: E731
    start = [dev(*t.shape) for t in tensors(first)]
    scratch = {"e": {}, "h": {}}
    for t in range(6):
        if P.COMPONENTS[t // 2] in act and P.COMPONENTS[_E_SRC[t]] in act:
            scratch["e"][t] = torch.zeros(prog.shapes[P.COMPONENTS[t // 2]], device="cuda")
        if P.COMPONENTS[3 + t // 2] in act and P.COMPONENTS[_H_SRC[t]] in act:
            scratch["h"][t] = torch.zeros(prog.shapes[P.COMPONENTS[3 + t // 2]], device="cuda")

    def struct(step, curl_of, grads, with_scratch):
        a = abi.FdtdAdjointStep()
        a.abi_version, a.step = abi.FDTD_ABI_VERSION, step
        for i in e_act:
            a.curl[i], a.grad[i] = abi.buffer_of(curl_of(i)), abi.buffer_of(grads[i])
        a.box_lo[:], a.box_hi[:] = list(lo), list(hi)
        if with_scratch:
            for t, b in scratch["e"].items():
                a.scratch_e[t] = abi.buffer_of(b)
            for t, b in scratch["h"].items():
                a.scratch_h[t] = abi.buffer_of(b)
        return a

    got = []
    for run in (True, False):
        st = R.initial_state(prog)
        for t, v in zip(tensors(st), start):
            t.copy_(v)
        grads = {i: torch.zeros(box, device="cuda") for i in e_act}
        s = prog.fill(st, 0)
        if run:
            a = struct(9, lambda i: curls[i], grads, False)
            abi.check(prog.lib.fdtd_adjoint_steps(R._stream(prog), ctypes.byref(s), ctypes.byref(a), count), "steps")
        else:
            for n in reversed(range(count)):
                a = struct(7 + n, lambda i: curls[i][n], grads, True)
                abi.check(prog.lib.fdtd_adjoint_step(R._stream(prog), ctypes.byref(s), ctypes.byref(a)), "step")
        torch.cuda.synchronize()
        got.append(tensors(st) + list(grads.values()))
    assert all(torch.equal(x, y) for x, y in zip(*got))
    if not e_act:
        return
    assert all(bool(g.abs().max() > 0) for g in got[0][-len(e_act):])
    bad = struct(9, lambda i: curls[i][:2], grads, False)  # curls of two steps for a run of three
    assert prog.lib.fdtd_adjoint_steps(R._stream(prog), ctypes.byref(s), ctypes.byref(bad), count) == 1
