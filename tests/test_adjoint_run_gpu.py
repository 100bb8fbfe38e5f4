"""fdtd_adjoint_steps rejects a run that would pass step 0 (its samples would be
step 0's, injected again), before it enqueues anything."""

from __future__ import annotations

import ctypes

import pytest

torch = pytest.importorskip("torch")

from beamz_b200 import abi  # noqa: E402
from beamz_b200 import runtime as R  # noqa: E402
from tests.scenarios import scenario_2d  # noqa: E402

pytestmark = pytest.mark.gpu


def test_runs_end_at_step_zero():
    prog = R.compile_program(scenario_2d(grid=(20, 30), nsteps=8), schedule="phases", layout="dense")
    lam = R.initial_state(prog)
    g = torch.ones_like(lam.dft_re)
    a = abi.FdtdAdjointStep()
    a.abi_version = abi.FDTD_ABI_VERSION
    a.dft_grad_re, a.dft_grad_im = abi.buffer_of(g), abi.buffer_of(g)
    s = prog.fill(lam, 0)

    def run(step, count):
        a.step = step
        return prog.lib.fdtd_adjoint_steps(R._stream(prog), ctypes.byref(s), ctypes.byref(a), count)

    for step, count in ((1, 3), (0, 2), (-1, 1), (5, 0)):
        assert run(step, count) == 1
    torch.cuda.synchronize()
    assert all(float(f.abs().sum()) == 0.0 for f in lam.fields if f.numel())
    assert run(2, 3) == 0
    assert any(float(f.abs().sum()) > 0.0 for f in lam.fields if f.numel())
