"""One adjoint step of a program whose components hold almost 2^31 elements: the
loops over their sites pass 2^31 with the last stride."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from beamz_b200 import abi  # noqa: E402
from beamz_b200 import plan as P  # noqa: E402
from beamz_b200 import runtime as R  # noqa: E402

pytestmark = pytest.mark.gpu


def test_h_scaling_reaches_the_last_element():
    grid = (32766, 65536)  # Hz holds 2^31 - 2^17 elements, less than one stride below 2^31
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB of device memory")
    one = np.float32(1.0)
    dt = 0.7 * 20e-9 / (P.LIGHT_SPEED * np.sqrt(2.0))
    spec = P.ProgramSpec(grid, dt, 20e-9, polarization="te",
                         e_site={c: (one, np.float32(1e-3)) for c in ("Ex", "Ey")},
                         h_site={"Hz": (np.float32(0.5), np.float32(1e-3))}, total_steps=2)
    prog = R.compile_program(spec, schedule="phases", layout="dense")
    lam = R.initial_state(prog)
    hz = lam.fields[P.COMPONENT_INDEX["Hz"]]
    hz.fill_(1.0)
    a = abi.FdtdAdjointStep()
    a.abi_version, a.step = abi.FDTD_ABI_VERSION, 0
    s = prog.fill(lam, 0)
    abi.check(prog.lib.fdtd_adjoint_steps(R._stream(prog), ctypes.byref(s), ctypes.byref(a), 1), "fdtd_adjoint_steps")
    # lambda_E = 0: the E transpose leaves lambda_H, whose identity part is its decay.
    assert float(hz.min()) == 0.5 and float(hz.max()) == 0.5
    # lambda_E = D^T (source lambda_H): zero inside, where lambda_H is constant.
    assert float(lam.fields[P.COMPONENT_INDEX["Ex"]][1:-1].abs().max()) == 0.0
