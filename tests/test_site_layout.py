"""Which programs take the pitched layout with per-site coefficients: its padded
fields must stay below 2^31 elements where the dense components do."""

from __future__ import annotations

import types

import numpy as np
import pytest

from beamz_b200 import adjoint as A
from beamz_b200 import runtime as R


@pytest.mark.parametrize("grid,ok", [
    ((1023, 1023, 2043), True),    # 2^20 x 2044: the last pitch below 2^11
    ((1023, 1023, 2044), False),   # dense 2^20 x 2045 fits, its pitch 2048 does not
    ((1, 1, 4), True),
])
def test_padded_fields_stay_below_the_element_limit(grid, ok):
    assert R.pitched_size_ok(grid) is ok


def test_gradients_beyond_the_limit_stay_dense():
    problem = object.__new__(A.AdjointProblem)
    problem.curl_record = object()
    one = (np.float32(1.0), np.float32(0.5))
    spec = types.SimpleNamespace(ndim=3, metrics=None, voxel_ids=None, e_site={c: one for c in ("Ex", "Ey", "Ez")},
                                 h_coefficients=lambda: {c: one for c in ("Hx", "Hy", "Hz")})
    spec.grid_shape = (64, 64, 64)
    assert problem._forward_layout(spec) == "site"
    spec.grid_shape = (1023, 1023, 2044)
    assert problem._forward_layout(spec) == "dense"
