"""Site coefficients of a voxel permittivity: the values of clipped gathers, and
only of grids with as many axes as the function is for."""

from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from beamz_b200 import adjoint as A  # noqa: E402
from beamz_b200 import plan as P  # noqa: E402


@pytest.mark.parametrize("shape", [(4, 5, 6), (3,), (2, 4, 5, 6)])
def test_2d_coefficients_need_two_axes(shape):
    with pytest.raises(ValueError):
        A.eps_to_coefficients_2d(torch.ones(shape), 1e-17, P.EPS_0)


@pytest.mark.parametrize("shape", [(5, 6), (3,), (2, 4, 5, 6)])
def test_3d_coefficients_need_three_axes(shape):
    with pytest.raises(ValueError):
        A.eps_to_coefficients_3d(torch.ones(shape), 1e-17, P.EPS_0)


@pytest.mark.parametrize("shape", [(1, 1, 1), (4, 5, 6), (2, 1, 7)])
def test_coefficients_equal_clipped_gathers(shape):
    gen = torch.Generator().manual_seed(1)
    v = 2.0 + 10.0 * torch.rand(shape, generator=gen)
    lo = [torch.clamp(torch.arange(-1, n), 0, n - 1) for n in shape]
    hi = [torch.clamp(torch.arange(0, n + 1), 0, n - 1) for n in shape]

    def pair(a, dim):
        return 0.5 * (a.index_select(dim, lo[dim]) + a.index_select(dim, hi[dim]))

    want = [pair(pair(v, 0), 1), pair(pair(v, 0), 2), pair(pair(v, 1), 2)]
    ratio = torch.tensor(np.float32(np.float32(1e-17) / np.float32(P.EPS_0)))
    for got, eps in zip(A.eps_to_coefficients_3d(v, 1e-17, P.EPS_0), want):
        assert torch.equal(got, ratio * (1.0 / eps))
    rows, cols = hi[1], hi[2]
    eps = v[0][rows][:, cols]
    assert torch.equal(A.eps_to_coefficients_2d(v[0], 1e-17, P.EPS_0),
                       torch.tensor(np.float32(1e-17)) / (torch.tensor(np.float32(P.EPS_0)) * eps))
