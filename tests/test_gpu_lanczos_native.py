"""The Lanczos recurrence in one library call against the recurrence over the operator's apply."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


# an odd box (vectors of an odd length in one work buffer) and an even one; one step to the default's; both stencils
@pytest.mark.parametrize("shape,order", [((15, 15, 17), 8), ((16, 18, 24), 8), ((15, 17, 16), 4)])
@pytest.mark.parametrize("steps", [1, 2, 12])
def test_native_recurrence_matches(pkg, cuda, shape, order, steps):
    grid = pkg.UniformGrid(shape, 0.4, tuple(-0.4 * (s // 2) for s in shape), device=cuda, fd_order=order)
    geo = pkg.build_cusp_geometry(grid, (2.0,), ((0.0, 0.0, 0.0),))
    ham = pkg.CuspFactoredHamiltonian(geo.grid, geo.factor, quadrature=geo.quadrature)
    start = torch.randn(geo.grid.n_points, dtype=torch.float64, generator=torch.Generator().manual_seed(3)).to(cuda)
    before = ham.apply_count
    got = pkg.operators._native_lanczos(ham, start, steps)
    assert ham.apply_count - before == steps
    # the same launches on the same values
    assert torch.equal(got, pkg.operators._lanczos_recurrence(ham, start, steps))
