"""The triangular solve that writes the apply's lanes, against the solve and the apply as calls of their own."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


# odd and even block widths (a thread takes two systems or one), an odd number of systems (a half-empty last pair),
# a last lane with an empty slot, odd and even rows; the widest, one beyond it and another order, which take two calls
@pytest.mark.parametrize("m,systems,shape,order", [
    (1, 1, (15, 15, 17), 8), (1, 2, (15, 15, 16), 8), (2, 3, (15, 15, 17), 8), (3, 3, (15, 17, 19), 8),
    (5, 1, (15, 16, 17), 8), (5, 4, (16, 15, 18), 8), (6, 2, (15, 15, 17), 8), (7, 5, (15, 15, 15), 8),
    (8, 3, (15, 15, 21), 8), (9, 2, (15, 15, 17), 8), (4, 2, (15, 15, 17), 4)])
def test_matches_the_two_calls(pkg, cuda, m, systems, shape, order):
    grid = pkg.UniformGrid(shape, 0.4, tuple(-0.4 * (s // 2) for s in shape), device=cuda, fd_order=order)
    geo = pkg.build_cusp_geometry(grid, (2.0,), ((0.0, 0.0, 0.0),))
    n = grid.n_points
    g = torch.Generator().manual_seed(m)
    pots = torch.randn((systems, n), dtype=torch.float64, generator=g).to(cuda)
    h = pkg.batch.BatchedHamiltonian(grid, geo.factor, geo.quadrature, pots)
    block = torch.randn((systems, m, n), dtype=torch.float64, generator=g).to(cuda)
    lower = (0.3 * torch.randn((systems, m, m), dtype=torch.float64, generator=g).tril()
             + 1.5 * torch.eye(m, dtype=torch.float64)).to(cuda)
    basis, want = torch.empty_like(block), torch.empty_like(block)
    pkg._lib.call("cdftb_block_trsm_lower_f64", lower.data_ptr(), block.data_ptr(), m * n, want.data_ptr(), 0, m * n, m, n,
                  systems, torch.cuda.current_stream().cuda_stream)
    got = h.apply_solved(lower, block, basis)
    # the same operations in the same order
    assert torch.equal(basis, want)
    assert torch.equal(got, h.apply(want))
