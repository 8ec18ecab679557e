"""The two-call Rayleigh--Ritz step of the eigensolver iteration against the separate entry points."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ham(pkg, cuda):
    grid = pkg.UniformGrid((17, 19, 23), 0.4, (-3.2, -3.6, -4.4), device=cuda)
    geo = pkg.build_cusp_geometry(grid, (2.0,), ((0.0, 0.0, 0.0),))
    return pkg.CuspFactoredHamiltonian(geo.grid, geo.factor, quadrature=geo.quadrature)


def _block(m, n, dev):
    return torch.randn((m, n), dtype=torch.float64, generator=torch.Generator().manual_seed(m)).to(dev)


# one orbital, a partial and a full lane, the last width with register kernels for eigh and products, the widest
@pytest.mark.parametrize("m,n_states", [(1, 1), (2, 1), (3, 3), (5, 2), (6, 6), (7, 1), (8, 5)])
def test_step_matches_the_entry_points(pkg, cuda, ham, m, n_states):
    n = ham.grid.n_points
    block = _block(m, n, cuda)
    previous = torch.linspace(-1.0, 1.0, m, dtype=torch.float64, device=cuda)
    evals, vectors, residuals, summary = pkg.eigen.RitzStep(ham.measure, m, block.device)(ham, block, previous, n_states)
    e, v, orth = pkg.rayleigh_ritz(ham, block, ham.measure)
    r = pkg.residual_norms(ham, e, v, ham.measure)
    # the same kernels but for the residual's sum (positive terms in another order): n eps
    assert torch.equal(evals, e) and torch.equal(vectors, v)
    torch.testing.assert_close(residuals, r, rtol=2e-12, atol=0.0)
    want = [float(r[:n_states].max()), float((e - previous)[:n_states].abs().max()), orth, float(e[-1]), 0.0]
    torch.testing.assert_close(summary.cpu(), torch.tensor(want, dtype=torch.float64), rtol=2e-12, atol=0.0)


def test_step_reports_a_dependent_block(pkg, cuda, ham):
    block = _block(4, ham.grid.n_points, cuda)
    block[3] = 0.0  # the Gram matrix' last pivot is exactly zero
    step = pkg.eigen.RitzStep(ham.measure, 4, block.device)
    summary = step(ham, block, torch.zeros(4, dtype=torch.float64, device=cuda), 2)[3]
    assert float(summary[4]) == 4.0
