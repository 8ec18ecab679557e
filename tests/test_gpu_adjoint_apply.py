"""The one-call backward pass of the order-8 apply against the torch composition it stands for."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(shape, seed, dev):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(shape, dtype=torch.float64, generator=g).to(dev)


# odd z lengths (misaligned rows), boxes under one tile and over several, batches that fill lanes or not
@pytest.mark.parametrize("shape,lead", [((15, 15, 17), (1,)), ((17, 15, 37), (3,)), ((21, 25, 33), (2, 2)), ((15, 40, 25), ())])
@pytest.mark.parametrize("needs_potential", [True, False])
def test_backward_matches_the_torch_composition(pkg, cuda, shape, lead, needs_potential):
    h = 0.4
    grid = pkg.UniformGrid(shape, h, tuple(-h * (s // 2) for s in shape), device=cuda)
    geo = pkg.build_cusp_geometry(grid, (2.0,), ((0.0, 0.0, 0.0),))
    ham = pkg.CuspFactoredHamiltonian(geo.grid, geo.factor, quadrature=geo.quadrature)
    n = geo.grid.n_points
    phi = _rand((*lead, n), 1, cuda).requires_grad_(True)
    pot = (ham.graph_potential() + 0.1 * _rand((n,), 2, cuda)).requires_grad_(needs_potential)
    y_bar = _rand((*lead, n), 3, cuda)
    out = pkg.adjoint.CuspApply.apply(phi, pot, ham)
    wanted = (phi, pot) if needs_potential else (phi,)
    got = torch.autograd.grad(out, wanted, y_bar, retain_graph=True)
    ref = torch.autograd.grad(out, wanted, y_bar.requires_grad_(True), create_graph=True)  # the torch route
    # sums of ~60 terms (divergence) or the batch's, each rounded at 1.1e-16 of terms below the largest value
    # times the stencil's cancellation (< 20): 1e-12 of the largest value
    for a, b in zip(got, ref):
        assert a.shape == b.shape
        assert float((a - b.detach()).abs().max()) <= 1e-12 * float(b.detach().abs().max())
