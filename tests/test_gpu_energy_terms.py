"""The energies of a Kohn--Sham step: which of them belong to the orbitals and which to the density passed in."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def state(pkg, cuda):
    grid = pkg.UniformGrid((21, 21, 21), 0.4, (-4.0, -4.0, -4.0), device=cuda)
    geo = pkg.build_cusp_geometry(grid, (2.0,), ((0.0, 0.0, 0.0),))
    step = pkg.KohnShamStep(geo, "lda_vwn", 2.0)
    p_in = step.potentials(pkg.initial_density(step))
    eigen = step.diagonalise(step.hamiltonian(p_in), max_iterations=2)[0]
    return step, p_in, eigen, step.occupy(eigen.eigenvalues)


def test_kinetic_energy_is_that_of_the_orbitals(pkg, state):
    """A mixed density changes the terms that are integrals of it, not the kinetic energy."""
    step, p_in, eigen, occupations = state
    rho_out = step.output_density(eigen, occupations)[1]
    ham = step._bare
    kinetic = ham.kinetic_energy_tensor(eigen.eigenvectors, occupations[0])
    for rho in (rho_out, 0.7 * rho_out):
        terms = step.energy_terms(eigen, occupations, rho, p_in, None)
        assert torch.equal(terms["kinetic"], kinetic)
        assert torch.equal(terms["external_direct"], ham.external_energy_direct_tensor(rho))


def test_shared_integrals_change_nothing(pkg, state):
    step, p_in, eigen, occupations = state
    rho_out = step.output_density(eigen, occupations)[1]
    want = step.energy_terms(eigen, occupations, rho_out, p_in, None)
    got = step.energy_terms(eigen, occupations, rho_out, p_in, None, rho_is_of_orbitals=True)
    assert all(torch.equal(got[k], want[k]) for k in want)
