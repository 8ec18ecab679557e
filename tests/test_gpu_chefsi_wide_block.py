"""The eigensolver's iteration for start blocks wider than the wanted states and their extra ones, and for operators
that return their result in another shape."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ham(pkg, cuda):
    grid = pkg.UniformGrid((17, 19, 23), 0.4, (-3.2, -3.6, -4.4), device=cuda)
    geo = pkg.build_cusp_geometry(grid, (2.0,), ((0.0, 0.0, 0.0),))
    return geo


def _solve(pkg, geo, n_states, block, operator=None):
    h = pkg.CuspFactoredHamiltonian(geo.grid, geo.factor, quadrature=geo.quadrature)
    lower = []

    def engine(hamiltonian, vectors, degree, low, *bounds):
        lower.append(low)
        return pkg.chebyshev_filter(hamiltonian, vectors, degree, low, *bounds)

    solver = pkg.ChebyshevFilteredSubspace(geo.grid, pkg.EigenConfig(max_iterations=3), filter_engine=engine)
    result = solver.solve(operator(h) if operator else h, n_states, initial=block, generator=torch.Generator().manual_seed(5))
    return lower, result, h


# one state: 5 rows wanted of 6 and of 8; two: 6 of 7; a block of just the wanted rows and one that is filled up
@pytest.mark.parametrize("n_states,rows", [(1, 6), (1, 8), (2, 7), (2, 6), (3, 4)])
def test_filter_bound_is_the_wanted_blocks_top(pkg, cuda, ham, monkeypatch, n_states, rows):
    """The interval starts at the value of row n_states + extra, whichever code forms the Ritz step."""
    n = ham.grid.n_points
    block = torch.randn((rows, n), dtype=torch.float64, generator=torch.Generator().manual_seed(rows)).to(cuda)
    lower, result, h = _solve(pkg, ham, n_states, block)
    monkeypatch.setattr(pkg.eigen.RitzStep, "MOST", 0)  # the separate entry points
    want_lower, want, want_h = _solve(pkg, ham, n_states, block)
    # the same steps up to the order of sums; 3 filters of a random block amplify 1e-16 by far less than 1e6
    assert len(lower) == 3 and lower == pytest.approx(want_lower, rel=1e-9)
    torch.testing.assert_close(result.eigenvalues, want.eigenvalues, rtol=1e-9, atol=1e-9)
    assert (result.n_iterations, h.apply_count) == (want.n_iterations, want_h.apply_count)


class _Reshaping:
    """An operator whose apply returns ``(1, m, N)``."""

    def __init__(self, inner):
        self._inner = inner

    def __getattr__(self, name):
        return getattr(self._inner, name)

    def apply(self, phi):
        return self._inner.apply(phi)[None]


def test_operator_may_return_another_shape(pkg, cuda, ham):
    block = torch.randn((5, ham.grid.n_points), dtype=torch.float64, generator=torch.Generator().manual_seed(1)).to(cuda)
    want = _solve(pkg, ham, 1, block)[1]
    got = _solve(pkg, ham, 1, block, _Reshaping)[1]
    assert torch.equal(got.eigenvalues, want.eigenvalues)
