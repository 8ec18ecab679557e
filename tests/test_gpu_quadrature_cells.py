"""L and L^T over nodes sorted by base cell, against the entry points over the list of entries and over single nodes."""

from __future__ import annotations

import pytest
import torch


pytestmark = pytest.mark.gpu

GRIDS = [((17, 17, 17), 0.5, ((0.0, 0.0, 0.0),), (2.0,)),
         ((25, 30, 43), 0.31, ((0.03, -0.02, -0.8), (0.0, 0.05, 0.9)), (1.0, 1.0))]


@pytest.fixture(scope="module", params=range(len(GRIDS)))
def quadrature(request, pkg):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    shape, h, positions, charges = GRIDS[request.param]
    grid = pkg.UniformGrid(shape, h, tuple(-h * (n // 2) for n in shape), device="cuda:0")
    return pkg.build_cusp_geometry(grid, charges, positions).quadrature


def _entry_list_lift(pkg, q, x):
    """``cdftb_quadrature_lift_f64`` over the (point, node) entry list, field by field."""
    n, m = q.grid.n_points, q.n_nodes
    out = torch.empty((x.shape[0], n), dtype=torch.float64, device=x.device)
    pkg._lib.call("cdftb_quadrature_lift_f64", q.base.data_ptr(), q.w1d.data_ptr(), q.row_ptr.data_ptr(),
                  q.col.data_ptr(), q.lift_values.data_ptr(), *q.grid.shape, x.data_ptr(), x.shape[0], m,
                  out.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
    return out


@pytest.mark.parametrize("nf", [1, 2, 3, 4, 5, 7, 8, 31, 32, 33, 41])
def test_lift_matches_the_entry_list(pkg, quadrature, nf):
    """A point sums at most a few thousand products of either sign: 1e-13 of the sum of magnitudes."""
    g = torch.Generator().manual_seed(nf)
    x = torch.randn((nf, quadrature.n_nodes), dtype=torch.float64, generator=g).cuda()
    got = quadrature._lift_raw(x, nf)
    want = _entry_list_lift(pkg, quadrature, x)
    torch.testing.assert_close(got, want, rtol=0, atol=1e-13 * float(want.abs().max()))
    assert torch.equal(got == 0.0, want == 0.0)


@pytest.mark.parametrize("nf", [2, 9])
def test_lift_keeps_a_nodes_infinity_to_its_own_points(pkg, quadrature, nf):
    x = torch.ones((nf, quadrature.n_nodes), dtype=torch.float64, device="cuda:0")
    x[0, quadrature.n_nodes // 2] = float("inf")
    x[nf - 1, 3] = float("nan")
    got = quadrature._lift_raw(x, nf)
    want = _entry_list_lift(pkg, quadrature, x)
    assert torch.equal(torch.isfinite(got), torch.isfinite(want))
    torch.testing.assert_close(got[torch.isfinite(want)], want[torch.isfinite(want)], rtol=0, atol=1e-12)


@pytest.mark.parametrize("nf", [2, 9])
def test_lift_takes_strided_rows(pkg, quadrature, nf):
    q = quadrature
    n, m = q.grid.n_points, q.n_nodes
    x = torch.randn((nf, m + 5), dtype=torch.float64, device="cuda:0")
    out = torch.full((nf, n + 3), 7.0, dtype=torch.float64, device="cuda:0")
    box = q._cell_box.ctypes.data
    nbytes = pkg._lib.library().cdftb_lift_cells_scratch_bytes(m, *q.grid.shape, box, nf)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda:0")
    pkg._lib.call("cdftb_quadrature_lift_cells_f64", q._cell_plan.data_ptr(), q._cell_plan.numel(), m, *q.grid.shape, box,
                  x.data_ptr(), nf, m + 5, out.data_ptr(), n + 3, scratch.data_ptr(), nbytes,
                  torch.cuda.current_stream().cuda_stream)
    assert torch.equal(out[:, :n], q._lift_raw(x[:, :m].contiguous(), nf))
    assert bool((out[:, n:] == 7.0).all())


@pytest.mark.parametrize("nf", [1, 2, 3, 4, 5, 6, 7])
def test_interpolant_of_a_few_fields(pkg, quadrature, nf):
    """Groups of a cell against a warp per node and the many-field kernel: 512 products of sums of weights
    below 3 per axis, 1e-13 of the largest value."""
    q = quadrature
    n, m = q.grid.n_points, q.n_nodes
    g = torch.Generator().manual_seed(nf)
    fields = torch.randn((nf, n), dtype=torch.float64, generator=g).cuda()
    got = q._interp_raw(fields, nf)
    one = torch.full((nf, m + 3), 7.0, dtype=torch.float64, device="cuda:0")
    pkg._lib.call("cdftb_quadrature_interpolate_f64", q.base.data_ptr(), q.w1d.data_ptr(), m, *q.grid.shape,
                  fields.data_ptr(), nf, n, one.data_ptr(), m + 3, torch.cuda.current_stream().cuda_stream)
    many = q._interp_raw(fields.repeat(8, 1), 8 * nf)[:nf]
    scale = float(many.abs().max())
    torch.testing.assert_close(got, many, rtol=0, atol=1e-13 * scale)
    torch.testing.assert_close(one[:, :m], many, rtol=0, atol=1e-13 * scale)
    assert bool((one[:, m:] == 7.0).all())
