"""The (point, node) lists of L^T, which are built when first read, and the many-field lift over them."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _quadrature(pkg):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    grid = pkg.UniformGrid((25, 30, 43), 0.31, (-3.72, -4.65, -6.51), device="cuda:0")
    return pkg.build_cusp_geometry(grid, (1.0, 1.0), ((0.03, -0.02, -0.8), (0.0, 0.05, 0.9))).quadrature


def test_lists_are_whole_on_every_stream(pkg):
    """Read first on one stream, behind other work, and then on another one."""
    q = _quadrature(pkg)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda._sleep(200_000_000)
        q.row_ptr
    names = ("row_ptr", "col", "lift_values", "seg_ptr", "seg_row")
    early = [getattr(q, k).cpu() for k in names]
    torch.cuda.synchronize()
    segments = int(q.seg_ptr[-1])
    for name, got in zip(names, early):
        count = segments if name == "seg_row" else got.numel()
        assert torch.equal(got[:count], getattr(q, name).cpu()[:count]), name


@pytest.mark.parametrize("nf", [1, 8, 32, 33])
def test_many_field_lift_over_segments(pkg, nf):
    """Sums of a few thousand products per point in another order: 1e-13 of the largest."""
    q = _quadrature(pkg)
    n, m = q.grid.n_points, q.n_nodes
    x = torch.randn((nf, m), dtype=torch.float64, generator=torch.Generator().manual_seed(nf)).cuda()
    out = torch.empty((nf, n), dtype=torch.float64, device="cuda:0")
    scratch = q._many_scratch(x.device)
    pkg._lib.call("cdftb_quadrature_lift_many_f64", q.row_ptr.data_ptr(), q.col.data_ptr(), q.lift_values.data_ptr(),
                  q.seg_ptr.data_ptr(), q.seg_row.data_ptr(), q.seg_capacity, *q.grid.shape, m, x.data_ptr(), nf, m,
                  out.data_ptr(), n, scratch.data_ptr(), scratch.numel(), torch.cuda.current_stream().cuda_stream)
    want = q._lift_raw(x, nf)
    torch.testing.assert_close(out, want, rtol=0, atol=1e-13 * float(want.abs().max()))
