"""The LDA potentials with their sums formed on the way, and the cusp coefficients straight from the density,
against the separate entry points."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(shape, seed, dev, low=0.0):
    g = torch.Generator().manual_seed(seed)
    return low + torch.rand(shape, dtype=torch.float64, generator=g).to(dev)


def _close(got, want, terms=None):
    scale = float(want.abs().max()) if terms is None else float(terms)
    torch.testing.assert_close(got, want, rtol=0.0, atol=1e-13 * scale)


# points and nodes below, at and above a multiple of a CTA's 512; no node at all
@pytest.mark.parametrize("batch,n,m,na", [(1, 511, 0, 1), (1, 512, 1, 2), (3, 513, 512, 8), (2, 1500, 1025, 3), (33, 7, 3, 1)])
def test_sums_match_the_terms(pkg, cuda, batch, n, m, na):
    call = pkg._lib.call
    stream = torch.cuda.current_stream().cuda_stream
    empty = lambda *s: torch.empty(s, dtype=torch.float64, device=cuda)  # noqa: E731
    dens, rho, vs = (_rand((batch, n), k, cuda, 0.1) for k in (1, 2, 3))
    f2, far, mass, v1s = (_rand(s, k, cuda, 0.2) for k, s in ((4, n), (5, n), (6, n), (7, (na, n))))
    coef, lifted = _rand((batch, na), 8, cuda, -0.5), _rand((batch, 2, n), 9, cuda, -0.5)
    fields, w, f2n, v1sn = (_rand(s, k, cuda, 0.1) for k, s in ((10, (2, batch, m)), (11, m), (12, m), (13, (na, m))))
    x, e_w = empty(batch, 2, m), empty(batch, m)
    call("cdftb_potentials_node_lda_f64", fields.data_ptr(), m, w.data_ptr(), f2n.data_ptr(), v1sn.data_ptr(),
         coef.data_ptr(), na, batch, x.data_ptr(), e_w.data_ptr(), stream)
    eff, vh, vx, terms = empty(batch, n), empty(batch, n), empty(batch, n), empty(batch, 3, n)
    common = [t.data_ptr() for t in (dens, rho, f2, far, mass, vs, v1s, coef)] + [na, lifted.data_ptr()]
    call("cdftb_potentials_grid_lda_f64", *common, n, batch, eff.data_ptr(), vh.data_ptr(), terms.data_ptr(),
         vx.data_ptr(), stream)
    nbytes = pkg._lib.library().cdftb_potentials_lda_work_bytes(m, n, batch)
    work = torch.empty(nbytes, dtype=torch.uint8, device=cuda)
    x2, eff2, vh2, vx2, energies = empty(batch, 2, m), empty(batch, n), empty(batch, n), empty(batch, n), empty(batch, 3)
    call("cdftb_potentials_node_lda_sums_f64", fields.data_ptr(), m, n, w.data_ptr(), f2n.data_ptr(), v1sn.data_ptr(),
         coef.data_ptr(), na, batch, x2.data_ptr(), work.data_ptr(), nbytes, stream)
    call("cdftb_potentials_grid_lda_sums_f64", *common, m, n, batch, eff2.data_ptr(), vh2.data_ptr(), vx2.data_ptr(),
         energies.data_ptr(), work.data_ptr(), nbytes, stream)
    for got, want in ((x2, x), (eff2, eff), (vh2, vh), (vx2, vx)):
        if want.numel():
            _close(got, want)
    sums = terms.sum(dim=2)
    want = torch.stack([0.5 * sums[:, 0], sums[:, 1], e_w.sum(dim=1) + sums[:, 2]], dim=1)
    _close(energies, want, float(terms.abs().sum(dim=2).max() + (e_w.abs().sum(dim=1).max() if m else 0.0)))


# nuclei whose stencils touch the box's faces; one to the most nuclei; several systems
@pytest.mark.parametrize("shape,na,batch", [((8, 8, 8), 1, 1), ((9, 11, 14), 2, 3), ((12, 8, 17), 8, 40)])
def test_coefficients_match_the_interpolant(pkg, cuda, shape, na, batch):
    call = pkg._lib.call
    stream = torch.cuda.current_stream().cuda_stream
    n = shape[0] * shape[1] * shape[2]
    dens, f2 = _rand((batch, n), 1, cuda, 0.1), _rand(n, 2, cuda, 0.2)
    base = torch.tensor([[3 if a % 2 else s - 5 for s in shape] for a in range(na)], dtype=torch.int32, device=cuda)
    w1d, nf2 = _rand((na, 24), 3, cuda, -0.3), _rand(na, 4, cuda, 0.5)
    overlap = torch.eye(na, dtype=torch.float64, device=cuda) + 0.05 * _rand((na, na), 5, cuda)
    rho, smooth, at, want, got = (torch.empty(s, dtype=torch.float64, device=cuda)
                                  for s in ((batch, n), (batch, n), (batch, na), (batch, na), (batch, na)))
    call("cdftb_hartree_split_f64", dens.data_ptr(), f2.data_ptr(), None, None, 0, n, batch, rho.data_ptr(),
         smooth.data_ptr(), stream)
    call("cdftb_quadrature_interpolate_f64", base.data_ptr(), w1d.data_ptr(), na, *shape, rho.data_ptr(), batch, n,
         at.data_ptr(), na, stream)
    call("cdftb_cusp_coefficients_f64", at.data_ptr(), nf2.data_ptr(), overlap.data_ptr(), na, batch, want.data_ptr(),
         stream)
    call("cdftb_cusp_coefficients_density_f64", dens.data_ptr(), f2.data_ptr(), base.data_ptr(), w1d.data_ptr(),
         nf2.data_ptr(), overlap.data_ptr(), na, *shape, batch, got.data_ptr(), stream)
    # 512 products of weights up to 0.7^3 and quotients up to 5.5, rounded at 1.1e-16 each, times |S^-1| f2 < 3
    torch.testing.assert_close(got, want, rtol=0.0, atol=512 * 0.35 * 5.5 * 3 * 8 * 1.1e-16)
