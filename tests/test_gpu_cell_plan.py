"""The cell plan of L^T checks what it is built from, and a lift what plan it is given."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _build_geometry(pkg):
    grid = pkg.UniformGrid((19, 18, 21), 0.45, (-4.05, -3.9, -4.6), device="cuda:0")
    return pkg.build_cusp_geometry(grid, (2.0,), ((0.05, -0.02, 0.1),))


@pytest.fixture(scope="module")
def parts(pkg):
    """``(quadrature, keys, order, box)`` as the quadrature's own plan is built from."""
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    q = _build_geometry(pkg).quadrature
    b = q.base[q.group_nodes.long()].long()
    keys = (b[:, 0] * q.grid.shape[1] + b[:, 1]) * q.grid.shape[2] + b[:, 2]
    return q, keys, q.group_nodes.clone(), q._cell_box.copy()


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _plan(pkg, q, keys, order, box):
    lib = pkg._lib.library()
    nbytes = lib.cdftb_cell_plan_bytes(q.n_nodes, *q.grid.shape, box.ctypes.data)
    plan = torch.empty(nbytes, dtype=torch.uint8, device="cuda:0")
    pkg._lib.call("cdftb_cell_plan_build", q.base.data_ptr(), q.w1d.data_ptr(), order.data_ptr(), keys.data_ptr(),
                  q.n_nodes, *q.grid.shape, box.ctypes.data, plan.data_ptr(), nbytes, _stream())
    return plan


def _lift(pkg, q, plan, box, nf, m=None):
    m = m or q.n_nodes
    n = q.grid.n_points
    x = torch.ones((nf, q.n_nodes), dtype=torch.float64, device="cuda:0")
    out = torch.empty((nf, n), dtype=torch.float64, device="cuda:0")
    nbytes = pkg._lib.library().cdftb_lift_cells_scratch_bytes(m, *q.grid.shape, box.ctypes.data, nf)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda:0")
    pkg._lib.call("cdftb_quadrature_lift_cells_f64", plan.data_ptr(), plan.numel(), m, *q.grid.shape, box.ctypes.data,
                  x.data_ptr(), nf, q.n_nodes, out.data_ptr(), n, scratch.data_ptr(), nbytes, _stream())
    return out


def _bad(plan):
    return int(plan[:8].view(torch.int64))


@pytest.mark.parametrize("nf", [2, 9])
def test_sound_plan(pkg, parts, nf):
    q, keys, order, box = parts
    plan = _plan(pkg, q, keys, order, box)
    assert _bad(plan) == 0
    x = torch.ones((nf, q.n_nodes), dtype=torch.float64, device="cuda:0")
    assert torch.equal(_lift(pkg, q, plan, box, nf), q._lift_raw(x, nf))


def _reversed(keys, order, box, m, cells):
    return keys.flip(0).contiguous(), order.flip(0).contiguous(), box


def _one_wrong_key(keys, order, box, m, cells):
    keys = keys.clone()
    keys[m // 2] += 1
    return keys, order, box


def _no_such_node(keys, order, box, m, cells):
    order = order.clone()
    order[0], order[m - 1] = -1, m
    return keys, order, box


def _small_box(axis, side):
    def change(keys, order, box, m, cells):
        box = np.concatenate([cells.min(axis=0), cells.max(axis=0)]).astype(np.int32)  # the cells that hold nodes
        box[axis + 3 * side] += -1 if side else 1
        return keys, order, box
    return change


@pytest.mark.parametrize("nf", [2, 9])
@pytest.mark.parametrize("change", [_reversed, _one_wrong_key, _no_such_node, *(_small_box(a, s) for a in range(3) for s in (0, 1))])
def test_unsound_plan_lifts_nan(pkg, parts, nf, change):
    q, keys, order, box = parts
    keys, order, box = change(keys, order, box, q.n_nodes, q.base.cpu().numpy())
    plan = _plan(pkg, q, keys, order, box)
    assert _bad(plan) > 0
    out = _lift(pkg, q, plan, box, nf)
    # NaN at the points the box reaches, zero elsewhere
    assert bool(torch.isnan(out).any()) and bool((torch.isnan(out) | (out == 0.0)).all())
    assert bool(torch.isnan(out).reshape(nf, *q.grid.shape)[:, box[0]:box[3] + 1, box[1]:box[4] + 1, box[2]:box[5] + 1].all())


@pytest.mark.parametrize("nf", [2, 9])
def test_plan_of_another_call_lifts_nan(pkg, parts, nf):
    q, keys, order, box = parts
    plan = _plan(pkg, q, keys, order, box)
    other = box.copy()
    other[:3] += 1
    assert bool(torch.isnan(_lift(pkg, q, plan, other, nf)).any())
    assert bool(torch.isnan(_lift(pkg, q, plan, box, nf, m=q.n_nodes - 1)).any())


def test_quadrature_refuses_a_box_that_misses_nodes(pkg, parts, monkeypatch):
    call = pkg.geometry.call

    def smaller(name, *args):
        if name == "cdftb_cell_plan_build":
            box = parts[3].copy()
            box[0] += 2
            return call(name, *args[:8], box.ctypes.data, *args[9:])
        return call(name, *args)

    monkeypatch.setattr(pkg.geometry, "call", smaller)
    with pytest.raises(ValueError, match="outside the spheres' box"):
        _build_geometry(pkg)
