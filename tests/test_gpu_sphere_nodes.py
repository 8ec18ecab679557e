"""The quadrature spheres' nodes made on the device against the oracle's rule."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import geometry as ogeometry

pytestmark = pytest.mark.gpu


# the smallest sphere (polar order 4 throughout), ordinary ones, the widest; one to three spheres in a launch
@pytest.mark.parametrize("radii,h,node_spacing", [((0.9,), 0.4, 1.0), ((2.87, 1.3), 0.25, 0.7), ((1.15, 0.61, 0.3), 0.1, 0.7)])
def test_nodes_match_the_rule(pkg, cuda, radii, h, node_spacing):
    centres = np.array([[0.0, 0.0, 0.0], [0.31, -0.2, 1.7], [-4.0, 0.11, 3.0]])[:len(radii)]
    shells = [pkg.geometry.sphere_shells(r, h, 6, node_spacing) for r in radii]
    points, base, owner = (t.cpu().numpy() for t in pkg.geometry.sphere_nodes(centres, shells, cuda))
    at = 0
    for i, (centre, r) in enumerate(zip(centres, radii)):
        p, w = ogeometry.sphere_rule(centre, r, h, 6, node_spacing)[:2]
        # the same few products, each within an ulp of the oracle's: 1e-14 of the sphere's extent
        np.testing.assert_allclose(points[at:at + len(p)], p, rtol=0, atol=1e-14 * (r + np.abs(centre).max()))
        np.testing.assert_allclose(base[at:at + len(p)], w, rtol=1e-13)
        assert (owner[at:at + len(p)] == i).all()
        at += len(p)
    assert at == len(points)
