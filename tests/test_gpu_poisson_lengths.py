"""The Poisson solve at the edges of its transform lengths against the oracle's padded FFT."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle.operators import CoulombCutoffPoisson

pytestmark = pytest.mark.gpu

#: shape, pad factor, batch: box sizes at, one under and one over a length's limit (2n - 1 = 135, 143, 161, 191),
#: an odd number of z lines, lengths the definition already has, and an axis beyond the register kernels
CASES = [((68, 5, 68), 2.5, 1), ((72, 73, 9), 2.0, 2), ((67, 68, 69), 2.5, 1), ((81, 13, 96), 2.5, 3), ((1, 7, 3), 2.5, 5),
         ((18, 19, 24), 2.0, 1), ((60, 30, 25), 2.0, 1), ((165, 3, 170), 2.0, 1)]


class _Grid:
    def __init__(self, shape, spacing):
        self.shape, self.spacing = shape, spacing


@pytest.mark.parametrize("shape,pad,batch", CASES)
def test_matches_the_padded_transform(pkg, shape, pad, batch):
    """Transforms of up to 2^24 points are off by about 24 roundings of 1.1e-16: 1e-14 of the largest value."""
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    h = 0.3
    rng = np.random.default_rng(sum(shape))
    rho = rng.standard_normal((batch, int(np.prod(shape))))
    grid = pkg.UniformGrid(shape, h, (0.0, 0.0, 0.0), device="cuda:0")
    got = pkg.CoulombCutoffPoisson(grid, pad_factor=pad, max_batch=batch).solve_batch(torch.from_numpy(rho).cuda())
    oracle = CoulombCutoffPoisson(_Grid(shape, h), pad)
    want = np.stack([oracle.solve(r) for r in rho])
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=0, atol=1e-14 * np.abs(want).max())
