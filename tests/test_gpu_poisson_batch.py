"""The Poisson solves of a batch are independent: each system's potential is that of its own solve, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

#: odd and even counts of z lines (nx ny), of whole and partial blocks of 16, and a z axis beyond the register kernels
SHAPES = [(1, 1, 18), (3, 5, 7), (4, 4, 9), (9, 5, 24), (17, 17, 17), (33, 33, 33), (3, 5, 170)]


@pytest.mark.parametrize("shape", SHAPES)
def test_systems_of_a_batch_do_not_touch_each_other(pkg, shape):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    n = int(np.prod(shape))
    scales = (1.0, 1e10, 1e-10, 1.0, 1e12, 1.0, 1.0)
    rho = np.random.default_rng(n).standard_normal((len(scales), n)) * np.array(scales)[:, None]
    rho[3, [0, n // 2, n - 1]] = np.nan  # on the first and the last z line too
    rho[5, n - 1] = np.inf
    grid = pkg.UniformGrid(shape, 0.3, (0.0, 0.0, 0.0), device="cuda:0")
    poisson = pkg.CoulombCutoffPoisson(grid, pad_factor=2.0, max_batch=len(scales))
    densities = torch.from_numpy(rho).cuda()
    together = poisson.solve_batch(densities)
    for i in range(len(scales)):
        alone = poisson.solve_batch(densities[i:i + 1])[0]
        if i in (3, 5):
            assert not bool(torch.isfinite(together[i]).any())
        else:
            assert bool(torch.isfinite(together[i]).all())
            assert torch.equal(together[i], alone)
