"""Every transform length of the register kernels along every axis, and the solve's error against 80-bit transforms."""

from __future__ import annotations

import numpy as np
import pytest
import scipy.fft
import torch

from oracle.operators import CoulombCutoffPoisson

pytestmark = pytest.mark.gpu

#: the lengths with a factor pair (fourstep_pair in csrc/poisson.cu)
LENGTHS = (36, 48, 64, 72, 80, 90, 96, 100, 108, 120, 128, 135, 144, 150, 160, 162, 180, 192, 200, 216, 225, 240, 256, 270,
           288, 300, 320)


class _Grid:
    def __init__(self, shape, spacing):
        self.shape, self.spacing = shape, spacing


def _solve(pkg, shape, spacing, pad, rho):
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    grid = pkg.UniformGrid(shape, spacing, (0.0, 0.0, 0.0), device="cuda:0")
    solver = pkg.CoulombCutoffPoisson(grid, pad_factor=pad, max_batch=rho.shape[0])
    return solver.solve_batch(torch.from_numpy(rho).cuda()).cpu().numpy()


@pytest.mark.parametrize("length", LENGTHS)
def test_length_along_every_axis(pkg, length):
    """The largest and the smallest box a length takes, two systems. Transforms of up to 2^20 points are off by about
    20 roundings of 1.1e-16: 1e-14 of the largest value."""
    below = max((v for v in LENGTHS if v < length), default=0)
    for n in (below // 2 + 1, (length + 1) // 2):
        for axis in range(3):
            shape = [5, 3, 4]
            shape[axis] = n
            rho = np.random.default_rng(n + axis).standard_normal((2, int(np.prod(shape))))
            oracle = CoulombCutoffPoisson(_Grid(tuple(shape), 0.3), 2.0)
            want = np.stack([oracle.solve(r) for r in rho])
            np.testing.assert_allclose(_solve(pkg, tuple(shape), 0.3, 2.0, rho), want, rtol=0,
                                       atol=1e-14 * np.abs(want).max())


@pytest.mark.parametrize("n,length,pad", [(33, 72, 2.5), (65, 135, 2.5), (65, 135, 2.0)])
def test_error_against_extended_precision(pkg, n, length, pad):
    """The zero-padded definition with K, transforms and products in 80 bits.

    In doubles, two transforms along three axes are some 60 roundings one after the other; of the size 0.3 units each
    (1.1e-16, as a root of the mean square) they add up to 2.3 units in the mean square. 3e-16 is 2.7 units: a table
    of K carried over in plain doubles, or roots of unity from double angles, would not stay below it.
    """
    h = 0.25
    x = (np.arange(n) - n // 2) * h
    r2 = x[:, None, None] ** 2 + x[None, :, None] ** 2 + x[None, None, :] ** 2
    rho = 0.5 * np.exp(-0.5 * r2) + 0.05 * np.random.default_rng(n).standard_normal((n, n, n))
    padded = CoulombCutoffPoisson(_Grid((n, n, n), h), pad).padded_shape[0]
    wide = np.longdouble
    pi = wide("3.14159265358979323846264338327950288")
    index = np.arange(padded)
    k = 2 * pi * np.where(2 * index < padded, index, index - padded).astype(wide) / (wide(padded) * wide(h))
    radius = wide(0.5) * padded * wide(h)
    g2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :padded // 2 + 1] ** 2
    g2[0, 0, 0] = 1
    kernel = 4 * pi * (1 - np.cos(np.sqrt(g2) * radius)) / g2
    kernel[0, 0, 0] = 2 * pi * radius ** 2
    spectrum = scipy.fft.rfftn(rho.astype(wide), s=(padded,) * 3, workers=8) * kernel
    want = scipy.fft.irfftn(spectrum, s=(padded,) * 3, workers=8)[:n, :n, :n]
    assert want.dtype == wide and padded >= length
    got = _solve(pkg, (n, n, n), h, pad, rho.reshape(1, -1)).reshape(n, n, n)
    error = float(np.sqrt(((got - want) ** 2).sum() / (want ** 2).sum()))
    assert error < 3e-16
