"""The power spectrum's mass assignment through tiles (enough particles a tile) and particle by
particle, at grids whose last tile is partial or wraps onto the first: against the Fourier oracle."""
import os
import sys

import numpy as np
import pytest

from cosmictiger_b200 import ics

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))


@pytest.mark.parametrize("n,grid,fold", [
    (16, 8, 1), (17, 8, 1), (33, 8, 1),  # one tile of 8^3 cells, the fewest particles for it; a warp's second turn
    (500, 4, 1), (3000, 10, 1), (20000, 24, 2), (20000, 20, 1), (2000, 16, 3),  # tiles that wrap, partial last tiles, folded boxes
    (60000, 16, 1),  # a tile in several work units
    (1, 8, 1), (15, 8, 1), (200, 24, 1),  # fewer than 16 particles a tile: particle by particle
])
def test_deposit_paths(n, grid, fold):
    import fourier_oracle as F

    import cosmictiger_b200 as ct

    rng = np.random.default_rng(n + grid)
    p = rng.random((3, n))
    p[:, : n // 2] = 0.01 + 0.05 * rng.random((3, n // 2))  # half in one corner
    x, y, z = (ics.to_fixed32(q) for q in p)
    ctx = ct.Context(order=7)
    box = ctx.box(n)
    box.upload(x, y, z, np.zeros((n, 3), np.float32), np.zeros(n, np.int8))
    k, P, e = box.power_spectrum(grid, 100.0, fold)
    box.close()
    ctx.close()
    ok, oP, oe = F.power_spectrum(x, y, z, grid, fold, 100.0)[:3]
    # A tile's weights are rounded once from double (2^-24 each, three and a product to a cell), the transform
    # adds about 2^-24 for each of its 3 log2(grid) steps, and the device fuses the product of a position
    # with the grid into the fraction, which the oracle rounds first (2^-25 grid cells): the squares differ by
    # 2 (4 + 3 log2(grid) + grid / 2) 2^-24 = 1.4e-6 to 3.5e-6; measured over six seeds at most 5.8e-7 in P
    # and 1.1e-6 in its scatter.  Particle by particle the weights are the reference's mixed form, whose
    # terms cancel from 405 / 120 down to a weight at the edge: 3.4 2^-24 each, raised by the window's
    # inverse; measured at most 7.8e-6 and 1.2e-5.
    tiles = n >= 16 * (-(-grid // 8)) ** 3
    tol = 2 * (4 + 3 * np.log2(grid) + grid / 2) * 2.0 ** -24 if tiles else 3e-5
    assert np.allclose(k, ok, rtol=1e-6)
    assert np.linalg.norm(P - oP) <= tol * np.linalg.norm(oP)
    assert np.linalg.norm(e - oe) <= 2 * tol * np.linalg.norm(oe) + 1e-30
