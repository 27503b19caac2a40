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
    (1, 8, 1), (500, 4, 1), (3000, 10, 1), (20000, 24, 2), (20000, 20, 1),  # tiles (at least 16 particles a tile of 8^3)
    (200, 24, 1),                                                          # particle by particle
    (60000, 16, 1),                                                        # a tile in several work units
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
    # float positions in cells carry 2^-24 of the folded grid and the float sums as much a weight:
    # 2^-23 grid fold in a weight's slope, times 216 of them in a mode at most
    tol = 216 * 2.0 ** -23 * grid * fold
    assert np.allclose(k, ok, rtol=1e-6)
    assert np.linalg.norm(P - oP) <= tol * np.linalg.norm(oP)
    assert np.linalg.norm(e - oe) <= 2 * tol * np.linalg.norm(oe) + 1e-30
