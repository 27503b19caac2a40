"""The upsweep's grouping of a level's nodes (1 to 32 a block, a ragged last block, nodes above and
below the 256 particles that one warp goes through) and its shift in four parts: centres, radii and
boxes bit-exact and multipoles to rounding against the CPU oracle."""
import numpy as np
import pytest

from cosmictiger_b200 import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bucket", [(9, 1), (700, 4), (20001, 8), (50000, 300), (250003, 4)])
def test_upsweep_groups(oracle, n, bucket):
    import cosmictiger_b200 as ct

    rng = np.random.default_rng(n)
    x, y, z = (ics.to_fixed32(q) for q in rng.random((3, n)) ** 1.5)
    v, r = np.zeros((n, 3), np.float32), np.zeros(n, np.int8)
    ctx = ct.Context(order=7)
    box = ctx.box(n)
    box.upload(x, y, z, v, r)
    box.tree_create(0.7, 1e-4, bucket)
    a = box.tree()
    box.close()
    ctx.close()
    b = oracle.tree_build(x.copy(), y.copy(), z.copy(), v, r, 0.7, 1e-4, bucket)
    a, b = np.sort(a, order="key"), np.sort(b, order="key")
    for k in ("key", "pos", "radius", "box_begin", "box_end"):
        assert np.array_equal(a[k], b[k]), k
    # a component is the rounded sum of two shifted ones of at most 37 terms in double from float
    # multipoles whose leaf sums may differ in the last bit: a few float roundings (2^-24) of the
    # largest term a level, which the mass and the component bound; 20 levels of half a rounding
    m_a, m_b = a["multi"], b["multi"]
    assert np.max(np.abs(m_a - m_b) / (np.abs(m_b) + 1e-6 * np.abs(m_b[:, :1]) + 1e-30)) < 20 * 2.0 ** -24 * 4
