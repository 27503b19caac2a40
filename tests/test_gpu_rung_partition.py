"""The rung partition at the edges of its warps' and blocks' shares (1,024 and 8,192 particles), with
none, all and some below the rung and from a start inside the box: order bit-exact against the CPU oracle."""
import numpy as np
import pytest

from cosmictiger_b200 import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 1023, 1025, 8191, 8192, 8193, 70001])
@pytest.mark.parametrize("below", [0.0, 0.03, 0.6, 1.0])
def test_rung_partition_edges(oracle, n, below):
    import cosmictiger_b200 as ct

    rng = np.random.default_rng(n)
    x, y, z = (ics.to_fixed32(q) for q in rng.random((3, n)))
    v = rng.standard_normal((n, 3)).astype(np.float32)
    r = np.where(rng.random(n) < below, 0, rng.integers(1, 4, n)).astype(np.int8)
    ctx = ct.Context(order=7)
    box = ctx.box(n)
    box.upload(x, y, z, v, r)
    o = [q.copy() for q in (x, y, z, v, r)]
    begin = 0
    for rung in (1, 2, 3):
        begin = oracle.sort_by_rung(*o, rung, begin)
        assert box.sort_by_rung(rung) == begin
    got = box.download()
    box.close()
    ctx.close()
    for k, q in zip(("x", "y", "z", "v", "rung"), o):
        assert np.array_equal(got[k], q), k
