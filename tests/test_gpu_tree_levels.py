"""The tree build's level kernel at the sizes where its partition changes hands (one warp a node up
to 1,024 particles, tiles of 4,096 above) and where the node arrays run out in mid-build: order and
nodes bit-exact against the CPU oracle."""
import numpy as np
import pytest

from cosmictiger_b200 import ics

pytestmark = pytest.mark.gpu


def _state(n, kind):
    rng = np.random.default_rng(n)
    p = rng.random((3, n))
    if kind == "corner":  # deep, uneven splits: most particles in one corner
        p = p ** 4
    elif kind == "sorted":  # nothing to move on any level but the last
        p = np.sort(p, axis=1)
    x, y, z = (ics.to_fixed32(q) for q in p)
    return x, y, z, rng.standard_normal((n, 3)).astype(np.float32), rng.integers(0, 3, n).astype(np.int8)


@pytest.mark.parametrize("n,theta,bucket,kind", [
    (1, 0.7, 128, "random"), (31, 0.7, 8, "random"), (1024, 0.7, 64, "random"), (1025, 0.7, 64, "corner"), (4096, 0.55, 128, "random"),
    (4097, 0.55, 128, "corner"), (8193, 0.7, 1000, "sorted"), (70001, 0.7, 33, "corner"), (400003, 0.7, 128, "random"),
    (3000, 0.25, 128, "random"),  # small leaves by the opening angle: more nodes than the first arrays hold
])
def test_level_partition_edges(oracle, n, theta, bucket, kind):
    import cosmictiger_b200 as ct

    x, y, z, v, r = _state(n, kind)
    h = ics.softening(n, 0.02) if n > 100 else 1e-3
    ctx = ct.Context(order=7)
    box = ctx.box(n)
    box.upload(x, y, z, v, r)
    box.tree_create(theta, h, bucket)
    got, nodes = box.download(), box.tree()
    box.close()
    ctx.close()
    o = [q.copy() for q in (x, y, z, v, r)]
    ref = oracle.tree_build(*o, theta, h, bucket)
    for k, q in zip(("x", "y", "z", "v", "rung"), o):
        assert np.array_equal(got[k], q), k
    assert len(nodes) == len(ref)
    a, b = np.sort(nodes, order="key"), np.sort(ref, order="key")
    for k in ("key", "part_begin", "part_end", "leaf", "depth", "pos", "radius", "box_begin", "box_end"):
        assert np.array_equal(a[k], b[k]), k
