"""A tree build that stops for want of memory leaves every particle its own velocity and rung, and
the context's account of its device memory right.  The case outgrows the first node arrays, so that
among the budgets some end the build between two levels, others before or after them."""
import numpy as np
import pytest

from cosmictiger_b200 import ics

pytestmark = pytest.mark.gpu

N, THETA, H, BUCKET = 3000, 0.25, 1e-3, 128


def _state():
    rng = np.random.default_rng(7)
    x, y, z = (ics.to_fixed32(q) for q in rng.random((3, N)))
    # velocity and rung say which particle it is
    return x, y, z, np.stack([x, y, z], axis=1).astype(np.float32), (x % 11).astype(np.int8)


def _budgets():
    """The nodes of the tree, and budgets from what the particles take to what the build does."""
    import cosmictiger_b200 as ct

    ctx = ct.Context(order=7)
    box = ctx.box(N)
    box.upload(*_state())
    held = ctx.bytes_in_use()
    nodes = box.tree_create(THETA, H, BUCKET)
    after = ctx.bytes_in_use()
    box.close()
    ctx.close()
    assert nodes > 8192  # as many as the arrays of a first build hold
    return nodes, range(held, 2 * after - held, (after - held) // 24)


def test_failed_build_keeps_particles():
    import cosmictiger_b200 as ct

    x, y, z, v, r = _state()
    nodes, budgets = _budgets()
    moved = 0
    for budget in budgets:
        ctx = ct.Context(order=7, hbm_budget=budget)
        box = ctx.box(N)
        box.upload(x, y, z, v, r)
        failed = False
        try:
            assert box.tree_create(THETA, H, BUCKET) == nodes
        except ct.GravityError as e:
            assert "budget" in str(e)
            failed = True
        d = box.download()
        moved += failed and not np.array_equal(d["x"], x)
        for k, q in (("x", x), ("y", y), ("z", z)):
            assert np.array_equal(np.sort(d[k]), np.sort(q)), k
        assert np.array_equal(d["v"], np.stack([d["x"], d["y"], d["z"]], axis=1).astype(np.float32))
        assert np.array_equal(d["rung"], d["x"] % 11)
        box.close()
        ctx.close()
    assert moved  # some build stopped with particles moved
