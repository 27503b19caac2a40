"""An ensemble is kicked with all its particles active: a rung state set on it changes neither its
trees nor its forces (the build's and the kick's lists are sized by the active particles, and the
trees of an ensemble hold all of them)."""
import numpy as np
import pytest

from cosmictiger_b200 import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("begin", [1, 20000, 70000, 70001])
def test_rung_state_of_an_ensemble(begin):
    import cosmictiger_b200 as ct

    counts = [40000, 1, 30000]
    n, h, theta = sum(counts), 2e-3, 0.7
    rng = np.random.default_rng(3)
    x, y, z = (ics.to_fixed32(q) for q in rng.random((3, n)))
    v, r = rng.standard_normal((n, 3)).astype(np.float32), rng.integers(0, 3, n).astype(np.int8)
    ctx = ct.Context(order=7)
    out = []
    for start in (0, begin):
        box = ctx.ensemble(counts)
        box.upload(x, y, z, v, r)
        box.set_rung_state(start, [])
        box.tree_create(theta, h, 64)
        box.kick_ensemble(ct.KickParams.make(theta=theta, h=h, GM=1e-3, eta=ics.eta_default(), t0=1e-3))
        out.append((box.download(forces=True), box.counters()["leaves"], box.counters()["pp_pairs"]))
        box.close()
    ctx.close()
    a, b = out
    assert a[1:] == b[1:]
    for k in a[0]:
        assert np.array_equal(a[0][k], b[0][k]), k


def test_ensemble_without_particles():
    """Boxes that hold nothing return zeros, also when no box of the ensemble holds anything."""
    import cosmictiger_b200 as ct

    ctx = ct.Context(order=7)
    # an earlier ensemble of that size leaves its sums in the memory that the next one gets
    for counts in ([500, 700], [0, 0]):
        n = sum(counts)
        rng = np.random.default_rng(1)
        box = ctx.ensemble(counts)
        box.upload(*(ics.to_fixed32(q) for q in rng.random((3, n))), np.ones((n, 3), np.float32), np.full(n, 1, np.int8))
        box.tree_create(0.7, 1e-3, 32)
        got = box.kick_ensemble(ct.KickParams.make(theta=0.7, h=1e-3, GM=1e-3, eta=ics.eta_default(), t0=1e-3))
        box.close()
    ctx.close()
    for r in got:
        assert [getattr(r, f) for f, _ in r._fields_] == [0] * len(r._fields_)
