"""The node orders of the interaction kernels for a tree that one block orders, that two do (one node
over, or a few) and that several do: a box's forces are the same bits alone and beside its copies."""
import numpy as np
import pytest

from cosmictiger_b200 import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bucket,nodes", [(4, 200, (1, 4096)), (16, 6, (4000, 4096)), (11, 1, (4097, 4200)), (16, 1, (8193, 12288))])
def test_orders_hold_every_node(n, bucket, nodes):
    import cosmictiger_b200 as ct

    x, y, z, v, _ = ics.zeldovich_lattice(n, index=-1.5, rms_spacing=0.05, seed=n)
    N = len(x)
    ctx = ct.Context(order=7)

    def kick(copies):
        b = ctx.ensemble([N] * copies) if copies > 1 else ctx.box(N)
        b.upload(np.tile(x, copies), np.tile(y, copies), np.tile(z, copies), np.tile(v, (copies, 1)), np.zeros(copies * N, np.int8))
        b.tree_create(0.6, 2e-3, bucket)
        nn = len(b.tree())
        kp = ct.KickParams.make(theta=0.6, h=2e-3, GM=1e-3, eta=ics.eta_default(), t0=1e-3)
        b.kick_ensemble(kp) if copies > 1 else b.kick(kp)
        out = b.download(forces=True)
        b.close()
        return out, nn

    one, nn = kick(1)
    assert nodes[0] <= nn <= nodes[1], nn
    three, nn3 = kick(3)
    assert nn3 == 3 * nn
    assert np.all(np.isfinite(one["pot"])) and np.all(one["pot"] != 0)
    for k in ("gx", "gy", "gz", "pot", "rung"):
        for c in range(3):
            assert np.array_equal(three[k][c * N:(c + 1) * N], one[k]), (k, c)
    ctx.close()
