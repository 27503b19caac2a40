"""The particle-particle kernel that takes whole leaves against the one that takes tiles: an ensemble
has leaves enough for the first, each of its boxes alone only for the second, and the results are
the same bits.  The boxes hold leaves of one particle up to several groups of 128."""
import numpy as np
import pytest

from cosmictiger_b200 import ics

pytestmark = pytest.mark.gpu



def _line():
    """Leaves from which a warp takes whole ones: two a resident warp, 24 warps a multiprocessor."""
    import torch

    return 2 * 24 * torch.cuda.get_device_properties(0).multi_processor_count


def _leaves(tree, boxes):
    """All leaves of the trees of so many boxes, empty ones too, as the rule counts them."""
    n = (len(tree) + boxes) // 2
    assert n == np.count_nonzero(tree["leaf"])
    return n


def _box(i):
    rng = np.random.default_rng(100 + i)
    n = 12 + i % 4
    x, y, z, v, _ = ics.zeldovich_lattice(n, index=-1.5, rms_spacing=0.4, seed=i)
    m = 40 * i  # a clump: leaves filled up to the bucket
    p = (np.array([[0.3], [0.7], [0.2]]) + 0.004 * rng.standard_normal((3, m))) % 1.0
    c = [ics.to_fixed32(q) for q in p]
    x, y, z = (np.concatenate([a, b]) for a, b in zip((x, y, z), c))
    v = np.concatenate([v, np.zeros((m, 3), np.float32)])
    return x, y, z, np.ascontiguousarray(v), np.zeros(len(x), np.int8)


@pytest.mark.parametrize("bucket,stage,compensated", [(128, 128, True), (300, 128, True), (17, 64, True), (128, 256, False)])
def test_leaf_and_tile_kernels_agree(bucket, stage, compensated):
    import cosmictiger_b200 as ct

    boxes = [_box(i) for i in range(16)]
    h, theta = 2e-3, 0.5

    def kick(ctx, parts, counts):
        b = ctx.ensemble(counts) if len(counts) > 1 else ctx.box(counts[0])
        b.upload(*parts)
        b.tree_create(theta, h, bucket)
        kp = ct.KickParams.make(theta=theta, h=h, GM=1e-3, eta=ics.eta_default(), t0=1e-3)
        b.kick_ensemble(kp) if len(counts) > 1 else b.kick(kp)
        out, leaves = b.download(forces=True), _leaves(b.tree(), len(counts))
        pairs = b.counters()["pp_pairs"]
        b.close()
        return out, leaves, pairs

    ctx = ct.Context(order=7)
    ctx.set_tuning(p2p_stage=stage)
    ctx.set_compensated(compensated)
    whole, leaves, pairs = kick(ctx, [np.concatenate(q) for q in zip(*boxes)], [len(b[0]) for b in boxes])
    assert leaves >= _line()  # whole leaves
    at, total = 0, 0.0
    for b in boxes:
        one, few, p = kick(ctx, b, [len(b[0])])
        assert few < _line()  # tiles
        total += p
        for k in ("x", "v", "rung", "gx", "gy", "gz", "pot"):
            assert np.array_equal(whole[k][at:at + len(b[0])], one[k]), k
        at += len(b[0])
    assert pairs == total
    ctx.close()
