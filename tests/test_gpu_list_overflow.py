"""A kick whose interaction lists outgrow their first room walks again with more: it gives the bits of
a kick that found the room, and the walks that did not fit cost little beside it (the kernels behind
such a walk have nothing to do)."""
import time

import numpy as np
import pytest

from cosmictiger_b200 import ics

pytestmark = pytest.mark.gpu


def test_kick_after_lists_that_did_not_fit():
    import cosmictiger_b200 as ct

    n, theta, h = 64 ** 3, 0.3, 1e-4
    rng = np.random.default_rng(1)
    x, y, z = (ics.to_fixed32(q) for q in rng.random((3, n)))
    v, r = np.zeros((n, 3), np.float32), np.zeros(n, np.int8)
    kp = ct.KickParams.make(theta=theta, h=h, GM=1e-9, eta=ics.eta_default(), t0=1e-6)
    extra = []
    for _ in range(3):
        ctx = ct.Context(order=7)
        ctx.box(200 * 10 ** 6).close()  # 5 GB in the context's pool: no allocation below goes to the CUDA driver
        box = ctx.box(n)
        times, launches, out = [], [], []
        for _ in range(2):
            box.upload(x, y, z, v, r)
            box.tree_create(theta, h, 64)
            l0, t0 = ctx.launches(), time.perf_counter()
            box.kick(kp)
            times.append(time.perf_counter() - t0)
            launches.append(ctx.launches() - l0)
            out.append(box.download(forces=True))
        box.close()
        ctx.close()
        assert launches[0] % launches[1] == 0 and launches[0] > launches[1]  # walked more than once
        for k in out[0]:
            assert np.array_equal(out[0][k], out[1][k]), k
        extra.append((times[0] - times[1]) / times[1] / (launches[0] // launches[1] - 1))
    # an attempt that does not fit takes its walk (0.6 of the kick's 11.8 ms) and empty launches: measured
    # 0.05 to 0.07 of a kick; with its lists worked off as far as they go it took 0.50 to 0.54
    assert min(extra) < 0.2, extra
