"""Initial conditions of two grids at once, from two host threads with a context each: the
interpolation's shared memory depends on the grid, and what one thread's launches may use must not
follow from the other's grid."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_grids_from_two_threads():
    import cosmictiger_b200 as ct

    k = np.exp(np.linspace(np.log(1e-5), np.log(1e3), 400)).astype(np.float32)
    P = (2e4 * (k / 0.02) / (1 + (k / 0.02) ** 2) ** 1.8).astype(np.float32)
    want, got, errors = {}, {}, []

    def runs(n, times):
        try:
            ctx = ct.Context(order=7)
            box = ctx.box(n ** 3)
            out = []
            for _ in range(times):
                box.initialize(n, 100.0, k, P)
                d = box.download()
                out.append(np.concatenate([d["x"], d["y"], d["z"], d["v"].view(np.uint32).ravel()]))
            box.close()
            ctx.close()
            return out
        except Exception as e:  # (a thread's exception would be lost)
            errors.append(e)
            return []

    for n in (64, 16):
        want[n] = runs(n, 1)
    threads = [threading.Thread(target=lambda n=n, t=t: got.__setitem__(n, runs(n, t))) for n, t in ((64, 100), (16, 400))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    for n in (64, 16):
        assert all(np.array_equal(want[n][0], g) for g in got[n]), n
