"""The context's account of its device memory over tree builds that stop for want of memory: it does
not grow with each of them, and ends where it was once the box is closed."""
import pytest

from tests.test_gpu_tree_budget import BUCKET, H, N, THETA, _budgets, _state

pytestmark = pytest.mark.gpu


def test_failed_builds_keep_the_account():
    import cosmictiger_b200 as ct

    nodes, budgets = _budgets()
    stopped = 0
    for budget in budgets:
        ctx = ct.Context(order=7, hbm_budget=budget)
        left = []
        for _ in range(2):
            box = ctx.box(N)
            box.upload(*_state())
            used = []
            for _ in range(4):
                try:
                    assert box.tree_create(THETA, H, BUCKET) == nodes
                except ct.GravityError:
                    stopped += 1
                used.append(ctx.bytes_in_use())
            assert used[1:] == used[:-1]
            box.close()
            left.append(ctx.bytes_in_use())  # the context's scratch
        assert left[0] == left[1]
        ctx.close()
    assert stopped
