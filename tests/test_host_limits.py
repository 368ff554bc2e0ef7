"""The library's host code where a device or a system runs short, on a CUDA runtime that runs nothing (fake_runtime.py): what
it launches, allocates and reports, not what the kernels compute."""
import numpy as np
import pytest

import fake_runtime
from fake_runtime import LAUNCHES


@pytest.fixture
def fake():
    gsb, dev = fake_runtime.load()
    dev.fake_set_capacity(1 << 40)
    dev.fake_reset()
    yield gsb, dev
    dev.fake_set_capacity(1 << 40)


def plan(n):
    import workloads
    return workloads.matching_instance(n, n, 11, 8, 20000)["plan"]


@pytest.mark.parametrize("prec", [128, 64])
@pytest.mark.parametrize("n,prefix", [(16, 0), (36, 0), (36, 20)])
def test_launches_per_item(fake, n, prefix, prec):
    """Every mode's count is what a call of one item queues (beside the item index, and the least conditional of a
    'prob'): a whole item of a narrow plan is one launch, without an index."""
    gsb, dev = fake
    with gsb.Engine.from_text(plan(n), precision=prec) as eng:
        eng.set_hybrid_prefix(prefix)
        line = np.zeros((1, eng.ns), np.int8)
        index = 0 if n == 16 else 1

        def queued(call):
            before = dev.fake_count(LAUNCHES)
            call()
            return dev.fake_count(LAUNCHES) - before - index
        assert queued(lambda: eng.hybrid(line, 1)) == eng.launches_per_item(2)
        assert queued(lambda: eng.sample(1, 1)) == eng.launches_per_item(1)
        assert queued(lambda: eng.chain(line)) == eng.launches_per_item(0)
        if n == 16:
            assert [eng.launches_per_item(m) for m in range(3)] == [1, 1, 1]
        else:   # a hybrid item without a prefix: a norm and a write pass per wide step, as unfused sampling
            eng.set_hybrid_prefix(0)
            hybrid = eng.launches_per_item(2)
            eng.set_fusion(1)
            assert hybrid == eng.launches_per_item(1) == eng.launches_per_item(2)
