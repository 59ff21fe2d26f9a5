"""Host-fed runs through the pinned staging block: fresh values on every call, several schedules in turn, runs above and
below the size that is staged, f16 leaves beside f32 ones."""
import numpy as np
import pytest

from anneal_b200.device import Device
from anneal_b200.tensor import Tensor
from anneal_b200.uop import dtypes
from util import schedule

pytestmark = pytest.mark.gpu


def _product(n, seed, dtype=dtypes.float32):
    rng = np.random.default_rng(seed)
    a, b = (rng.standard_normal(n).astype(np.float32) for _ in range(2))
    x = Tensor.new_leaf((n,), dtype).set_data(a)
    y = Tensor.new_leaf((n,), dtype).set_data(b)
    return schedule([x.mul(y), x.add(y)])


@pytest.mark.parametrize("n", [1, 63, 64, 1000, (1 << 20) - 1, (1 << 20) + 64])     # two leaves of 4 MB each are the limit
def test_values_follow_the_call(cuda, oracle, n):
    items, ids, inputs = _product(n, 1)
    other = _product(n + 3, 2)
    for k in range(3):
        fed = {i: v * np.float32(k + 1) for i, v in inputs.items()}
        got = cuda.run(items, fed)
        between = cuda.run(other[0], other[2])
        want = oracle.run(items, fed)
        for i in ids:
            assert np.array_equal(got[i], want[i])
        w2 = oracle.run(other[0], other[2])
        for i in other[1]:
            assert np.array_equal(between[i], w2[i])


def test_half_leaves_and_many_schedules(cuda, oracle):
    """More schedules than are kept parsed, twice around."""
    all_ = [_product(100 + k, k, dtypes.float16 if k % 2 else dtypes.float32) for k in range(11)]
    for _ in range(2):
        for items, ids, inputs in all_:
            got, want = cuda.run(items, inputs), oracle.run(items, inputs)
            for i in ids:
                assert np.array_equal(got[i], want[i])


def test_runs_go_on_without_the_pinned_block():
    """The host may have no pinned memory left: the copies then go one by one, and the refusal is not reported by a later
    launch (an f16 output is converted by a kernel before its copy)."""
    dev = Device(0)
    try:
        plain, half = _product(1000, 3), _product(1000, 4, dtypes.float16)
        before = [dev.run(items, inputs) for items, _, inputs in (plain, half)]
        dev._check(dev.L.anl_inject_host_stage_failure(dev.h, 1))
        for _ in range(2):
            for (items, ids, inputs), want in zip((plain, half), before):
                got = dev.run(items, inputs)
                for i in ids:
                    assert np.array_equal(got[i], want[i])
                got = dev.replay(items, inputs)
                for i in ids:
                    assert np.array_equal(got[i], want[i])
        dev._check(dev.L.anl_inject_host_stage_failure(dev.h, 0))
        got = dev.run(plain[0], plain[2])
        assert all(np.array_equal(got[i], before[0][i]) for i in plain[1])
    finally:
        dev.close()
