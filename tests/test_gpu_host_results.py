"""Host results of `run`: arrays of the caller's own, one per final output, whatever is placed and whatever is symbolic."""
import numpy as np
import pytest

from anneal_b200 import uop as U, workloads as W
from anneal_b200.tensor import Tensor
from util import schedule

pytestmark = pytest.mark.gpu


# leaves below, at and above the piece that is sent on while the next is staged; a scalar; one element
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 17), (256, 128), (257, 128), (700, 1000), (1500, 1600)])
def test_results_are_independent(cuda, rows, cols):
    a, b, c = (Tensor.new_leaf((rows, cols)).set_data(W.normal(91, k, rows * cols)) for k in (1, 2, 3))
    items, ids, inputs = schedule([a.add(b), b.mul(c), a.mul(c).sum()])
    first = cuda.run(items, inputs)
    kept = {k: v.copy() for k, v in first.items()}
    mine = np.full(rows * cols, np.float32(7))
    other = {t.node.idx: inputs[t.node.idx] + np.float32(1) for t in (a, b, c)}
    second = cuda.run(items, other, placed={ids[0]: mine})
    assert second[ids[0]] is mine and set(first) == set(second) == set(ids)
    va, vb, vc = (inputs[t.node.idx] for t in (a, b, c))
    assert np.array_equal(first[ids[0]], va + vb) and np.array_equal(first[ids[1]], vb * vc) and first[ids[2]].shape == (1,)
    assert np.array_equal(mine, (va + np.float32(1)) + (vb + np.float32(1)))
    for k in ids:
        assert np.array_equal(first[k], kept[k]) and first[k].flags.writeable and first[k].dtype == np.float32
        assert not np.shares_memory(first[k], second[k])


def test_symbolic_results(cuda):
    var = U.Var("n", 1, 64)
    x = Tensor.new_symbolic_batch_input(var, (8,))
    w = Tensor.new_leaf((8,)).set_data(W.normal(92, 1, 8))
    out = x.mul(x)
    items, ids, inputs = schedule([out, w.add(w)])
    for n in (5, 64, 1):
        v = W.normal(92, n, n * 8)
        got = cuda.run(items, {**inputs, x.node.idx: v}, binding={"n": n})
        assert np.array_equal(got[ids[0]], v * v) and np.array_equal(got[ids[1]], inputs[w.node.idx] * 2)
