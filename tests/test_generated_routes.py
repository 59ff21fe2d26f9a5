"""Which form a generated kernel takes, by the notes of the lowering (no GPU), and its values against the oracle."""
import numpy as np
import pytest

from anneal_b200 import workloads as W
from anneal_b200.device import lower
from anneal_b200.tensor import Tensor
from util import rel_err, schedule


def _leaf(shape, seed):
    return Tensor.new_leaf(shape).set_data(W.normal(71, seed, int(np.prod(shape))))


def _pieces(shape, axis, count, terms=1):
    """`count` slices side by side along `axis`, each the sum of `terms` leaves: a sum of padded pieces."""
    out = None
    for k in range(count * terms):
        at = k // terms
        pad = [(0, 0)] * len(shape)
        pad[axis] = (at * shape[axis], (count - 1 - at) * shape[axis])
        piece = _leaf(shape, k).pad(pad)
        out = piece if out is None else out.add(piece)
    return [out]


# few pieces; pieces along the last range, where neighbouring threads are in different ones; four elements behind the range |
# many pieces; a convolution's patches (several terms a channel); eight elements behind the range
CASES = [((64, 32), 1, 4, 1, False), ((100, 1, 8), 1, 8, 1, False), ((500, 2), 1, 16, 1, False), ((32, 1, 4), 1, 8, 4, False),
         ((9, 1, 8), 1, 16, 1, True), ((3, 1, 49), 1, 4, 9, True), ((1, 300), 0, 24, 1, True)]


@pytest.mark.parametrize("shape,axis,count,terms,switch", CASES)
def test_gathers_are_enumerated_where_it_pays(shape, axis, count, terms, switch):
    items, _, _ = schedule(_pieces(shape, axis, count, terms))
    assert len(items) == 1
    assert ("switch over" in lower(items, 0)["note"]) == switch


@pytest.mark.gpu
@pytest.mark.parametrize("shape,axis,count,terms,switch", CASES)
def test_gather_values(cuda, oracle, shape, axis, count, terms, switch):
    items, ids, inputs = schedule(_pieces(shape, axis, count, terms))
    assert np.array_equal(cuda.run(items, inputs)[ids[0]], oracle.run(items, inputs)[ids[0]])


# more than 64 trips a lane and fewer than 256 blocks: 128 x 128 and 256 x 256 in all; rows summed away with few and many columns
@pytest.mark.parametrize("shape,axes,split", [((128, 128), [0, 1], False), ((256, 256), [0, 1], True), ((1024, 1024), [0], False), ((256, 1024), [0], False),
                                              ((8192, 1000), [0], True), ((8192, 8192), [0], False), ((100, 8192), [1], False), ((8, 100000), [1], True)])
def test_reductions_are_split_where_it_pays(shape, axes, split):
    items, _, _ = schedule([Tensor.new_leaf(shape).sum(axes)])
    assert ("split reduce" in lower(items, 0)["note"]) == split


# 31, 32 and 33 trips a lane; the sweep of a row-broadcast kernel behind its reduction
@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(992, 40), (1024, 40), (1056, 40), (65, 257), (1, 20001)])
def test_loop_values(cuda, oracle, rows, cols):
    x = _leaf((rows, cols), 5)
    total = x.mul(x).sum((1,)).reshape((rows, 1)).expand((rows, cols))
    for target in (x.sum((0,)), x.mul(total)):
        items, ids, inputs = schedule([target])
        got, want = cuda.run(items, inputs)[ids[0]], oracle.run(items, inputs)[ids[0]]
        terms = rows if target.shape == (cols,) else cols
        # f32 sums of `terms` values in two orders: a random walk of sqrt(terms) roundings of 2^-24 each, four of them for the spread
        assert rel_err(got, want) <= 4 * np.sqrt(terms) * 2.0 ** -24 + 1e-6
