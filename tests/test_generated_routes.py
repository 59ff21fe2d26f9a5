"""Which form a generated kernel takes, by the notes of the lowering (no GPU), and its values against the oracle."""
import numpy as np
import pytest

from anneal_b200 import workloads as W
from anneal_b200.device import lower
from anneal_b200.tensor import Tensor
from util import schedule


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
