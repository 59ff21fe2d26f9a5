"""Row chains and shared memory: members that run in one launch must not write what another row still reads."""
import numpy as np
import pytest

import util_chains as C
from anneal_b200.device import lower_chain
from anneal_b200.tensor import Tensor
from util import rel_err


def _refused(items, first, count):
    with pytest.raises(Exception, match="another row may still read"):
        lower_chain(items, first, count)


@pytest.mark.parametrize("n", [64, 2048])
def test_value_a_row_over_a_column_vector(n):
    """As many rows as columns: a value a row has the count and type of the vector that every row reads."""
    items, _, _ = C.plan(C.column_vector(n))
    assert C.slots(items) == [0, 1, 0, 1, -1]
    for first, count in ((1, 2), (1, 3), (1, 4)):
        _refused(items, first, count)
    # a value a row over one that the row itself reads from memory: refused as well, as every thread reads it
    _refused(items, 2, 2)
    assert "2 stages" in lower_chain(items, 3, 2)["note"]


def test_whole_row_over_values():
    items, _, _ = C.plan(C.row_over_value(70, 300))
    assert C.slots(items) == [0, 1, 0, -1]
    _refused(items, 0, 3)
    _refused(items, 1, 2)
    assert "2 stages" in lower_chain(items, 0, 2)["note"]


def test_whole_row_over_its_own_operand_stays_a_chain():
    items, _, _ = C.plan(C.row_over_operand(70, 300))
    assert C.slots(items) == [0, 1, 0, -1]
    assert "2 stages" in lower_chain(items, 1, 2)["note"]


def test_vectors_alone_are_no_chain():
    """Kernels of one value a row with nothing to run along it are elementwise kernels, a thread a value."""
    leaf = lambda n: Tensor.new_leaf((n,)).set_data(np.ones(n, np.float32))
    items, _, _ = C.plan([v.mul(v) for v in (leaf(1000), leaf(1000), leaf(1000))])
    with pytest.raises(Exception, match="runs along the row"):
        lower_chain(items, 0, 3)
    x, v = Tensor.new_leaf((300, 40)).set_data(np.ones(12000, np.float32)), leaf(300)
    items, _, _ = C.plan([x.sum((1,)).mul(v), v.mul(v)])
    assert "2 stages" in lower_chain(items, 0, 2)["note"]


@pytest.mark.gpu
@pytest.mark.parametrize("make", [lambda: C.column_vector(64), lambda: C.column_vector(2048), lambda: C.row_over_value(70, 300),
                                  lambda: C.row_over_value(2048, 512), lambda: C.row_over_operand(70, 300), lambda: C.row_over_operand(1500, 600)],
                         ids=["column 64", "column 2048", "value 70", "value 2048", "operand 70", "operand 1500"])
def test_values(cuda, oracle, make):
    """Against the oracle: maxima are exact, and the contraction's sum of cols f32 products rounds by 2^-24 a term, the 3 x TF32 form's
    bound of 1e-5 over it."""
    items, ids, inputs = C.plan(make())
    got, want = cuda.run(items, inputs)[ids[0]], oracle.run(items, inputs)[ids[0]]
    assert rel_err(got, want) <= 1e-5
    assert np.array_equal(cuda.run(items, inputs)[ids[0]], got)
