"""Row chains whose rows sit in registers: one thread, one warp or one block a row, rows that end inside a lane's
chunk, blocks that walk the rows while the next one is on its way, and the longest row that still fits."""
import numpy as np
import pytest

from anneal_b200 import workloads as W
from anneal_b200.tensor import Tensor
from util import rel_err, schedule

pytestmark = pytest.mark.gpu


def tol(cols):
    """Three sums over a row follow one another (the exponentials, the weighted gradient, its total), each rounding by 2^-24
    a term in an order of its own: a random walk of sqrt(cols) such steps each, four of those for the spread, and
    a few single roundings."""
    return 4 * np.sqrt(cols) * 2.0 ** -24 + 5e-6


def _softmax(cuda, oracle, rows, cols, mask=False):
    s = W.SoftmaxFwdBwd(rows, cols)
    ts, _ = s.graph()
    items, ids, inputs = schedule(ts)
    if mask:                                   # a masked position holds the type's lowest value
        for v in inputs.values():
            if v.size == rows * cols and np.array_equal(v, s.x.reshape(-1)):
                v = v.reshape(rows, cols)
                v[:, 1::3] = np.finfo(np.float32).min
    before = cuda.stats()["kernels_launched"]
    got = cuda.run(items, inputs)[ids[0]]
    launches = cuda.stats()["kernels_launched"] - before
    want = oracle.run(items, inputs)[ids[0]]
    assert np.isfinite(want).all()
    assert rel_err(got, want) <= tol(cols), (rows, cols, rel_err(got, want))
    again = cuda.run(items, inputs)[ids[0]]
    assert np.array_equal(got, again)
    return launches


# 16 | 17: a thread or a warp a row; 129 rows: the last block of 128 threads partly used; 511 | 512: one element or four
# a load; 513: chunks that end inside the row; 1300 x 2052 and 700 x 4999: the next row is fetched ahead
@pytest.mark.parametrize("rows,cols", [(1, 8), (129, 10), (5, 16), (5, 17), (64, 100), (3, 511), (7, 512), (2, 513), (1, 5000), (2, 16384),
                                       (1300, 2052), (700, 4999)])
def test_softmax_rows(cuda, oracle, rows, cols):
    launches = _softmax(cuda, oracle, rows, cols)
    assert launches == 1 or rows == 1          # the range of a single row folds away: nothing left to chain over


def test_rows_too_long_for_registers_keep_the_other_forms(cuda, oracle):
    assert _softmax(cuda, oracle, 3, 16385) > 1
    assert _softmax(cuda, oracle, 130, 16400) == 1


@pytest.mark.parametrize("rows,cols", [(9, 10), (9, 300), (700, 2100)])
def test_masked_positions(cuda, oracle, rows, cols):
    assert _softmax(cuda, oracle, rows, cols, mask=True) == 1


@pytest.mark.parametrize("batch,classes", [(33, 16), (70, 250), (300, 1000), (40, 24)])
def test_half_precision_cross_entropy(cuda, oracle, batch, classes):
    """The f16 cross-entropy's per-row kernels, forward and backward, in chains."""
    from anneal_b200 import realize as R
    from util import compare
    R.MATERIALIZE_CONTRACTION_OPERANDS = True
    try:
        m = W.WideMLP(batch=batch, width=64, classes=classes, depth=1)
        x, y = m.make_inputs()
        compare(cuda, oracle, m.graph(x, y).targets(), 2e-3, what=f"cross-entropy {batch}x{classes}")
    finally:
        R.MATERIALIZE_CONTRACTION_OPERANDS = False


def _deviation(cuda, oracle, rows, cols, shared):
    """sum((y - max(x))^2) a row, with y = x or another leaf of the same shape: item for item the same structure."""
    x = Tensor.new_leaf((rows, cols)).set_data(W.normal(51, 1, rows * cols))
    y = x if shared else Tensor.new_leaf((rows, cols)).set_data(W.normal(51, 2, rows * cols) + np.float32(3))
    d = y.sub(x.max((1,)).reshape((rows, 1)).expand((rows, cols)))
    items, ids, inputs = schedule([d.mul(d).sum((1,))])
    before = cuda.stats()["kernels_launched"]
    got = cuda.run(items, inputs)[ids[0]]
    assert cuda.stats()["kernels_launched"] - before == 1
    want = oracle.run(items, inputs)[ids[0]]
    assert rel_err(got, want) <= tol(cols), (rows, cols, shared, rel_err(got, want))


# a thread, a warp and a block a row, the next row fetched ahead, and rows that stay in memory
@pytest.mark.parametrize("rows,cols", [(33, 12), (40, 300), (300, 1000), (1300, 2052), (130, 16400)])
@pytest.mark.parametrize("first", [True, False])
def test_chains_that_differ_only_in_what_they_share(cuda, oracle, rows, cols, first):
    """A compiled chain is kept by its members' structure and by which of their operands coincide: on one device, either may
    come first.  (Its own row count a direction, so that neither direction finds the other's kernels.)"""
    rows += 0 if first else 1
    _deviation(cuda, oracle, rows, cols, first)
    _deviation(cuda, oracle, rows, cols, not first)


# 20 elements a lane, where that halves the block: the first and the last row length of each range, and rows that are fetched ahead
@pytest.mark.parametrize("rows,cols", [(3, 2049), (3, 2560), (3, 2561), (2, 8193), (2, 10240), (2, 10241), (700, 2501), (700, 9001)])
def test_rows_that_halve_the_block(cuda, rows, cols):
    """Against float64 (the oracle's serial f32 sums are themselves up to 3.8e-5 off at these lengths).  A lane adds at most 24
    terms, ten steps join the lanes, and three such sums follow one another: 3 x 34 roundings of 2^-24, doubled for the
    single ones of the exponential, the quotient and the products."""
    s = W.SoftmaxFwdBwd(rows, cols)
    items, ids, inputs = schedule(s.graph()[0])
    before = cuda.stats()["kernels_launched"]
    got = cuda.run(items, inputs)[ids[0]].reshape(rows, cols)
    assert cuda.stats()["kernels_launched"] - before == 1
    assert rel_err(got, s.reference_dx()) <= 2 * 3 * 34 * 2.0 ** -24
    assert np.array_equal(cuda.run(items, inputs)[ids[0]].reshape(rows, cols), got)
