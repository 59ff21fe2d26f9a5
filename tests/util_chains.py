"""Schedules whose row chains meet shared memory: an intermediate in a slot that another one has left."""
import numpy as np

from anneal_b200 import realize as R
from anneal_b200.tensor import Tensor
from anneal_b200.realize import leaf_inputs
from anneal_b200 import workloads as W


def _leaf(rows, cols, seed):
    return Tensor.new_leaf((rows, cols)).set_data(W.normal(61, seed, rows * cols))


def _row(v, rows, cols):
    return v.reshape((rows, 1)).expand((rows, cols))


def column_vector(n):
    """n x n: item 0 a value a column (slot 0); item 1 reads all of them for every row; item 2 writes a value a row into slot 0."""
    w, x, z, u, v = (_leaf(n, n, k) for k in range(5))
    m = x.add(w.max((0,)).reshape((1, n)).expand((n, n))).max((1,))
    s = z.sub(_row(m, n, n)).max((1,))
    t = u.sub(_row(s, n, n)).max((1,))
    return [v.sub(_row(t, n, n)).max((1,))]


def row_over_value(rows, cols):
    """Items 0 and 1 a value a row each (slots 0, 1); item 2 a whole row, into slot 0; item 3 a contraction over it."""
    x, y, z, b = _leaf(rows, cols, 1), _leaf(rows, cols, 2), _leaf(rows, cols, 3), _leaf(cols, 24, 4)
    m = x.max((1,))
    s = y.sub(_row(m, rows, cols)).max((1,))
    t = z.sub(_row(s, rows, cols)).max((1,))
    return [z.mul(_row(t, rows, cols)).matmul(b)]


def row_over_operand(rows, cols):
    """Item 0 a matrix (slot 0); item 1 its largest value a row (slot 1); item 2 a whole row, into slot 0: each over its own."""
    a, b, z, d = _leaf(rows, 40, 1), _leaf(40, cols, 2), _leaf(rows, cols, 3), _leaf(cols, 24, 4)
    m = a.matmul(b).max((1,))
    t = z.sub(_row(m, rows, cols)).max((1,))
    return [z.mul(_row(t, rows, cols)).matmul(d)]


def plan(targets):
    """(items, output ids, inputs), with a contraction's operands kept as buffers."""
    before, R.MATERIALIZE_CONTRACTION_OPERANDS = R.MATERIALIZE_CONTRACTION_OPERANDS, True
    try:
        items, ids = R.build_schedule(targets)
    finally:
        R.MATERIALIZE_CONTRACTION_OPERANDS = before
    return items, ids, leaf_inputs(targets)


def slots(items):
    return [it.bufs[0].slot for it in items]
