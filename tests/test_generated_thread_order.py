"""Kernels that work out a short REDUCE value by value may deal their outputs out to threads in another order of the ranges, also
where an output range is a switch over its values: every output still goes to its own place."""
import re

import numpy as np
import pytest

from anneal_b200.device import lower
from anneal_b200.tensor import Tensor
from anneal_b200 import workloads as W
from util import compare, schedule

# rows, terms (slices along the REDUCE), columns (slices along the last output range; 0: no slices); whether the order changes
SHAPES = [(2048, 9, 8, True), (64 * 196, 9, 8, True), (999, 11, 10, True), (999, 5, 7, False), (333, 12, 0, False), (40, 9, 33, True)]


def _pieces(shape, axis, seed):
    """[shape] put together from slices along `axis`."""
    whole = None
    for k in range(shape[axis]):
        part = tuple(1 if a == axis else n for a, n in enumerate(shape))
        t = Tensor.new_leaf(part).set_data(W.normal(73, 100 * seed + k, int(np.prod(part))))
        t = t.pad([(k, shape[axis] - 1 - k) if a == axis else (0, 0) for a in range(len(shape))])
        whole = t if whole is None else whole.add(t)
    return whole


def _product(rows, terms, cols):
    x = _pieces((rows, terms), 1, 1)
    w = _pieces((cols, terms), 0, 2) if cols else Tensor.new_leaf((16, terms)).set_data(W.normal(73, 900, 16 * terms))
    return x.matmul(w.permute((1, 0)))


@pytest.mark.parametrize("rows,terms,cols,moved", SHAPES)
def test_every_output_has_its_own_place(rows, terms, cols, moved):
    items, _, _ = schedule([_product(rows, terms, cols)])
    assert len(items) == 1
    low = lower(items, 0)
    assert "value-by-value reduce" in low["note"] and ("switch" in low["note"]) == (cols > 0)
    c = lambda e: re.sub(r"(\d)LL", r"\1", e).replace("(int)", "").replace("/", "//")
    ranges = re.findall(r"const int (r\d+) = ([^;]*%[^;]*|[^;]*/[^;]*|\(int\)[^;]*);", low["source"][:low["source"].index("{   //")])
    stores = set(re.findall(r"data0\[([^\]]*)\] = ", low["source"]))
    assert len(stores) == 1
    n = cols or 16
    seen = set()
    for g in range(rows * n):
        at = {"g": g}
        for name, e in ranges:
            at[name] = eval(c(e), {}, at)
        (place,) = (eval(c(e), {}, at) for e in stores)
        assert place == at["r0"] * n + at["r1"]
        seen.add(place)
    assert len(seen) == rows * n
    assert ("g" not in stores) == moved


@pytest.mark.gpu
@pytest.mark.parametrize("rows,terms,cols,moved", SHAPES)
def test_values(cuda, oracle, rows, terms, cols, moved):
    """A dozen f32 products in the oracle's order."""
    compare(cuda, oracle, [_product(rows, terms, cols)], 1e-6)
