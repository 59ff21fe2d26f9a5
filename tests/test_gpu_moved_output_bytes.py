"""Outputs that move out of their slots to be fused hold memory of their own to the end of the call: a deep forward pass moves a
bounded number of bytes, and its later layers run apart, with the same values."""
import numpy as np
import pytest

from anneal_b200 import nn, realize as R, workloads as W
from anneal_b200.device import Device
from anneal_b200.realize import leaf_inputs
from anneal_b200.tensor import Tensor
from anneal_b200.uop import dtypes

ROWS, WIDTH, LIMIT = 2048, 4096, 128 << 20


def _deep(layers):
    R.reset()
    before, R.MATERIALIZE_CONTRACTION_OPERANDS = R.MATERIALIZE_CONTRACTION_OPERANDS, "auto"
    try:
        h = Tensor.new_leaf((ROWS, WIDTH), dtypes.float16).set_data(W.normal(75, 0, ROWS * WIDTH))
        w = Tensor.new_leaf((WIDTH, WIDTH), dtypes.float16).set_data(W.normal(75, 1, WIDTH * WIDTH) * np.float32(1.7 / np.sqrt(WIDTH))).permute((1, 0))
        for _ in range(layers):
            h = nn.gelu_tanh(h.matmul(w))
        items, ids = R.build_schedule([h])
    finally:
        R.MATERIALIZE_CONTRACTION_OPERANDS = before
    return items, ids, leaf_inputs([h])


def _apart(items):
    """Layers whose consumer stays a launch of its own: its output is planned over what the contraction reads, and the bytes
    that may move have gone."""
    at, left, apart = {}, LIMIT, 0
    for raw, act in zip(items[::2], items[1::2]):
        out = act.bufs[0]
        place = out.slot if out.slot >= 0 else None
        if place is not None and place in [at.get(b.uop_idx) for b in raw.bufs[1:]]:
            if left >= ROWS * WIDTH * 2:
                left -= ROWS * WIDTH * 2
                place = None
            else:
                apart += 1
        at[out.uop_idx] = place
    return apart


@pytest.mark.gpu
@pytest.mark.parametrize("layers,over", [(16, False), (28, True)])
def test_bytes_that_move_are_bounded(layers, over):
    items, ids, inputs = _deep(layers)
    assert len(items) == 2 * layers and (_apart(items) > 0) == over
    got = []
    for flags in (0, Device.NO_EPILOGUE_FUSION):
        dev = Device(0, flags)
        try:
            got.append(dev.replay(items, inputs)[ids[0]].copy())
            assert dev.stats()["epilogues_fused"] == (0 if flags else layers - _apart(items))
        finally:
            dev.close()
    assert np.isfinite(got[0]).all() and np.abs(got[0]).max() > 0.1 and np.array_equal(*got)
