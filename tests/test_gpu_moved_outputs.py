"""An output that moves out of its slot, so that it can be fused behind the contraction that still reads that memory, is written by
a launch of the schedule like any other: in a captured graph the contraction that takes it on the right, whose operand may be
loaded early where nothing writes it, has to wait for it."""
import numpy as np
import pytest

from anneal_b200 import nn, realize as R, workloads as W
from anneal_b200.device import Device
from anneal_b200.realize import leaf_inputs
from anneal_b200.tensor import Tensor
from anneal_b200.uop import dtypes

N = 256


def _layers(order, cols):
    """x, and after each letter gelu(w x) ('r': the activation on the right), gelu(x w) ('l') or gelu(x x / 64) ('b')."""
    R.reset()
    before, R.MATERIALIZE_CONTRACTION_OPERANDS = R.MATERIALIZE_CONTRACTION_OPERANDS, "auto"
    try:
        x = h = Tensor.new_leaf((N, cols), dtypes.float16).set_data(W.normal(71, 0, N * cols))
        for k, side in enumerate(order):
            if side == "b":
                t = h.matmul(h).mul(Tensor.full((N, cols), 1.0 / 64, dtypes.float16))
            else:
                w = Tensor.new_leaf((N, N), dtypes.float16).set_data(W.normal(71, 1 + k, N * N) * np.float32(1.5 / np.sqrt(N)))
                t = w.matmul(h) if side == "r" else h.matmul(w)
            h = nn.gelu_tanh(t)
        items, ids = R.build_schedule([h])
    finally:
        R.MATERIALIZE_CONTRACTION_OPERANDS = before
    return x, items, ids, leaf_inputs([h])


ORDERS = [("rrrr", 64), ("rrrrrr", 200), ("rlrlrlrl", N), ("llrrllrr", N), ("rrbbrrb", N)]


@pytest.mark.parametrize("order,cols", ORDERS)
def test_slots_make_outputs_move(order, cols):
    """What the replays below rely on: a consumer's output is planned over what its contraction reads, and a later contraction
    takes it on the right."""
    _, items, _, _ = _layers(order, cols)
    assert len(items) == 2 * len(order)
    place, moved = {}, []              # where each output is, and the layers whose output has moved
    for k in range(len(order)):
        raw, act = items[2 * k], items[2 * k + 1]
        at = act.bufs[0].slot
        if at >= 0 and at in [place.get(b.uop_idx) for b in raw.bufs[1:]]:
            at = None
            moved.append(k)
        place[act.bufs[0].uop_idx] = at if at is not None and at >= 0 else None
    assert any(order[k + 1] in "rb" for k in moved if k + 1 < len(order))


@pytest.mark.gpu
@pytest.mark.parametrize("order,cols", ORDERS)
def test_replays_with_new_inputs(order, cols):
    x, items, ids, inputs = _layers(order, cols)
    feeds = [{**inputs, x.node.idx: W.normal(72, k, N * cols)} for k in range(6)]
    plain = Device(0, Device.NO_EPILOGUE_FUSION)
    try:
        want = [plain.run(items, f)[ids[0]] for f in feeds]
    finally:
        plain.close()
    dev = Device(0)
    try:
        got = [dev.replay(items, f)[ids[0]].copy() for f in feeds + feeds]
        assert dev.stats()["epilogues_fused"] == len(order)
    finally:
        dev.close()
    for k, y in enumerate(got):
        assert np.isfinite(y).all() and np.abs(y).max() > 1e-3
        assert np.array_equal(y, want[k % len(feeds)])
    assert not np.array_equal(want[0], want[1])


# one wave of tile pairs and of whole 128 x 128 tiles: apart; more pairs than fit at once, narrower tiles: joined
@pytest.mark.gpu
@pytest.mark.parametrize("rows,width,moves", [(1536, 2304, 0), (2304, 2304, 1), (2048, 1024, 0), (1024, 1024, 1), (2048, 2048, 1)])
def test_outputs_move_where_that_pays(rows, width, moves):
    R.reset()
    before, R.MATERIALIZE_CONTRACTION_OPERANDS = R.MATERIALIZE_CONTRACTION_OPERANDS, "auto"
    try:
        h = Tensor.new_leaf((rows, width), dtypes.float16).set_data(W.normal(74, 0, rows * width))
        w = W.normal(74, 1, width * width) * np.float32(1.5 / np.sqrt(width))
        for _ in range(3):
            h = nn.gelu_tanh(h.matmul(Tensor.new_leaf((width, width), dtypes.float16).set_data(w).permute((1, 0))))
        items, ids = R.build_schedule([h])
    finally:
        R.MATERIALIZE_CONTRACTION_OPERANDS = before
    inputs, got = leaf_inputs([h]), []
    for flags in (0, Device.NO_EPILOGUE_FUSION):
        dev = Device(0, flags)
        try:
            got.append(dev.replay(items, inputs)[ids[0]].copy())
            assert dev.stats()["epilogues_fused"] == (0 if flags else 2 + moves)
        finally:
            dev.close()
    assert np.isfinite(got[0]).all() and np.abs(got[0]).max() > 0.1 and np.array_equal(*got)
