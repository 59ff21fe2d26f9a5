"""A forward pass alone shares slots between layers: the output of a contraction's consumer is planned into the memory
the contraction reads.  Fused into one launch it needs memory of its own, and the values have to be the separate kernels'."""
import numpy as np
import pytest

from anneal_b200 import nn, realize as R, workloads as W
from anneal_b200.device import Device
from anneal_b200.realize import leaf_inputs
from anneal_b200.tensor import Tensor
from anneal_b200.uop import dtypes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,width,depth", [(32, 256, 4), (65, 256, 3), (520, 264, 3)])
@pytest.mark.parametrize("graph", [False, True])
def test_consumers_of_a_forward_pass_are_fused(batch, width, depth, graph):
    R.reset()
    before, R.MATERIALIZE_CONTRACTION_OPERANDS = R.MATERIALIZE_CONTRACTION_OPERANDS, "auto"
    try:
        x = Tensor.new_leaf((batch, width), dtypes.float16).set_data(W.normal(31, 1, batch * width))
        h = x
        for k in range(depth):
            w = Tensor.new_leaf((width, width), dtypes.float16).set_data(W.normal(31, 2 + k, width * width) * np.float32(1.5 / np.sqrt(width)))
            b = Tensor.new_leaf((width,), dtypes.float16).set_data(W.normal(32, 2 + k, width))
            h = nn.gelu_tanh(h.matmul(w.permute((1, 0))).add(b.reshape((1, width)).expand((batch, width))))
        items, ids = R.build_schedule([h])
    finally:
        R.MATERIALIZE_CONTRACTION_OPERANDS = before
    inputs = leaf_inputs([h])
    assert len(items) == 2 * depth and any(items[k + 1].bufs[0].slot == items[k - 1].bufs[0].slot for k in range(2, 2 * depth - 2, 2))
    got = []
    for flags in (0, Device.NO_EPILOGUE_FUSION):
        dev = Device(0, flags)
        try:
            for _ in range(2):
                e0 = dev.stats()["epilogues_fused"]
                y = (dev.replay(items, inputs) if graph else dev.run(items, inputs))[ids[0]]
                got.append(y)
                assert dev.stats()["epilogues_fused"] - e0 == (depth if not flags and (not graph or len(got) == 1) else 0)
        finally:
            dev.close()
    assert np.isfinite(got[0]).all() and np.abs(got[0]).max() > 0.1
    for y in got[1:]:
        assert np.array_equal(y, got[0])
