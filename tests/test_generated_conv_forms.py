"""Convolution kernels: the taps of a weight gradient side by side in one loop, neighbouring threads at neighbouring positions
of a forward pass, and their values against the oracle."""
import numpy as np
import pytest

from anneal_b200 import workloads as W
from anneal_b200.device import lower
from fullsize import check_every_kernel
from util import schedule

# batch, image, channels: many output groups of long sums (blocks of 256 to 1024 lanes); few groups (several blocks each, with
# a last part that is short or empty); sums too short for either; sums that no block size divides.  Last: whether positions run
# along the threads (100 positions of 8 channels touch nearly as many lines either way).
SHAPES = [(32, 28, 8, 16, True), (8, 16, 12, 24, True), (3, 20, 4, 8, False), (1, 16, 4, 8, True), (5, 36, 6, 10, True)]


@pytest.mark.parametrize("batch,hw,c1,c2,along", SHAPES)
def test_forms(batch, hw, c1, c2, along):
    m = W.SmallCNN(batch=batch, hw=hw, c1=c1, c2=c2)
    items, ids, _ = schedule(m.graph().targets())
    out = {it.bufs[0].uop_idx: k for k, it in enumerate(items)}
    grads = [lower(items, out[ids[k]])["note"] for k in (1, 3)]       # weight gradients of the two convolutions
    terms = (batch * hw * hw, batch * (hw // 2) ** 2)
    for note, t, groups in zip(grads, terms, (c1, c1 * c2)):
        assert ("9 outputs side by side" in note) == (t >= 1024), (note, t)
        assert ("split" in note) == (t >= 1024 and groups < 74 and t > 1024), (note, t)
    forward = [lower(items, k)["source"] for k, it in enumerate(items) if it.bufs[0].shape == (batch, (hw // 2) ** 2, c2)]
    assert len(forward) == 1
    assert (" * %dLL" % c2 in forward[0]) == along        # the store is then the one that strides


@pytest.mark.gpu
@pytest.mark.parametrize("batch,hw,c1,c2,along", SHAPES)
def test_values(cuda, oracle, batch, hw, c1, c2, along):
    """Sums of f32 products in another order: their rounding is part of the check's noise model, what is left is a few units."""
    m = W.SmallCNN(batch=batch, hw=hw, c1=c1, c2=c2)
    items, ids, inputs = schedule(m.graph().targets())
    _, got = check_every_kernel(cuda, oracle, items, inputs, 1e-6, samples=2048)
    again = cuda.run(items, inputs)
    for k in ids:
        assert np.array_equal(again[k], cuda.run(items, inputs)[k])
