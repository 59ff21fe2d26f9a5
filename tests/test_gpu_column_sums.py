"""Bias gradients from the one-CTA contraction kernel's epilogue where the warps of a tile's CTAs are more than its 32-row
groups, or do not divide them: the ones left over must not touch the next tile's sums."""
import numpy as np
import pytest

from anneal_b200 import realize as R, workloads as W
from anneal_b200.device import Device
from anneal_b200.realize import leaf_inputs

pytestmark = pytest.mark.gpu


# ten warps over 16 groups (K in chunks); clusters of two and four CTAs; one CTA a tile
@pytest.mark.parametrize("batch,width,classes", [(1536, 2048, 72), (300, 264, 136), (256, 1024, 72), (512, 2048, 72), (1024, 1024, 72)])
def test_column_sums(batch, width, classes):
    R.reset()
    before, R.MATERIALIZE_CONTRACTION_OPERANDS = R.MATERIALIZE_CONTRACTION_OPERANDS, True
    try:
        m = W.WideMLP(batch=batch, width=width, classes=classes, depth=2)
        x, y = m.make_inputs()
        g = m.graph(x, y)
        items, out_ids = R.build_schedule(g.targets())
    finally:
        R.MATERIALIZE_CONTRACTION_OPERANDS = before
    inputs = leaf_inputs(g.targets())
    got = []
    for flags in (0, 0, Device.NO_EPILOGUE_FUSION):
        dev = Device(0, flags)
        try:
            got.append(dev.run(items, inputs))
            assert (dev.stats()["colsums_fused"] > 0) == (flags == 0)
        finally:
            dev.close()
    fused, again, apart = got
    for k in out_ids:
        assert np.array_equal(fused[k], again[k])
        if apart[k].size == width:          # f16 addends summed in f32 in another order, one rounding to f16
            assert np.abs(fused[k] - apart[k]).max() <= 2e-3 * np.abs(apart[k]).max()
