"""A layer's weight gradient and the gradient of its input as one launch of the one-CTA contraction kernel: the values are those
of two launches (which is what an instrumented run makes), replayed or not, and nothing that depends on the first is paired."""
import numpy as np
import pytest

from anneal_b200 import realize as R, workloads as W
from anneal_b200.device import Device
from anneal_b200.realize import leaf_inputs
from anneal_b200.tensor import Tensor
from anneal_b200.uop import dtypes

pytestmark = pytest.mark.gpu


def _run(dev, items, inputs, graph=False):
    s0 = dev.stats()
    got = dev.replay(items, inputs) if graph else dev.run(items, inputs)
    s1 = dev.stats()
    return got, s1["kernels_launched"] - s0["kernels_launched"], s1["gemm_launched"] - s0["gemm_launched"]


# clusters of one, two and more CTAs a tile; rows and columns past the last tile; a head whose rows are copied first (its
# gradients are not paired); tiles that fill the machine by themselves (nothing is paired)
@pytest.mark.parametrize("batch,width,classes,depth,pairs", [(1024, 1024, 1000, 3, 3), (999, 1000, 250, 3, 2), (300, 264, 136, 2, 2), (64, 2048, 72, 2, None), (256, 1024, 512, 2, None), (2048, 2048, 1000, 2, None)])
def test_paired_launches_equal_separate_launches(batch, width, classes, depth, pairs):
    R.reset()
    R.MATERIALIZE_CONTRACTION_OPERANDS = True
    try:
        m = W.WideMLP(batch=batch, width=width, classes=classes, depth=depth)
        x, y = m.make_inputs()
        g = m.graph(x, y)
        items, out_ids = R.build_schedule(g.targets())
    finally:
        R.MATERIALIZE_CONTRACTION_OPERANDS = False
    inputs = leaf_inputs(g.targets())
    dev = Device(0)
    try:
        got, kernels, gemms = _run(dev, items, inputs)
        graph = dev.replay(items, inputs)
        again = dev.replay(items, inputs)
        dev.profile(True)
        want, kernels_apart, gemms_apart = _run(dev, items, inputs)
        dev.profile(False)
    finally:
        dev.close()
    plain = Device(0, Device.NO_EPILOGUE_FUSION)
    try:
        apart = plain.run(items, inputs)
    finally:
        plain.close()
    assert gemms == gemms_apart
    if pairs is not None:
        assert kernels == kernels_apart - pairs
    for k in out_ids:
        assert np.isfinite(want[k]).all()
        assert np.array_equal(got[k], want[k]) and np.array_equal(graph[k], want[k]) and np.array_equal(again[k], want[k])
        # against kernels of their own: the same bits but for bias gradients, whose f16 addends are summed in f32 in another order
        if want[k].size in (width, classes) and batch > 1:
            assert np.abs(want[k] - apart[k]).max() <= 2e-3 * np.abs(apart[k]).max()
        else:
            assert np.array_equal(want[k], apart[k])


def test_a_contraction_that_reads_the_one_before_is_not_paired(cuda):
    """Two products in a row without a consumer between them, and then two that share an operand."""
    n = 512
    f = lambda seed: Tensor.new_leaf((n, n), dtypes.float16).set_data(W.normal(51, seed, n * n) * np.float32(0.2))
    a, b, c = f(1), f(2), f(3)
    for out, launches in (([a.matmul(b).matmul(c)], 2), ([a.matmul(b), a.matmul(c)], 1)):
        items, ids = R.build_schedule(out)
        inputs = leaf_inputs(out)
        got, kernels, gemms = _run(cuda, items, inputs)
        assert gemms == 2 and kernels == launches + sum(1 for v in inputs.values()) + len(ids)      # conversions of leaves and outputs
        h = lambda t: inputs[t.node.idx].reshape(n, n).astype(np.float16).astype(np.float64)
        ab = h(a) @ h(b)
        ref = [ab.astype(np.float16).astype(np.float64) @ h(c)] if launches == 2 else [ab, h(a) @ h(c)]
        for k, r in zip(ids, ref):
            assert np.abs(got[k].reshape(n, n) - r).max() <= 2e-3 * np.abs(r).max()
