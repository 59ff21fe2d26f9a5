"""The one-CTA tensor-core contraction kernel: few rows or columns, K slices shared by a cluster, rows that do
not start on 16-byte boundaries, and the fused consumer and column sums in its epilogue."""
import numpy as np
import pytest

from anneal_b200 import nn, realize as R
from anneal_b200.tensor import Tensor
from anneal_b200.uop import dtypes
from anneal_b200 import workloads as W
from util import compare, schedule

pytestmark = pytest.mark.gpu
F16 = 2e-3      # one f16 rounding is 4.9e-4 of a value; sums of products that cancel get the oracle's noise on top


def hleaf(shape, seed):
    return Tensor.new_leaf(shape, dtypes.float16).set_data(W.normal(31, seed, int(np.prod(shape))) * np.float32(0.5))


# one row; a 32-row quadrant and one more; a 64-row stage and one more; one tile and one more row; few columns; odd
# extents, whose rows have to be copied first; slices of unequal length (17 k-blocks); the last k-block partly filled
@pytest.mark.parametrize("M,N,K", [(1, 4096, 1088), (32, 1000, 1024), (33, 264, 1030), (65, 136, 4096), (129, 72, 1096), (300, 10, 700),
                                   (255, 333, 999), (9, 4096, 1001)])
@pytest.mark.parametrize("layout", ["KK", "KM", "MM", "MK"])
def test_layouts(cuda, oracle, M, N, K, layout):
    a = hleaf((M, K), 1) if layout[0] == "K" else hleaf((K, M), 1).permute((1, 0))
    b = hleaf((N, K), 2).permute((1, 0)) if layout[1] == "K" else hleaf((K, N), 2)
    before = cuda.stats()["gemm_launched"]
    compare(cuda, oracle, [a.matmul(b)], F16, what=f"{layout} {M}x{N}x{K}")
    routed = cuda.stats()["gemm_launched"] - before
    # a row stored with its columns apart (one row, m "contiguous") is the k-contiguous form or stays generated
    assert routed == 1 or M * N * K < 1 << 23, "contraction was not routed to the tensor-core kernel"


@pytest.mark.parametrize("batch,width", [(1, 512), (5, 512), (32, 1024), (200, 136)])
def test_serving_layers_fuse_and_repeat(cuda, oracle, batch, width):
    """Logits of two layers: the bias and GELU run in the epilogue, and a second run gives the same bits."""
    x = hleaf((batch, width), 3)
    layers = [nn.Linear(width, width, True, dtypes.float16), nn.Linear(width, 72, True, dtypes.float16)]
    for k, l in enumerate(layers):
        for p in l.params():
            p.value[:] = W.normal(32, k, p.value.size) * np.float32(0.05)
            p.load()
    out = layers[1].forward(nn.gelu_tanh(layers[0].forward(x)))
    before = cuda.stats()["epilogues_fused"]
    R.MATERIALIZE_CONTRACTION_OPERANDS = "auto"       # as a serving program schedules it: the activations are buffers
    try:
        compare(cuda, oracle, [out], F16, what=f"serving {batch}x{width}")
        items, ids, inputs = schedule([out])
    finally:
        R.MATERIALIZE_CONTRACTION_OPERANDS = False
    if batch * width * width >= 1 << 20:
        assert cuda.stats()["epilogues_fused"] > before
    first, second = cuda.run(items, inputs)[ids[0]], cuda.run(items, inputs)[ids[0]]
    assert np.array_equal(first, second)


# 33 rows: one quadrant and a row; columns that end inside a piece of eight, or of four; 33 k-blocks (two slices at least:
# 1024 terms is the most one accumulates), an odd K, the longest K of this route
@pytest.mark.parametrize("M,N,K", [(33, 2048, 1024), (129, 520, 1000), (257, 1030, 300), (64, 1001, 1056), (600, 640, 601), (40, 1024, 4096)])
@pytest.mark.parametrize("layout", ["KK", "MM"])
def test_f32_form(cuda, M, N, K, layout):
    """3 x TF32 with K in slices, against float64: the bound of the pair kernel's form (1e-5 of the largest output), whose
    slices are as long at most and are added the same way; and the same bits twice."""
    f = lambda shape, seed: Tensor.new_leaf(shape, dtypes.float32).set_data(W.normal(41, seed, int(np.prod(shape))) * np.float32(0.5))
    a = f((M, K), 1) if layout[0] == "K" else f((K, M), 1).permute((1, 0))
    b = f((N, K), 2).permute((1, 0)) if layout[1] == "K" else f((K, N), 2)
    items, ids, inputs = schedule([a.matmul(b)])
    before = cuda.stats()
    y = cuda.run(items, inputs)[ids[0]].reshape(M, N)
    after = cuda.stats()
    assert after["gemm_launched"] - before["gemm_launched"] == 1
    assert after["kernels_launched"] - before["kernels_launched"] == 3      # two operand splits and the contraction
    la = [v for v in inputs.values() if v.size == M * K][0]
    lb = [v for v in inputs.values() if v.size == N * K and v is not la][0]
    am = (la.reshape(M, K) if layout[0] == "K" else la.reshape(K, M).T).astype(np.float64)
    bm = (lb.reshape(N, K) if layout[1] == "K" else lb.reshape(K, N).T).astype(np.float64)
    ref = am @ bm.T
    assert np.abs(y - ref).max() <= 1e-5 * np.abs(ref).max()
    assert np.array_equal(cuda.run(items, inputs)[ids[0]].reshape(M, N), y)


def _bias(cuda, M, N, K, dtype, layout="KK"):
    """Mean relative error against float64 of sums of K positive terms, and the standard error of that mean."""
    gen = np.random.default_rng(K)
    scale = np.sqrt(2000 / (2.25 * K)) if dtype is dtypes.float16 else 1.0        # f16 outputs near 2000
    np_type = np.float16 if dtype is dtypes.float16 else np.float32
    am, bm = ((gen.uniform(1, 2, (rows, K)) * scale).astype(np_type).astype(np.float32) for rows in (M, N))
    f = lambda m, kc: (Tensor.new_leaf(m.shape, dtype).set_data(m.reshape(-1)) if kc else Tensor.new_leaf(m.shape[::-1], dtype).set_data(m.T.reshape(-1)).permute((1, 0)))
    items, ids, inputs = schedule([f(am, layout[0] == "K").matmul(f(bm, layout[1] == "K").permute((1, 0)))])
    before = cuda.stats()["gemm_launched"]
    y = cuda.run(items, inputs)[ids[0]].reshape(M, N)
    assert cuda.stats()["gemm_launched"] == before + 1
    assert np.array_equal(cuda.run(items, inputs)[ids[0]].reshape(M, N), y)
    ref = am.astype(np.float64) @ bm.astype(np.float64).T
    e = y / ref - 1.0
    return abs(e.mean()), e.std() / np.sqrt(e.size)


# one tile of few columns; a chunk and a k-block, two chunks, slices of unequal length (one of them no longer than a
# chunk); narrow, wide and partly empty tiles; the longest K of the route
@pytest.mark.parametrize("M,N,K", [(256, 1024, 288), (256, 1024, 512), (64, 1024, 4096), (300, 1024, 4096), (2048, 1024, 1024), (512, 4096, 1024),
                                   (256, 4096, 1000), (64, 1001, 4001), (1000, 300, 545)])
def test_long_f32_sums_lose_no_more_than_one_chunk(cuda, M, N, K):
    """The tensor cores cut each partial sum, so the mean error of a sum of positive terms grows with the additions that one
    accumulator takes: K terms must show no more than the 256 of a chunk do (with a tenth and four standard errors in hand),
    plus one rounding for each chunk added in f32."""
    one, s1 = _bias(cuda, 256, 1024, 256, dtypes.float32)
    many, s2 = _bias(cuda, M, N, K, dtypes.float32)
    assert many <= 1.1 * one + 4 * (s1 + s2) + (K // 256) * 2.0 ** -25, (many, one)


@pytest.mark.parametrize("M,N,K,layout", [(40, 1024, 65536, "KK"), (40, 1024, 9000, "MM"), (300, 40, 20001, "KK"), (1, 4096, 32768, "KK"), (77, 333, 8191, "MK"),
                                          (256, 256, 16384, "KM"), (130, 96, 1100, "KK")])
def test_long_f16_sums_lose_no_more_than_one_chunk(cuda, M, N, K, layout):
    """The same with chunks of 1024 terms, 64 additions: each cuts less than 2^-22 of what has been added up so far, half of the
    total on average, so 32 x 2^-22 in all, below the 2^-12 of the one rounding to f16."""
    bias, se = _bias(cuda, M, N, K, dtypes.float16, layout)
    assert bias <= 32 * 2.0 ** -22 + 4 * se, bias


@pytest.mark.parametrize("M,N,K,layout", [(8, 8, 1 << 18, "KK"), (1, 64, 65536, "KK"), (10, 10, 40001, "MM"), (32, 32, 70000, "MK")])
def test_a_handful_of_outputs_is_split_over_the_machine(cuda, M, N, K, layout):
    """At most 1024 outputs stay with the generated reduction, in blocks that share each of them and add in f32 with rounding: sums
    of positive terms are the rounding to f16 (2^-11) away from float64, and at most a hundredth of it more."""
    gen = np.random.default_rng(M * N)
    am, bm = ((gen.uniform(1, 2, (rows, K)) * np.sqrt(2000 / (2.25 * K))).astype(np.float16).astype(np.float32) for rows in (M, N))
    a = Tensor.new_leaf((M, K), dtypes.float16).set_data(am.reshape(-1)) if layout[0] == "K" else Tensor.new_leaf((K, M), dtypes.float16).set_data(am.T.reshape(-1)).permute((1, 0))
    b = Tensor.new_leaf((N, K), dtypes.float16).set_data(bm.reshape(-1)).permute((1, 0)) if layout[1] == "K" else Tensor.new_leaf((K, N), dtypes.float16).set_data(bm.T.reshape(-1))
    items, ids, inputs = schedule([a.matmul(b)])
    before = cuda.stats()["gemm_launched"]
    y = cuda.run(items, inputs)[ids[0]].reshape(M, N)
    assert cuda.stats()["gemm_launched"] == before
    ref = am.astype(np.float64) @ bm.astype(np.float64).T
    assert np.abs(y / ref - 1.0).max() <= 1.01 * 2.0 ** -11


@pytest.mark.parametrize("batch,width,out", [(257, 4104, 264), (256, 12288, 136)])
def test_fused_consumer_behind_chunks(cuda, oracle, batch, width, out):
    """A layer whose slices of K are longer than a chunk, with its bias and GELU in the epilogue."""
    from anneal_b200.device import lower_gemm
    x, layers = hleaf((batch, width), 5), [nn.Linear(width, out, True, dtypes.float16), nn.Linear(out, 72, True, dtypes.float16)]
    for k, l in enumerate(layers):
        for p in l.params():
            p.value[:] = W.normal(33, k, p.value.size) * np.float32(0.05)
            p.load()
    y = layers[1].forward(nn.gelu_tanh(layers[0].forward(x)))
    R.MATERIALIZE_CONTRACTION_OPERANDS = "auto"
    try:
        source = lower_gemm(schedule([y])[0], 0, fuse_next=True)["source"]
        assert "#define CFG_CHUNK 16\n" in source and "#define CFG_EPI 1\n" in source
        before = cuda.stats()["epilogues_fused"]
        compare(cuda, oracle, [y], F16, what=f"chunks {batch}x{width}")
    finally:
        R.MATERIALIZE_CONTRACTION_OPERANDS = False
    assert cuda.stats()["epilogues_fused"] > before
