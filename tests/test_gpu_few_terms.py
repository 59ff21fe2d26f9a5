"""f32 contractions of few terms (weight gradients at a small batch) on the kernel that holds rows of outputs in a thread."""
import numpy as np
import pytest

from anneal_b200 import workloads as W
from anneal_b200.device import Device
from anneal_b200.tensor import Tensor
from util import schedule

pytestmark = pytest.mark.gpu


# one row a thread (few outputs) and four (many); rows and columns that end inside a thread, a warp and a block; operands that
# 128-bit loads cannot take; 1, 2, 7, 8, 9, 16, 17 and 64 terms around the unrolled ones
@pytest.mark.parametrize("M,N,K", [(128, 784, 64), (129, 513, 17), (700, 131, 9), (513, 132, 8), (1024, 4096, 2), (1027, 4096, 5), (4096, 1021, 7),
                                   (2050, 2052, 16), (1024, 3072, 33), (3, 65536, 9), (65536, 5, 9), (65539, 66, 64)])
def test_few_terms(cuda, M, N, K):
    a = Tensor.new_leaf((K, M)).set_data(W.normal(61, 1, K * M))
    b = Tensor.new_leaf((K, N)).set_data(W.normal(61, 2, K * N))
    items, ids, inputs = schedule([a.permute((1, 0)).matmul(b)])
    before = cuda.stats()["gemm_launched"]
    y = cuda.run(items, inputs)[ids[0]].reshape(M, N)
    assert cuda.stats()["gemm_launched"] - before == (1 if N >= 64 else 0)
    rows = np.unique(np.r_[0:min(M, 40), max(0, M - 40):M, np.random.default_rng(3).integers(0, M, 60)])
    am, bm = (inputs[t.node.idx].reshape(K, -1).astype(np.float64) for t in (a, b))
    ref = am[:, rows].T @ bm
    # K products added one after the other in f32: K roundings of at most half a unit of the partial sums
    bound = (K + 1) * 2.0 ** -24 * (np.abs(am[:, rows]).T @ np.abs(bm))
    assert (np.abs(y[rows] - ref) <= bound + 1e-30).all()


# two and four rows a thread on either side of the line (66 and 99 to 101 blocks of four rows); warps that hold the end of one
# row and the start of the next; one column group a row; a last group of one, two and three rows
@pytest.mark.parametrize("M,N,K", [(128, 1056, 8), (132, 1056, 9), (401, 505, 24), (402, 511, 3), (3000, 70, 9), (1021, 65, 64), (1025, 64, 2), (400, 700, 17), (65537, 64, 4), (66, 65536, 2)])
def test_threads_run_through_the_rows(cuda, M, N, K):
    test_few_terms(cuda, M, N, K)
