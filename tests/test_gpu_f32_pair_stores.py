"""f32 contractions on the two-CTA kernel: outputs are stored, and added to from chunk to chunk of K, in pieces that lanes exchange."""
import numpy as np
import pytest

from anneal_b200 import workloads as W
from anneal_b200.tensor import Tensor
from util import schedule

pytestmark = pytest.mark.gpu


# rows that end inside a group of four lanes, columns inside a piece of four (stored one by one) and inside a 32-column
# chunk; one chunk of K, two (the second short), three; K in slices
@pytest.mark.parametrize("M,N,K", [(2561, 2052, 1024), (2307, 1300, 1056), (2600, 1033, 2100), (2306, 2308, 2048), (1030, 1028, 9000)])
def test_f32_pair_stores(cuda, M, N, K):
    a = Tensor.new_leaf((M, K)).set_data(W.normal(81, 1, M * K))
    b = Tensor.new_leaf((N, K)).set_data(W.normal(81, 2, N * K))
    items, ids, inputs = schedule([a.matmul(b.permute((1, 0)))])
    y = cuda.run(items, inputs)[ids[0]].reshape(M, N)
    am, bm = (inputs[t.node.idx].reshape(-1, K).astype(np.float64) for t in (a, b))
    rows = np.unique(np.r_[0:36, M - 40:M, np.random.default_rng(1).integers(0, M, 40)])
    ref = am[rows] @ bm.T
    assert np.abs(y[rows] - ref).max() <= 1e-5 * np.abs(ref).max()        # the bound of this route's other tests
    assert np.array_equal(cuda.run(items, inputs)[ids[0]].reshape(M, N), y)
