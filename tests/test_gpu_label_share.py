"""A node's neighbour-label shares (edge features 12 and 13) by each of the ways
they are summed: one 32-entry chunk, a table of the row's labels, chunk by chunk
when the labels do not fit the table, a block for a very long row. Against the
FP64 restatement; standardised features, the tolerance of test_gpu_mlp."""
import numpy as np
import pytest

import mlp_oracle as mo
import sc_gpu
from sc_gpu.learned import EdgeMlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("labels", [2, 255, 300, 1100])
@pytest.mark.parametrize("degree", [31, 32, 33, 64, 65, 600, 1024, 1025])
def test_shares_of_a_long_row(degree, labels):
    n = 1200
    rng = np.random.default_rng(degree + labels)
    # node 0 joined to `degree` nodes, a ring among the others
    ring = np.arange(1, n)
    far = rng.permutation(np.arange(1, n))[:degree]
    src = np.concatenate([ring, np.zeros(degree, np.int64)])
    dst = np.concatenate([np.roll(ring, 1), far])
    g = sc_gpu.CSRNetwork.from_edge_arrays(n, src.astype(np.uint64), dst.astype(np.uint64),
                                           rng.uniform(0.25, 1.0, len(src)))
    coarse, fine = rng.integers(0, labels, n), rng.integers(0, 4, n) * 1000
    m = EdgeMlp(seed=1)
    feat, ei, ej = m.features(g, 0.7, context=(coarse, fine))
    ptr, nbr, w = g.to_csr_parts()
    raw, oi, oj = mo.edge_features(ptr, nbr, w, g.strengths(), g.total_weight(), 0.7, coarse, fine, embedding=None)
    assert np.array_equal(ei, oi) and np.array_equal(ej, oj)
    mean, istd = m.scaler()
    want = (raw - mean.astype(np.float64)) * istd.astype(np.float64)
    assert np.allclose(feat[:, 12:14], want[:, 12:14], rtol=1e-4, atol=1e-4)
