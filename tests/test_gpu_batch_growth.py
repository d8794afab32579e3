"""Batches of growing size on one handle: every buffer of the batched path that
is sized by its queries, the inputs and the answers among them, grows with the
largest batch.  Answers are the plain path's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    [(3, 10), (64, 10), (65, 10), (700, 10), (2, 10)],   # same k: only the queries grow
    [(5, 100), (300, 1), (40, 224), (301, 3)],           # more queries with fewer answers each
])
def test_growing_batches_match_plain_path(hg, gpu_available, sizes):
    X = hg.generate_walks(1184, 20000, 96)
    ix = hg.HerculesIndex.build(X, 1500)
    for nq, k in sizes:
        Q = hg.generate_queries(14784 + nq, X, np.resize(np.array([0.01, 0.1, 1.0]), nq))
        d, ids = ix.knn_batch(Q, k)
        pd, pi = ix.knn(Q, k, use_lb_sax=True)
        assert np.array_equal(d.view(np.uint32), pd.view(np.uint32)), (nq, k)
        assert np.array_equal(ids, pi), (nq, k)
    ix.close()
