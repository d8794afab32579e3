"""Bound-pass work lists whose chunks are shortened to even out a small batch
over the SMs, on a fresh handle (the list is sized for that batch alone):
answers must be the plain path's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf,nq,btpi", [
    (415000, 100000, 64, 16),   # a few uneven leaves, long chunks
    (415000, 100000, 64, 64),
    (450000, 45000, 64, 8),     # leaves of some 300 row tiles
    (450000, 45000, 1, 2),
])
def test_shortened_chunks_match_plain_path(hg, gpu_available, n, leaf, nq, btpi):
    X = hg.generate_walks(1184, n, 32)
    Q = hg.generate_queries(14784, X, np.resize(np.array([0.01, 0.1, 1.0]), nq))
    ix = hg.HerculesIndex.build(X, leaf)
    ix.set_tuning(bound_tiles_per_item=btpi)
    d, ids = ix.knn_batch(Q, 5)
    pd, pi = ix.knn(Q, 5, use_lb_sax=True)
    assert np.array_equal(d.view(np.uint32), pd.view(np.uint32))
    assert np.array_equal(ids, pi)
    ix.close()
