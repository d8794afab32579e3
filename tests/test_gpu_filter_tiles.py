"""The batched filter at the edges of its tiles: query tiles of one to four
64-query boxes, series lengths whose last K block is partly filled (with the
query tile resident, L <= 256, and streamed), leaves of one row tile, and work
items of the minimum length.  Answers must be the plain path's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,leaf,nq", [
    (20000, 48, 2500, 1),
    (20000, 96, 2500, 64),
    (20000, 96, 2500, 65),
    (20000, 208, 2500, 192),
    (20000, 256, 2500, 193),
    (20000, 272, 2500, 130),   # streamed, one K = 16 step in the last block
    (12000, 336, 2500, 257),
    (12000, 1024, 130, 300),   # leaves of one or two row tiles
])
def test_filter_tile_edges_match_plain_path(hg, gpu_available, n, L, leaf, nq):
    X = hg.generate_walks(1184, n, L)
    Q = hg.generate_queries(14784, X, np.resize(np.array([0.01, 0.1, 1.0]), nq))
    ix = hg.HerculesIndex.build(X, leaf)
    for dense in (False, True):
        d, ids, st = ix.knn_batch(Q, 3, stats=True, dense_filter=dense)
        assert st["survivors"] > 0, st
        pd, pi = ix.knn(Q, 3, use_lb_sax=True)
        assert np.array_equal(d.view(np.uint32), pd.view(np.uint32))
        assert np.array_equal(ids, pi)
    ix.close()
