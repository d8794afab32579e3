"""The batched path's exact re-rank, at the sizes where its work split changes.

Segments of a query's survivors are as long as the rows of all queries ask
for: one query with thousands of survivors gives more parts than the merge's
eight warps take in one go, a batch with few survivors gives segments of the
minimum length (16 rows, 4 for series of 4,096 points or more), and the bound
ranks rows 8 or 4 at a time.  The answers must be the plain path's, bit for
bit (itself pinned to the oracle)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,leaf,noisy,fresh,k", [
    (120000, 64, 12000, 0, 1, 200),   # one query with thousands of survivors: > 256 parts
    (120000, 64, 12000, 3, 1, 10),    # one query holds nearly every row
    (30000, 80, 500, 33, 0, 1),       # few survivors: the shortest segments, L off the slot width
    (30000, 16, 3000, 9, 9, 10),      # two chunks a row
    (2500, 4096, 300, 5, 2, 10),      # 8 lanes per row
    (1500, 16384, 1000, 3, 1, 10),
])
def test_batch_rerank_equals_plain_path(hg, gpu_available, n, L, leaf, noisy, fresh, k):
    X = hg.generate_walks(1184, n, L)
    Q = [hg.generate_queries(14784, X, np.array([0.01, 0.1, 1.0] * noisy)[:noisy])] if noisy else []
    if fresh:
        Q.append(hg.generate_walks(777, fresh, L))
    Q = np.concatenate(Q)
    ix = hg.HerculesIndex.build(X, leaf)
    d, ids, st = ix.knn_batch(Q, k, stats=True)
    pd, pi = ix.knn(Q, k, use_lb_sax=True)
    ix.close()
    assert st["survivors"] > 0, st
    assert np.array_equal(d.view(np.uint32), pd.view(np.uint32))
    assert np.array_equal(ids, pi)
