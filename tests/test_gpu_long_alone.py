"""One query over long series: a row of the leaf scan goes to a warp or to 8 lanes
by the leaf size, a row of the list that follows by the rows it turns out to
hold (4,736 warps of 148 SMs of 32).  Answers on both sides of that against the
scan of every row, which takes 8 lanes throughout."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,leaf", [
    (2368, 4096, 2368),   # leaf scans of a warp per row
    (2369, 4096, 4000),   # one leaf, 8 lanes per row, nothing left after it
    (6001, 4096, 600),    # lists of few rows, and of nearly all
    (2371, 8192, 2500),   # 32-warp blocks
    (6003, 8192, 900),
])
def test_one_long_query_matches_scan(hg, gpu_available, n, L, leaf):
    X = hg.generate_walks(1184, n, L)
    rng = np.random.default_rng(n)
    Q = np.concatenate([hg.generate_queries(14784, X, np.array([0.01, 1.0])),
                        rng.standard_normal((2, L)).astype(np.float32)])  # white noise: nothing is pruned
    ix = hg.HerculesIndex.build(X, leaf)
    for q in range(len(Q)):
        for k in (1, 30):
            sd, si = ix.pscan(Q[q:q + 1], k)
            for lb in (False, True):
                d, ids = ix.knn(Q[q:q + 1], k, use_lb_sax=lb)
                assert np.array_equal(d.view(np.uint32), sd.view(np.uint32)), (q, k, lb)
                assert np.array_equal(ids, si), (q, k, lb)
    ix.close()
