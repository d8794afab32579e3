"""The plain path answers the queries of a call in groups that share each
launch: every query's answer must be the oracle's, whatever the group's size
(one query, a full group, one more than a full group) and whichever branch of
the merge its lists take (all lists at once, or 32 at a time where k entries
of every list do not fit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(x):
    return np.asarray(x, np.float32).view(np.uint32)


@pytest.fixture(scope="module")
def indexes(hg, oracle_mod, gpu_available):
    made = {}

    def get(n, L, leaf):
        if (n, L, leaf) not in made:
            X = hg.generate_walks(1184, n, L)
            Q = np.concatenate([hg.generate_queries(14784, X, np.array([0.01, 0.1, 1.0] * 24)),
                                hg.generate_walks(4242, 9, L)])
            Q = Q[np.random.default_rng(1).permutation(len(Q))]
            made[n, L, leaf] = X, Q, hg.HerculesIndex.build(X, leaf), oracle_mod.OracleIndex.build(X, leaf)
        return made[n, L, leaf]

    yield get
    for X, Q, ix, oi in made.values():
        ix.close()


@pytest.mark.parametrize("n,L,leaf,nq,k,lbsax,seed_leaves", [
    (40000, 64, 700, 1, 10, True, 0),
    (40000, 64, 700, 2, 1, True, 0),
    (40000, 64, 700, 32, 10, False, 0),
    (40000, 64, 700, 33, 10, True, 0),
    (40000, 64, 700, 65, 3, True, 4),
    (40000, 64, 30000, 7, 224, False, 0),   # lists of 224 entries from hundreds of blocks
    (40000, 64, 30000, 1, 224, True, 0),
    (3000, 4096, 400, 33, 10, True, 0),     # 8 lanes per row
    (3000, 4096, 400, 1, 10, True, 0),      # a warp per row
    (600, 16384, 200, 1, 3, True, 0),       # the same, 32-warp blocks
    (600, 16384, 200, 40, 3, False, 0),
])
def test_grouped_queries_match_oracle(indexes, n, L, leaf, nq, k, lbsax, seed_leaves):
    X, Q, ix, oi = indexes(n, L, leaf)
    Q = Q[:nq]
    d, ids = ix.knn(Q, k, use_lb_sax=lbsax, approx_leaves=seed_leaves)
    rows = oi.row_ids()
    for j, q in enumerate(Q):
        od, orow, _, _ = oi.knn(q, k, tie_lowest=True)
        assert np.array_equal(bits(d[j]), bits(od)), j
        assert np.array_equal(ids[j], rows[orow]), j


@pytest.mark.parametrize("nq,k", [(1, 224), (5, 10), (33, 1)])
def test_grouped_scan_matches_oracle(indexes, oracle_mod, nq, k):
    X, Q, ix, oi = indexes(40000, 64, 700)
    d, ids = ix.pscan(Q[:nq], k)
    for j in range(nq):
        od, oid = oracle_mod.pscan(X, Q[j], k)
        assert np.array_equal(bits(d[j]), bits(od)) and np.array_equal(ids[j], oid), j
