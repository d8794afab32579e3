"""Index construction against the oracle's one-row-at-a-time insertion, where
the build takes its edges: leaves that split several times within one window of
rows, leaves of two rows, a single leaf, rows that repeat (every one of them
goes the same way at a split), series at both sides of the length that is
staged in shared memory, and row counts off the tile sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,leaf,repeat", [
    (3001, 16, 2, 0),
    (70001, 32, 300, 0),       # two windows, hundreds of leaves split together
    (20000, 48, 900, 2000),    # a tenth of the rows are one row
    (3000, 512, 40, 0),        # the longest staged series
    (3000, 528, 40, 0),        # the shortest read by a warp per row
    (999, 2064, 100, 0),
    (1000, 64, 5000, 0),       # one leaf
    (33, 64, 10, 33),          # nothing but one row
])
def test_build_matches_oracle(hg, oracle_mod, gpu_available, n, L, leaf, repeat):
    X = hg.generate_walks(1184, n, L)
    if repeat:
        X[np.random.default_rng(7).permutation(n)[:repeat]] = X[0]
    ix = hg.HerculesIndex.build(X, leaf)
    oi = oracle_mod.OracleIndex.build(X, leaf)
    assert ix.leaves() == oi.leaves()
    ids = ix.row_ids()
    assert np.array_equal(ids, oi.row_ids())
    rows, _ = ix.rows()
    assert np.array_equal(rows.view(np.uint32), X[ids].view(np.uint32))
    for i in range(ix.info.num_leaves):
        pts, env = ix.leaf_envelope(i)
        opts, oenv = oi.leaf_envelope(i)
        assert np.array_equal(pts, opts) and np.array_equal(env.view(np.uint32), oenv.view(np.uint32)), i
    ix.close()
