"""Batch queries that do not verify run through the plain path in groups of
equal k (hg_index.cu, knn_batch_impl): leaves of fewer rows than k leave every
query without a bound, so the answers of all come from there, each written to
its own row of the output whatever the order of the k values."""
import numpy as np
import pytest
import torch

import hercules_b200 as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,leaf,ks", [
    (4001, 64, 20, [50]),                                  # one query left
    (4001, 64, 20, [50] * 33),                             # more than a group
    (4001, 96, 20, [60, 3, 60, 1, 224, 3, 60, 30, 224]),   # several k, some verified
    (3000, 4096, 30, [40, 50, 40, 40]),
])
def test_unverified_queries_in_groups(n, L, leaf, ks):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + len(ks))
    X = torch.randn((n, L), generator=gen, device="cuda").cumsum(1)
    Q = X[torch.randint(n, (len(ks),), generator=gen, device="cuda")]
    Q = Q + 0.3 * torch.randn((len(ks), L), generator=gen, device="cuda")
    for t in (X, Q):
        t.sub_(t.mean(1, keepdim=True)).div_(t.std(1, keepdim=True, unbiased=False))
    torch.cuda.synchronize()
    ix = H.HerculesIndex.build_device(X.data_ptr(), n, L, leaf)
    Q = Q.cpu().numpy()
    d, ids, st = ix.knn_batch(Q, np.array(ks, dtype=np.uint32), stats=True)[:3]
    assert st["fallback_queries"] >= sum(k > leaf for k in ks)
    for q, k in enumerate(ks):
        pd, pi = ix.pscan(Q[q:q + 1], k)
        np.testing.assert_array_equal(d[q, :k], pd[0])
        np.testing.assert_array_equal(ids[q, :k], pi[0])
        assert np.all(np.isinf(d[q, k:])) and np.all(ids[q, k:] == -1)
    ix.close()
