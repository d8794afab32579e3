"""Exact search without LB_SAX: every row of the candidate leaves is listed, a
warp per range of 32-row units (hg_kernels.cu, k_list_rows).  Against the scan
of all rows, which lists nothing: leaves of a few rows (many per unit run),
odd leaf borders, fewer units than a warp's least share, ranges of many units,
and the seeded search's two candidate ranges."""
import numpy as np
import pytest
import torch

import hercules_b200 as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,leaf,nq,k,seeds", [
    (97, 64, 10, 1, 3, 0),
    (3001, 64, 7, 3, 5, 0),
    (3001, 64, 7, 1, 5, 4),
    (3001, 64, 7, 3, 50, 0),  # the approximate leaf leaves the bound open
    (60013, 96, 701, 1, 10, 0),
    (60013, 96, 701, 7, 10, 3),
    (400009, 64, 20000, 2, 100, 0),
    (400009, 64, 400009, 33, 1, 0),
])
def test_listed_rows_hold_the_answer(n, L, leaf, nq, k, seeds):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + nq)
    X = torch.randn((n, L), generator=gen, device="cuda").cumsum(1)
    Q = X[torch.randint(n, (nq,), generator=gen, device="cuda")] + 0.3 * torch.randn((nq, L), generator=gen, device="cuda")
    for t in (X, Q):
        t.sub_(t.mean(1, keepdim=True)).div_(t.std(1, keepdim=True, unbiased=False))
    torch.cuda.synchronize()
    ix = H.HerculesIndex.build_device(X.data_ptr(), n, L, leaf)
    Q = Q.cpu().numpy()
    pd, pi = ix.pscan(Q, k)
    d, ids = ix.knn(Q, k, use_lb_sax=False, approx_leaves=seeds)
    np.testing.assert_array_equal(d, pd)
    np.testing.assert_array_equal(ids, pi)
    ix.close()
