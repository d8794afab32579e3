"""A batch whose survivor pairs do not fit the pair list.  Rows far from the
origin with little spread defeat the BF16 filter: every one of them survives
for a query among them, more rows than the list has room for, while the queries
of the same batch near the other rows keep few.  Rows that were lost must be
found again (retry rounds, then the plain path), and a bucket must be read no
further than it was written.  Answers are the plain path's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_FAR, N_NEAR, L = 1600000, 40000, 32


@pytest.fixture(scope="module")
def mixed(hg, gpu_available):
    import torch
    g = torch.Generator(device="cuda").manual_seed(1184)
    X = torch.randn((N_NEAR + N_FAR, L), generator=g, device="cuda")
    X[:N_NEAR] = X[:N_NEAR].cumsum(1)
    X[:N_NEAR] -= X[:N_NEAR].mean(1, keepdim=True)
    X[:N_NEAR] /= X[:N_NEAR].std(1, keepdim=True, unbiased=False)
    X[N_NEAR:] = 0.01 * X[N_NEAR:] + 100.0 * torch.randn((1, L), generator=g, device="cuda")
    torch.cuda.synchronize()
    ix = hg.HerculesIndex.build_device(X.data_ptr(), len(X), L, 20000)
    yield X, ix
    ix.close()


@pytest.mark.parametrize("far,near,k", [
    (1, 9, 10),     # one query fills the list, nine lose rows to it
    (100, 28, 10),  # 160M survivors for 3.3M slots: the slot counter's range
])
def test_lost_pairs_are_found_again(mixed, far, near, k):
    import torch
    X, ix = mixed
    g = torch.Generator(device="cuda").manual_seed(far)
    # slots of the list: 16,384 per query and a block of 1,024 for each of 8 warps of 148 SMs
    assert far * N_FAR > (far + near) * 16384 + 148 * 8 * 1024
    base = torch.cat([torch.randint(N_NEAR, (near,), generator=g, device="cuda"),
                      N_NEAR + torch.randint(N_FAR, (far,), generator=g, device="cuda")])
    Q = (X[base] + 0.01 * torch.randn((far + near, L), generator=g, device="cuda")).cpu().numpy()
    d, ids, st = ix.knn_batch(Q, k, stats=True)
    # no query of the first round may count as verified
    assert st["retried_queries"] + st["fallback_queries"] >= far + near, st
    pd, pi = ix.knn(Q, k, use_lb_sax=True)
    assert np.array_equal(d.view(np.uint32), pd.view(np.uint32))
    assert np.array_equal(ids, pi)
