"""The survivor lists of a group (a word per row of the collection and query):
searches that read none do not allocate them, and a batched call that lacks
room gets theirs.  The same for the device copies of a host call's queries and
answers."""
import numpy as np
import pytest

from test_gpu_out_of_memory import Filled, MiB, same

pytestmark = pytest.mark.gpu

N, L, NQ = 2000000, 64, 32  # 32 lists: 256 MB; BF16 rows 256 MB, norms 32 MB


def make(hg):
    import torch
    X = torch.randn((N, L), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).cumsum(1)
    X -= X.mean(1, keepdim=True)
    X /= X.std(1, keepdim=True, unbiased=False)
    Q = (X[:NQ] + 0.1 * torch.randn((NQ, L), device="cuda")).cpu().numpy()
    torch.cuda.synchronize()
    ix = hg.HerculesIndex.build_device(X.data_ptr(), N, L, 20000)
    del X
    torch.cuda.empty_cache()
    return ix, Q


def test_scans_take_no_lists(hg, gpu_available):
    import torch
    ix, Q = make(hg)
    free = torch.cuda.mem_get_info()[0]
    pd, pi = ix.pscan(Q, 10)
    ix.knn(Q[:2], 10, epsilon=2.0)
    ix.knn(Q[:2], 10, nprobes=4)
    assert free - torch.cuda.mem_get_info()[0] < 128 * MiB
    # a search of the leaves gets its lists beside the scratch that is there
    d, ids = ix.knn(Q, 10)
    assert np.array_equal(d.view(np.uint32), pd.view(np.uint32)) and np.array_equal(ids, pi)
    ix.close()


def test_batch_gets_the_room_of_the_lists(hg, gpu_available):
    ix, Q = make(hg)
    d0, i0 = ix.knn(Q, 10, use_lb_sax=True)
    with Filled(200 * MiB):
        for _ in range(2):
            d, ids = ix.knn_batch(Q[:8], 10)
            assert np.array_equal(d.view(np.uint32), d0[:8].view(np.uint32)) and np.array_equal(ids, i0[:8])
            # groups of as many queries as fit now
            d, ids = ix.knn(Q, 10, use_lb_sax=True)
            assert np.array_equal(d.view(np.uint32), d0.view(np.uint32)) and np.array_equal(ids, i0)
    same(ix, Q, 10)
    ix.close()


def test_lists_beside_a_large_group(hg, gpu_available):
    """A group's scratch without lists took the room: a query at a time then."""
    ix, Q = make(hg)
    small = hg.HerculesIndex.build(hg.generate_walks(1, 3000, L), 500)
    small.knn(Q[:2], 10)   # the kernels are loaded while there is room
    small.close()
    pd, pi = ix.pscan(Q, 10)
    with Filled(4 * MiB):
        d, ids = ix.knn(Q, 10)
        assert np.array_equal(d.view(np.uint32), pd.view(np.uint32)) and np.array_equal(ids, pi)
    ix.close()


def test_host_copies_are_given_back(hg, gpu_available):
    """The copies of a call's queries and answers: those of a call that fails
    are freed, and a batch gets the room of those kept."""
    import torch
    ix, Q = make(hg)
    big = np.resize(Q, (600000, L))  # 154 MB, above what is kept
    ix.knn(Q[:1], 10)
    free = torch.cuda.mem_get_info()[0]
    with Filled(200 * MiB):
        with pytest.raises(hg.HerculesError) as e:
            ix.knn(big, 100)         # answers of 720 MB
        assert e.value.status == -5
    assert free - torch.cuda.mem_get_info()[0] < 32 * MiB
    kept = np.resize(Q, (250000, L))  # 64 MB
    ix.pscan(kept[:1], 10)
    with pytest.raises(hg.HerculesError):
        ix.knn(kept, 0)              # refused, its copy kept
    d0, i0 = ix.pscan(Q[:8], 10)
    with Filled(270 * MiB):          # BF16 rows and norms 288 MB
        d, ids = ix.knn_batch(Q[:8], 10)
    assert np.array_equal(d.view(np.uint32), d0.view(np.uint32)) and np.array_equal(ids, i0)
    ix.close()
