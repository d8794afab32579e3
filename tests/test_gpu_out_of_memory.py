"""Batched calls that the device has no room for return HG_ERR_NOMEM, and what
they leave behind does not meet the next call: with the memory given back, or
for a batch that fits, the same handle answers as the plain path does, bit for
bit.  The room is taken by plain allocations of the test."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HG_ERR_NOMEM = -5
MiB = 1 << 20


class Filled:
    """All but `leave` bytes of the device's free memory, while it is open."""

    def __init__(self, leave):
        self.leave = leave

    def __enter__(self):
        import torch
        gc.collect()
        torch.cuda.empty_cache()
        self.blocks = []
        for piece in (4096 * MiB, 256 * MiB, 2 * MiB):
            while torch.cuda.mem_get_info()[0] - self.leave >= piece:
                try:
                    self.blocks.append(torch.empty(piece, dtype=torch.uint8, device="cuda"))
                except torch.OutOfMemoryError:
                    break
        return self

    def __exit__(self, *exc):
        import torch
        self.blocks.clear()
        gc.collect()
        torch.cuda.empty_cache()


def same(ix, Q, k):
    d, ids = ix.knn_batch(Q, k)
    pd, pi = ix.knn(Q[-64:], k, use_lb_sax=True)
    assert np.array_equal(d[-64:].view(np.uint32), pd.view(np.uint32))
    assert np.array_equal(ids[-64:], pi)


@pytest.mark.parametrize("nq,k,leave", [
    (200000, 10, 300),   # the exact keys of the queries do not fit
    (4096, 10, 300),     # the survivor pairs do not
    (4096, 10, 800),     # the buckets do not
    (20000, 224, 6400),  # nor here, after parts of 224 entries
])
def test_batch_that_does_not_fit(hg, gpu_available, nq, k, leave):
    X = hg.generate_walks(1184, 20000, 96)
    Q = hg.generate_queries(14784, X, np.resize(np.array([0.01, 0.1, 1.0]), nq))
    ix = hg.HerculesIndex.build(X, 1500)
    same(ix, Q[:8], 10)
    with Filled(leave * MiB):
        for _ in range(2):
            with pytest.raises(hg.HerculesError) as e:
                ix.knn_batch(Q, k)
            assert e.value.status == HG_ERR_NOMEM, str(e.value)
            same(ix, Q[:8], 10)   # a batch that fits
            same(ix, Q[:5], 100)
    if nq <= 4096:
        same(ix, Q, k)
    same(ix, Q[:9], k)
    ix.close()


def test_half_a_bf16_copy(hg, gpu_available):
    """The BF16 rows (288 MB) fit, their norms (24 MB) do not."""
    import torch
    n, L = 1500000, 96
    X = torch.randn((n, L), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).cumsum(1)
    X -= X.mean(1, keepdim=True)
    X /= X.std(1, keepdim=True, unbiased=False)
    Q = X[:64].cpu().numpy()
    torch.cuda.synchronize()
    ix = hg.HerculesIndex.build_device(X.data_ptr(), n, L, 20000)
    del X
    ix.knn(Q[:1], 10)
    with Filled(n * L * 2 + 12 * MiB):
        for _ in range(2):
            with pytest.raises(hg.HerculesError) as e:
                ix.knn_batch(Q, 10)
            assert e.value.status == HG_ERR_NOMEM, str(e.value)
            ix.knn(Q[:1], 10)
    same(ix, Q, 10)
    ix.close()
