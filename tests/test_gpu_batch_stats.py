"""The phase times of a batched call, taken from stamps on the device: none is
negative and together they are no more than the call's device time, whichever
filter kernel runs and whether its leaves are pruned first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cta_pair", [1, 2])
@pytest.mark.parametrize("dense", [False, True])
def test_phase_times_add_up(hg, gpu_available, cta_pair, dense):
    X = hg.generate_walks(1184, 30000, 128)
    Q = hg.generate_queries(14784, X, np.resize(np.array([0.01, 0.1, 1.0]), 90))
    ix = hg.HerculesIndex.build(X, 2500)
    ix.set_tuning(filter_cta_pair=cta_pair)
    for bucket_cap in (0, 64):  # 64: some queries are retried
        for _ in range(2):
            st = ix.knn_batch(Q, 5, stats=True, bucket_cap=bucket_cap, dense_filter=dense)[2]
        phases = [st["bound_ms"], st["gemm_ms"], st["rerank_ms"], st["fallback_ms"]]
        assert min(phases) >= 0.0 and min(phases[:3]) > 0.0, st
        assert sum(phases) <= st["device_ms"] * (1 + 1e-9), st
    ix.close()
