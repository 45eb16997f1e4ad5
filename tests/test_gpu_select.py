"""The selection over the threshold scan's segments (select_block_kernel, csrc/select.cu): both block
sizes (up to 384 queries and above), shortlists ordered by counting (up to 128 entries) and by the
bitonic sort, row widths that leave a partial step of eight columns, and integer data whose ties at
the shortlist's end are settled by the index.  Bit-exact against the oracle: integer arithmetic, or
the oracle's own re-rank order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Q,k,D,hi", [(1, 1, 5, 256), (3, 100, 16, 8), (384, 100, 64, 256), (385, 100, 16, 8),
                                      (700, 300, 129, 256), (384, 300, 16, 8), (385, 17, 7, 64), (500, 112, 41, 4)])
def test_integer_rows_bit_exact(engine, oracle, Q, k, D, hi):
    import torch
    rng = np.random.default_rng(Q + k + D)
    X = rng.integers(0, hi, (20000, D)).astype(np.float32)
    Qs = rng.integers(0, hi, (Q, D)).astype(np.float32)
    d, i = engine.search(torch.from_numpy(X).cuda(), torch.from_numpy(Qs).cuda(), k)
    st = engine.last_stats()
    assert st["scan_keys"] == 2
    od, oi = oracle.knn_gemm(X, Qs, k, kp=st["kp"], rerank=True)
    np.testing.assert_array_equal(i.cpu().numpy(), oi)
    np.testing.assert_array_equal(d.cpu().numpy(), od)


@pytest.mark.parametrize("Q,k", [(100, 100), (600, 10)])
def test_exact_integer_keys_skip_the_rerank(engine, oracle, Q, k):
    # BF16 keys that are exact integers: distances read off the keys
    import torch
    rng = np.random.default_rng(Q)
    X = rng.integers(0, 256, (140_000, 24)).astype(np.float32)
    Qs = rng.integers(0, 256, (Q, 24)).astype(np.float32)
    d, i = engine.search(torch.from_numpy(X).cuda(), torch.from_numpy(Qs).cuda(), k)
    st = engine.last_stats()
    assert st["scan_keys"] == 3
    od, oi = oracle.knn_gemm(X, Qs, k, kp=st["kp"], rerank=True)
    np.testing.assert_array_equal(i.cpu().numpy(), oi)
    np.testing.assert_array_equal(d.cpu().numpy(), od)
