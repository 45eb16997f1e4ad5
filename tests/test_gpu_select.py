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


@pytest.mark.parametrize("N,Q,k", [(16384, 5, 1), (32768, 300, 16), (131071, 384, 100), (131072, 385, 10),
                                   (140_000, 1536, 10), (150_000, 1537, 10), (300_000, 20, 512), (40_000, 30, 300),
                                   (270_000, 100, 100)])
def test_seeding_sizes(engine, oracle, N, Q, k):
    # dense seeding passes of few and many rows (rank counted among the keys below a bound, or by
    # histogram for the long shortlists), the levels after them by warp and by block
    import torch
    rng = np.random.default_rng(N + Q)
    X = rng.integers(0, 256, (N, 32)).astype(np.float32)
    X[::3, 0] += 0.5 if N < 200_000 else 0.0
    Qs = rng.integers(0, 256, (Q, 32)).astype(np.float32)
    d, i = engine.search(torch.from_numpy(X).cuda(), torch.from_numpy(Qs).cuda(), k)
    st = engine.last_stats()
    assert st["scan"] == 1 and engine.last_fixups() <= 2
    sub = rng.choice(Q, min(Q, 40), replace=False)
    od, oi = oracle.knn_gemm(X, Qs[sub], k, kp=st["kp"], rerank=True)
    np.testing.assert_array_equal(i.cpu().numpy()[sub], oi)
    np.testing.assert_array_equal(d.cpu().numpy()[sub], od)


def test_rows_that_are_not_finite_leave_the_thresholds_open(engine, oracle):
    # most sample rows are NaN or infinite: too few finite keys for a threshold, every query is
    # answered all the same
    import torch
    rng = np.random.default_rng(2)
    X = rng.random((20000, 24), dtype=np.float32)
    keep = np.zeros(20000, bool)
    keep[5::32] = True
    X[~keep, 4] = np.where(np.arange(20000)[~keep] % 2, np.nan, np.inf)
    Qs = rng.random((50, 24), dtype=np.float32)
    d, i = engine.search(torch.from_numpy(X).cuda(), torch.from_numpy(Qs).cuda(), 10)
    d, i = d.cpu().numpy(), i.cpu().numpy()
    good = np.flatnonzero(keep)
    assert keep[i].all()
    od, oi = oracle.knn_gemm(X[good], Qs, 10, kp=32, rerank=True)
    oracle.check_parity(X[good], Qs, 10, d, np.searchsorted(good, i), ref_idx=oi, gap_rel=1e-6, dist_rel=1e-5)


@pytest.mark.parametrize("D", [1, 8, 31, 32, 33, 63, 64, 65, 100, 127, 128, 129, 255])
@pytest.mark.parametrize("Q", [60, 400])
def test_rerank_row_widths(engine, oracle, Q, D):
    # the re-rank takes four, two or one rows of a group at a time by the row width; every partial sum
    # rounds, so the distances show the oracle's order of the sums
    import torch
    rng = np.random.default_rng(Q + D)
    X = (rng.random((17_003, D)) * 1000).astype(np.float32)
    Qs = (rng.random((Q, D)) * 1000).astype(np.float32)
    d, i = engine.search(torch.from_numpy(X).cuda(), torch.from_numpy(Qs).cuda(), 37)
    od, oi = oracle.knn_gemm(X, Qs, 37, kp=engine.last_stats()["kp"], rerank=True)
    np.testing.assert_array_equal(d.cpu().numpy(), od)
    np.testing.assert_array_equal(i.cpu().numpy(), oi)


@pytest.mark.parametrize("kind", ["int", "float"])
@pytest.mark.parametrize("N,Q,k", [(262_144, 128, 10), (262_145, 128, 10), (270_000, 129, 10), (600_001, 100, 100),
                                   (1_000_003, 3, 1), (400_000, 40, 512)])
def test_few_queries_seed_from_one_level(engine, oracle, kind, N, Q, k):
    # one tile of queries on a large corpus: thresholds from the dense pass alone, with more candidates per
    # query in the main pass and its selection
    import torch
    rng = np.random.default_rng(N + Q)
    if kind == "int":
        X = rng.integers(0, 256, (N, 66)).astype(np.float32)
        Qs = rng.integers(0, 256, (Q, 66)).astype(np.float32)
    else:
        X = rng.standard_normal((N, 66), dtype=np.float32)
        Qs = rng.standard_normal((Q, 66), dtype=np.float32)
    d, i = engine.search(torch.from_numpy(X).cuda(), torch.from_numpy(Qs).cuda(), k)
    st = engine.last_stats()
    assert st["scan"] == 1 and engine.last_fixups() <= 1
    sub = rng.choice(Q, min(Q, 12), replace=False)
    od, oi = oracle.knn_gemm(X, Qs[sub], k, kp=st["kp"], rerank=True)
    np.testing.assert_array_equal(i.cpu().numpy()[sub], oi)
    np.testing.assert_array_equal(d.cpu().numpy()[sub], od)


@pytest.mark.parametrize("Q", [152, 153])
@pytest.mark.parametrize("N,k", [(20_000, 10), (140_000, 100), (300_000, 300)])
def test_block_sizes_by_queries(engine, oracle, Q, N, k):
    # 512 threads a query up to a query an SM, 256 above: thresholds and selections, shortlists counted and sorted
    import torch
    rng = np.random.default_rng(N + Q)
    X = rng.integers(0, 64, (N, 20)).astype(np.float32)
    Qs = rng.integers(0, 64, (Q, 20)).astype(np.float32)
    d, i = engine.search(torch.from_numpy(X).cuda(), torch.from_numpy(Qs).cuda(), k)
    st = engine.last_stats()
    sub = rng.choice(Q, 20, replace=False)
    od, oi = oracle.knn_gemm(X, Qs[sub], k, kp=st["kp"], rerank=True)
    np.testing.assert_array_equal(i.cpu().numpy()[sub], oi)
    np.testing.assert_array_equal(d.cpu().numpy()[sub], od)


@pytest.mark.parametrize("Q", [1536, 1537, 3000])
@pytest.mark.parametrize("N,hi", [(16_384, 2), (20_001, 3), (33_333, 2), (140_000, 4)])
def test_dense_thresholds_with_ties(engine, oracle, Q, N, hi):
    # thresholds from dense keys by a block (1,536 queries) and by a warp: few distinct keys, so that more
    # words reach the bound than the warp's list holds
    import torch
    rng = np.random.default_rng(N + Q)
    X = rng.integers(0, hi, (N, 9)).astype(np.float32)
    Qs = rng.integers(0, hi, (Q, 9)).astype(np.float32)
    d, i = engine.search(torch.from_numpy(X).cuda(), torch.from_numpy(Qs).cuda(), 10)
    st = engine.last_stats()
    sub = rng.choice(Q, 30, replace=False)
    od, oi = oracle.knn_gemm(X, Qs[sub], 10, kp=st["kp"], rerank=True)
    np.testing.assert_array_equal(i.cpu().numpy()[sub], oi)
    np.testing.assert_array_equal(d.cpu().numpy()[sub], od)


@pytest.mark.parametrize("N,D,kind", [(140_000, 64, "float"), (140_000, 64, "int"), (60_000, 64, "float"), (60_000, 300, "float")])
def test_fixups_are_counted_whichever_keys_run(engine, N, D, kind):
    # a query at a row that half of the corpus repeats: its candidates overflow, every other query's do not
    import torch
    g = torch.Generator(device="cuda").manual_seed(N + D)
    rows = lambda n: (torch.rand((n, D), generator=g, device="cuda") if kind == "float" else
                      torch.randint(0, 100, (n, D), generator=g, device="cuda").float())
    c, q = rows(N), rows(30)
    c[:N // 2] = c[0]  # (every other row would be every row of the seeding sample)
    q[3] = c[0]
    engine.search(c, q, 10)
    assert engine.last_stats()["scan"] == 1 and 1 <= engine.last_fixups() <= 3
    engine.search(rows(N), q, 10)
    assert engine.last_fixups() <= 2
    engine.search(rows(1000), q, 10)
    assert engine.last_fixups() == 0


@pytest.mark.parametrize("N,Q,D,k", [(9000, 300, 1000, 10), (16000, 200, 600, 300), (12000, 2600, 130, 10)])
def test_certified_shortlists_of_ordinary_data_hold(engine, N, Q, D, k):
    import torch
    g = torch.Generator(device="cuda").manual_seed(N + D)
    c, q = torch.rand((N, D), generator=g, device="cuda"), torch.rand((Q, D), generator=g, device="cuda")
    engine.search(c, q, k)
    assert engine.last_fixups() == 0
    # a common offset leaves the split keys too few bits: FP32 keys answer
    engine.search(c + 500, q + 500, k)
    assert engine.last_fixups() == Q
