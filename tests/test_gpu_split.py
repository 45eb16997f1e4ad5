"""The threshold scan on FP16-split keys (csrc/scan_f16.cu) at the edges of its tiles, K chunks and
key rule: row widths around 64, 128, 192 and 256 columns (accumulator layouts, partial K steps, the
kernel with both operands in shared memory), corpora and query counts that leave remainders, rows
whose magnitudes differ by many powers of two, rows that are not finite, and the searches that keep
3xTF32 keys (shortlists without a margin, distances read off the keys).

Bars as in test_gpu_parity.py: the oracle's indices except where the FP64 distances of the competing
candidates differ by less than 1e-6 relative, distances within 1e-5 relative of FP64.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GAP = 1e-6
DIST_REL = 1e-5


def run(engine, X, Qs, k, **kw):
    import torch
    d, i = engine.search(torch.from_numpy(X).cuda(), torch.from_numpy(Qs).cuda(), k, **kw)
    return d.cpu().numpy(), i.cpu().numpy(), engine.last_stats()


@pytest.mark.parametrize("N,Q,D,k", [(16384, 1, 1, 1), (16385, 127, 16, 10), (16511, 129, 63, 5), (16640, 64, 64, 16),
                                     (17001, 200, 65, 16), (16384, 33, 128, 100), (20001, 130, 129, 16),
                                     (16895, 20, 192, 16), (17000, 128, 193, 40), (16384, 65, 256, 16),
                                     (16641, 129, 257, 16), (16500, 5, 321, 200)])
def test_tile_edges(engine, oracle, N, Q, D, k):
    rng = np.random.default_rng(N + D)
    X = rng.standard_normal((N, D), dtype=np.float32)
    Qs = rng.standard_normal((Q, D), dtype=np.float32)
    d, i, st = run(engine, X, Qs, k)
    assert st["scan_keys"] == 2
    od, oi = oracle.knn_gemm(X, Qs, k, kp=st["kp"], rerank=True)
    oracle.check_parity(X, Qs, k, d, i, ref_idx=oi, gap_rel=GAP, dist_rel=DIST_REL)


@pytest.mark.parametrize("D", [96, 300])
def test_rows_of_very_different_magnitude(engine, oracle, D):
    # every row has its own scale, 2^-20 .. 2^20, so does every query
    rng = np.random.default_rng(D)
    X = (rng.standard_normal((18000, D)) * np.exp2(rng.integers(-20, 21, (18000, 1)))).astype(np.float32)
    Qs = (rng.standard_normal((90, D)) * np.exp2(rng.integers(-20, 21, (90, 1)))).astype(np.float32)
    d, i, st = run(engine, X, Qs, 20)
    assert st["scan_keys"] == 2
    od, oi = oracle.knn_gemm(X, Qs, 20, kp=st["kp"], rerank=True)
    oracle.check_parity(X, Qs, 20, d, i, ref_idx=oi, gap_rel=GAP, dist_rel=DIST_REL)


@pytest.mark.parametrize("D", [80, 272])
def test_rows_that_are_not_finite_are_never_returned(engine, oracle, D):
    rng = np.random.default_rng(D)
    X = rng.random((17000, D), dtype=np.float32)
    Qs = rng.random((40, D), dtype=np.float32)
    bad = rng.choice(17000, 300, replace=False)
    X[bad[:100], 3] = np.inf
    X[bad[100:200], D - 1] = -np.inf
    X[bad[200:], 0] = np.nan
    good = np.setdiff1d(np.arange(17000), bad)
    d, i, st = run(engine, X, Qs, 12)
    assert st["scan_keys"] == 2
    assert not np.isin(i, bad).any()
    od, oi = oracle.knn_gemm(X[good], Qs, 12, kp=st["kp"], rerank=True)
    oracle.check_parity(X[good], Qs, 12, d, np.searchsorted(good, i), ref_idx=oi, gap_rel=GAP, dist_rel=DIST_REL)


@pytest.mark.parametrize("N,k,rerank", [(40000, 512, True), (40000, 496, True), (40000, 16, False),
                                        (140000, 128, True)])
def test_index_answers_as_the_search_whichever_keys_serve_it(engine, N, k, rerank):
    # k = 512 and (from 131,072 rows) k = 128 leave the shortlist no margin, rerank = False returns
    # the keys: 3xTF32 copies, made by the index's first such search; k = 496 has a margin (FP16)
    import torch
    rng = np.random.default_rng(k)
    X = torch.from_numpy(rng.random((N, 48), dtype=np.float32)).cuda()
    Qs = torch.from_numpy(rng.random((70, 48), dtype=np.float32)).cuda()
    d, i = engine.search(X, Qs, k, rerank=rerank, scan=engine.SCAN_AUTO)
    ix = engine.Index(X)
    for _ in range(2):
        d2, i2 = ix.search(Qs, k, rerank=rerank)
        np.testing.assert_array_equal(i.cpu().numpy(), i2.cpu().numpy())
        np.testing.assert_array_equal(d.cpu().numpy(), d2.cpu().numpy())
    ix.close()


@pytest.mark.parametrize("where", ["first row", "last row", "scattered", "everywhere", "queries", "nowhere"])
@pytest.mark.parametrize("D,pad", [(33, 0), (96, 0), (100, 3)])
def test_adaptive_preparation_by_where_the_data_stop_being_bf16_exact(engine, where, D, pad):
    # one pass writes the BF16 side of the rows it sees before, the FP16 side of those after the data
    # turn out not to be BF16-exact; a second one catches up.  Same answers as the split-key scan
    # alone, which writes the FP16 side of every row.
    import torch
    g = torch.Generator(device="cuda").manual_seed(D + pad)
    N = 200_003
    X = torch.randint(0, 200, (N, D + pad), generator=g, device="cuda").float()[:, :D]
    Qs = torch.randint(0, 200, (90, D), generator=g, device="cuda").float()
    if where == "first row":
        X[0, 1] += 0.37
    elif where == "last row":
        X[N - 1, D - 1] += 0.37
    elif where == "scattered":
        X[::4001, 2] += 0.37
    elif where == "everywhere":
        X += torch.rand((N, D), generator=g, device="cuda")
    elif where == "queries":
        Qs[7, 3] += 0.37
    d, i = engine.search(X, Qs, 20)
    assert engine.last_stats()["scan_keys"] == 3
    d2, i2 = engine.search(X, Qs, 20, scan=engine.SCAN_TF32)
    assert torch.equal(i, i2) and torch.equal(d, d2)


@pytest.mark.parametrize("D", [385, 511, 512, 513, 1000, 1024, 1025, 2047, 2048, 2049])
def test_norms_of_wide_rows(engine, oracle, D):
    # rerank = False returns key + ||q||^2 from the CUDA-core keys: bit-exact only with the norms of
    # the oracle's convention (the float rounding of the double sum in column order)
    rng = np.random.default_rng(D)
    X = (rng.standard_normal((300, D)) * 10.0 ** rng.uniform(-6, 6, (300, 1))).astype(np.float32)
    X[::7] = rng.integers(0, 256, X[::7].shape)
    X[5] = 0.0
    Qs = rng.standard_normal((40, D)).astype(np.float32)
    d, i, st = run(engine, X, Qs, 30, algo=engine.ALGO_SIMT, rerank=False)
    od, oi = oracle.knn_gemm(X, Qs, 30)
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_array_equal(d, od)


@pytest.mark.parametrize("Q", [1, 129, 256, 300])
@pytest.mark.parametrize("N,D", [(16_385, 257), (33_000, 300), (40_001, 700)])
def test_wide_rows_narrow_dense_tiles(engine, oracle, N, D, Q):
    # rows wider than 256 columns: a seeding pass of few tiles takes 128-row tiles, of more 256-row ones
    import torch
    rng = np.random.default_rng(N + Q)
    X = rng.standard_normal((N, D), dtype=np.float32)
    Qs = rng.standard_normal((Q, D), dtype=np.float32)
    d, i = engine.search(torch.from_numpy(X).cuda(), torch.from_numpy(Qs).cuda(), 20)
    st = engine.last_stats()
    assert st["scan"] == 1 and engine.last_fixups() <= 1
    sub = rng.choice(Q, min(Q, 20), replace=False)
    od, oi = oracle.knn_gemm(X, Qs[sub], 20, kp=st["kp"], rerank=True)
    np.testing.assert_array_equal(i.cpu().numpy()[sub], oi)
    np.testing.assert_array_equal(d.cpu().numpy()[sub], od)
