"""Double-precision library (the reference's libcuknn_double) and the file-based
drivers knn_test / knn_test_double (src/knnTest.cu interface).

Bar for the double library: the exact FP64 top-k by (direct-difference distance,
index) -- indices and distances identical to the FP64 oracle of the FP64 inputs
(oracle_knn_f64d: the same distance, summed in d order with separate multiply
and add).  The reference's own double tests hold distances to a 1e-7 / 1e-6
norm tolerance (demo/Testbin.m:86, demo/knnTestDouble.m:30); identity is
stronger.  The float driver is held to the parity bars of test_gpu_parity.py.
"""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BUILD = os.path.join(ROOT, "knn-toolbox_gb300", "_build")


@pytest.mark.parametrize("N,Q,D,k", [(3000, 40, 17, 5), (20000, 130, 128, 100), (150_000, 64, 96, 32),
                                     (500, 7, 3, 500)])
def test_double_library_exact(engine, oracle, N, Q, D, k):
    rng = np.random.default_rng(N + D)
    X = rng.standard_normal((N, D))
    Qs = rng.standard_normal((Q, D))
    d, i = engine.search_host_f64(X, Qs, k)
    od, oi = oracle.knn_f64d(X, Qs, k)
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_array_equal(d, od)


def test_double_library_near_duplicates_fall_back(engine, oracle):
    # 200 rows per base vector that differ below FP32 resolution: more FP32 ties than the
    # shortlist holds, so the acceptance test fails and the FP64 search decides
    rng = np.random.default_rng(3)
    base = rng.standard_normal((50, 16))
    X = np.repeat(base, 200, axis=0) + 1e-12 * rng.standard_normal((10000, 16))
    Qs = base[:20] + 1e-13 * rng.standard_normal((20, 16))
    k = 60
    d, i = engine.search_host_f64(X, Qs, k)
    od, oi = oracle.knn_f64d(X, Qs, k)
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_array_equal(d, od)


def test_double_dropin(engine, oracle):
    rng = np.random.default_rng(4)
    X = rng.random((6000, 50))
    Qs = rng.random((33, 50))
    vals, idxs, t = engine.gpuknnsBitonic_f64(Qs, X, 8)
    od, oi = oracle.knn_f64d(X, Qs, 8)
    np.testing.assert_array_equal(idxs.astype(np.int64), oi)
    np.testing.assert_array_equal(vals, od)
    assert t > 0


@pytest.mark.parametrize("double", [False, True])
def test_file_driver(engine, oracle, tmp_path, double):
    rng = np.random.default_rng(5)
    dt = np.float64 if double else np.float32
    N, Q, D, k = 4096, 60, 20, 12
    X = rng.random((N, D)).astype(dt)
    Qs = rng.random((Q, D)).astype(dt)
    X.tofile(tmp_path / "data.bin")
    Qs.tofile(tmp_path / "queries.bin")
    exe = os.path.join(BUILD, "knn_test_double" if double else "knn_test")
    r = subprocess.run([exe, "data.bin", "queries.bin", str(N), str(Q), str(D), str(k)], cwd=tmp_path,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "Time Elapsed:" in r.stdout
    dist = np.fromfile(tmp_path / "KNNdist.bin", dt).reshape(Q, k)   # demo/importData.m: [k Q]
    idx = np.fromfile(tmp_path / "KNNidx.bin", dt).reshape(Q, k)
    if double:
        od, oi = oracle.knn_f64d(X, Qs, k)
        np.testing.assert_array_equal(idx.astype(np.int64), oi)
        np.testing.assert_array_equal(dist, od)
    else:
        oracle.check_parity(X, Qs, k, dist, idx.astype(np.int64), gap_rel=1e-6, dist_rel=1e-5)
    # a short input file is an error, not a search of uninitialised memory
    r = subprocess.run([exe, "data.bin", "queries.bin", str(N + 1), str(Q), str(D), str(k)], cwd=tmp_path,
                       capture_output=True, text=True)
    assert r.returncode == 1


@pytest.mark.parametrize("N,Q,D,k", [(70, 5, 7, 70), (300, 3, 9, 1), (20000, 64, 33, 256), (20000, 65, 300, 100),
                                     (600, 10, 8, 512), (30000, 1, 128, 128)])
@pytest.mark.parametrize("scale", [1.0, 1e-20, 1e15])
def test_double_library_candidate_bound(engine, oracle, N, Q, D, k, scale):
    # the FP64 distances are computed for the candidates within the FP32 error bound of the k-th only
    # (all of them where the shortlist covers the corpus); scales whose squares leave the float range
    # fall back to the brute force
    rng = np.random.default_rng(N + D)
    X = rng.standard_normal((N, D)) * scale
    X[N // 2:N // 2 + 3] = X[:3]            # ties
    Qs = rng.standard_normal((Q, D)) * scale
    d, i = engine.search_host_f64(X, Qs, k)
    od, oi = oracle.knn_f64d(X, Qs, k)
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_array_equal(d, od)


@pytest.mark.parametrize("lo,hi", [(-150, -120), (-30, 20), (110, 130)])
def test_double_library_rounding_to_float(engine, oracle, lo, hi):
    # rows halfway between two floats, zeros, and magnitudes below, across and above FP32's normal range
    rng = np.random.default_rng(abs(hi))
    X = rng.standard_normal((3000, 12)).astype(np.float32).astype(np.float64)
    X *= 1.0 + 2.0 ** -24 * rng.integers(-1, 2, X.shape)
    X *= 2.0 ** rng.integers(lo, hi, (3000, 1))
    X[rng.random(X.shape) < 0.1] = 0.0
    Qs = X[::100] * (1.0 + 2.0 ** -30)
    d, i = engine.search_host_f64(X, Qs, 10)
    od, oi = oracle.knn_f64d(X, Qs, 10)
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_array_equal(d, od)


@pytest.mark.parametrize("N,D,k,scale", [(40, 6, 10, 1e20), (70, 9, 70, 1e20), (5, 3, 5, 1e25), (42, 300, 10, 1e20)])
def test_double_library_distances_past_the_float_range(engine, oracle, N, D, k, scale):
    # the FP32 shortlist could hold every row (N <= max(k + 32, 2 k)), but holds none of these
    rng = np.random.default_rng(N)
    X, Qs = rng.standard_normal((N, D)) * scale, rng.standard_normal((7, D)) * scale
    d, i = engine.search_host_f64(X, Qs, k)
    od, oi = oracle.knn_f64d(X, Qs, k)
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_array_equal(d, od)


@pytest.mark.parametrize("N", [100, 20000])
def test_double_library_norms_past_the_float_range(engine, oracle, N):
    # the nearest rows have squared norms above 3.4e38, so no FP32 key, but small distances; every other
    # row has both
    X = np.concatenate([np.linspace(1.5e19, 1.8e19, N - 10), np.linspace(1.846e19, 1.86e19, 10)])[:, None]
    Qs = np.array([[1.84e19], [-1e19]])
    d, i = engine.search_host_f64(X, Qs, 10)
    od, oi = oracle.knn_f64d(X, Qs, 10)
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_array_equal(d, od)


@pytest.mark.parametrize("N", [11, 36])  # k + 32 rows and fewer
def test_double_library_infinite_query_of_a_covered_corpus(engine, N):
    # no distance is finite; the rows that the FP32 shortlist holds come back by index
    rng = np.random.default_rng(N)
    X, Qs = rng.random((N, 412)) + 0.1, rng.random((3, 412))
    X[N - 1, 5] = np.inf
    Qs[1, 3] = np.inf
    d, i = engine.search_host_f64(X, Qs, 4)
    assert np.isinf(d[1]).all()
    np.testing.assert_array_equal(i[1], np.arange(4))
    assert np.isfinite(d[[0, 2]]).all()
