"""Searches of corpora below 16,384 rows that nothing but the defaults is asked of: the direct kernel
(exact distances of every row), the dense keys of the FP16-split scan with their selection, in one or
several chunks of queries, and the threshold scan for many queries -- against the oracle, and against
the shortlist kernel that the same searches ran on (pilot = False still does).  Forms of the call: odd
sizes and pitches, k of every row, ties, rows that are not finite, an index, host buffers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GAP = 1e-6
DIST_REL = 1e-5


def both(engine, c, q, k, **kw):
    d, i = engine.search(c, q, k, **kw)
    st = engine.last_stats()
    d0, i0 = engine.search(c, q, k, pilot=False, **kw)
    return d, i, d0, i0, st


@pytest.mark.parametrize("N,Q,D,k", [(1, 1, 1, 1), (7, 3, 2, 7), (31, 5, 8, 4), (33, 40, 9, 20), (500, 152, 33, 10),
                                     (1023, 153, 15, 100), (4100, 9, 36, 5), (2000, 60, 108, 300),
                                     (129, 300, 640, 16), (3000, 70, 250, 10), (4097, 129, 128, 50),
                                     (9001, 385, 257, 10), (16383, 40, 64, 100), (15000, 3, 1025, 7), (12000, 384, 63, 200)])
@pytest.mark.parametrize("kind", ["normal", "int"])
def test_against_the_oracle_and_the_shortlist_kernel(engine, oracle, N, Q, D, k, kind):
    import torch
    rng = np.random.default_rng(N + Q + D)
    gen = (lambda n: rng.integers(0, 16, (n, D)).astype(np.float32)) if kind == "int" else \
          (lambda n: rng.standard_normal((n, D), dtype=np.float32))
    X, Qs = gen(N), gen(Q)
    # row pitches of their own
    c = torch.from_numpy(np.pad(X, ((0, 0), (0, 3)))).cuda()[:, :D]
    q = torch.from_numpy(np.pad(Qs, ((0, 0), (0, 1)))).cuda()[:, :D]
    d, i, d0, i0, st = both(engine, c, q, k)
    assert st["scan"] == 0
    assert torch.equal(i, i0) and torch.equal(d, d0)
    od, oi = oracle.knn_gemm(X, Qs, k, kp=st["kp"], rerank=True)
    if kind == "int":
        np.testing.assert_array_equal(i.cpu().numpy(), oi)
        np.testing.assert_array_equal(d.cpu().numpy(), od)
    else:
        oracle.check_parity(X, Qs, k, d.cpu().numpy(), i.cpu().numpy(), ref_idx=oi, gap_rel=GAP, dist_rel=DIST_REL,
                            dist_abs=1e-6)


@pytest.mark.parametrize("N,Q,D", [(3000, 9000, 64), (8191, 3300, 20), (6000, 4500, 300), (8192, 3200, 64), (16000, 1700, 130)])
def test_many_queries(engine, N, Q, D):
    # more keys than are held at once: chunks of queries, or the threshold scan from 8,192 rows
    import torch
    g = torch.Generator(device="cuda").manual_seed(N)
    c, q = torch.rand((N, D), generator=g, device="cuda"), torch.rand((Q, D), generator=g, device="cuda")
    d, i, d0, i0, st = both(engine, c, q, 12)
    assert st["scan"] == (1 if N >= 8192 else 0)
    assert torch.equal(i, i0) and torch.equal(d, d0)


@pytest.mark.parametrize("N,D", [(900, 12), (5000, 90)])
def test_rows_that_are_not_finite(engine, N, D):
    # fewer finite rows than k: they come first, then (+inf, -1)
    import torch
    g = torch.Generator(device="cuda").manual_seed(N)
    c, q = torch.rand((N, D), generator=g, device="cuda"), torch.rand((20, D), generator=g, device="cuda")
    c[10:, 3] = float("nan")
    c[20:40, 3] = float("inf")
    d, i, d0, i0, st = both(engine, c, q, 16)
    assert (i[:, :10] >= 0).all() and (i[:, :10] < 10).all()
    assert (i[:, 10:] == -1).all() and torch.isinf(d[:, 10:]).all()
    assert torch.equal(i, i0) and torch.equal(d, d0)


@pytest.mark.parametrize("N,D,Q,k", [(1000, 16, 30, 10), (6000, 100, 200, 10), (3000, 64, 100, 128)])
def test_index_host_and_dropin_agree(engine, N, D, Q, k):
    import torch
    rng = np.random.default_rng(N)
    X, Qs = rng.random((N, D), dtype=np.float32), rng.random((Q, D), dtype=np.float32)
    c, q = torch.from_numpy(X).cuda(), torch.from_numpy(Qs).cuda()
    d, i = engine.search(c, q, k)
    d, i = d.cpu().numpy(), i.cpu().numpy()
    ix = engine.Index(c)
    for rerank in (True, False):
        dx, ixx = ix.search(q, k, rerank=rerank)
        if rerank:
            np.testing.assert_array_equal(ixx.cpu().numpy(), i)
            np.testing.assert_array_equal(dx.cpu().numpy(), d)
    ix.close()
    dh, ih = engine.search_host(X, Qs, k)
    np.testing.assert_array_equal(ih, i)
    np.testing.assert_array_equal(dh, d)
    v, f, _ = engine.gpuknnsBitonic(Qs, X, k)
    np.testing.assert_array_equal(f, i.astype(np.float32))
    np.testing.assert_array_equal(v, d)
    # without the exact form's copies an index refuses the exact form, whatever the size
    bare = engine.Index(c, tf32=False)
    with pytest.raises(engine.KnnsError):
        bare.search(q, k)
    bare.close()
