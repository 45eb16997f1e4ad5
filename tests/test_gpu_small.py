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


@pytest.mark.parametrize("N,Q,D,k", [(10000, 100, 300, 10), (12000, 2600, 130, 10), (8000, 100, 64, 200), (3000, 60, 1024, 5),
                                     (16000, 40, 2048, 64), (5000, 40, 200, 493), (16000, 600, 530, 300)])
@pytest.mark.parametrize("offset", [0, 20, 80])
def test_split_keys_are_no_further_off_than_fp32_keys(engine, N, Q, D, k, offset):
    # wide rows and long shortlists: FP32 keys without the split-key paths.  A common offset costs the keys
    # their low bits: a shortlist that is not certain to hold the neighbours is replaced by that of FP32 keys
    import torch
    g = torch.Generator(device="cuda").manual_seed(N + D)
    c = torch.rand((N, D), generator=g, device="cuda") + offset
    q = torch.rand((Q, D), generator=g, device="cuda") + offset
    d, i, d0, i0, st = both(engine, c, q, k)
    n = min(Q, 60)
    ex = torch.stack([torch.topk(((x - c.double()) ** 2).sum(1), k, largest=False).values for x in q[:n].double()])
    far, far0 = ((t[:n].double() / ex).max().item() for t in (d, d0))
    assert far <= max(far0, 1 + DIST_REL)
    if offset == 0:
        # distances in FP32 and FP64 may order near-ties differently, nothing else
        assert far < 1 + DIST_REL


@pytest.mark.parametrize("N,Q,D,k", [(9000, 70, 200, 10), (5000, 3000, 600, 4), (4000, 400, 40, 150)])
def test_ties_across_the_end_of_a_split_key_shortlist(engine, N, Q, D, k):
    # equal distances inside and outside the shortlist: the lowest indices, as from FP32 keys
    import torch
    g = torch.Generator(device="cuda").manual_seed(N)
    c = torch.rand((N, D), generator=g, device="cuda")
    c[N // 3:N // 3 + 700] = c[5]
    q = torch.rand((Q, D), generator=g, device="cuda")
    q[::7] = c[5]
    d, i, d0, i0, st = both(engine, c, q, k)
    assert torch.equal(i, i0) and torch.equal(d, d0)


@pytest.mark.parametrize("N,Q,D", [(9000, 20, 200), (40, 20, 9000), (9000, 300, 1000)])
def test_infinite_queries_of_wide_rows(engine, N, Q, D):
    import torch
    g = torch.Generator(device="cuda").manual_seed(N)
    c, q = torch.randn((N, D), generator=g, device="cuda"), torch.randn((Q, D), generator=g, device="cuda")
    q[3, 1], q[4, 2], q[5, 0], q[6, 7] = float("inf"), float("-inf"), float("nan"), 3e38
    d, i, d0, i0, st = both(engine, c, q, 9)
    assert torch.equal(i, i0) and torch.equal(d, d0)


@pytest.mark.parametrize("N,Q,D", [(9000, 3000, 200), (9000, 30, 200), (3000, 9, 20)])
def test_index_without_copies(engine, N, Q, D):
    # wide rows are searched on the CUDA cores, which need no copies; others are refused
    import torch
    g = torch.Generator(device="cuda").manual_seed(N + Q)
    c, q = torch.rand((N, D), generator=g, device="cuda"), torch.rand((Q, D), generator=g, device="cuda")
    ix = engine.Index(c, tf32=False)
    if D > 128:
        d, i = ix.search(q, 10)
        d0, i0 = engine.search(c, q, 10, pilot=False)
        assert torch.equal(i, i0) and torch.equal(d, d0)
    else:
        with pytest.raises(engine.KnnsError):
            ix.search(q, 10)
    ix.close()


@pytest.mark.parametrize("N,Q,D,most", [(2, 400_000, 300, 400e6), (40, 300_000, 200, 400e6)])
def test_workspace_of_many_queries(engine, N, Q, D, most):
    # rows of keys are padded to whole tiles: a handful of corpus rows must not cost a million queries half a
    # kilobyte each (a fresh process: the engine's buffers only grow)
    import subprocess
    import sys
    code = ("import sys; sys.path.insert(0, 'knn-toolbox_gb300')\nimport torch, cuknns\n"
            "g = torch.Generator(device='cuda').manual_seed(3)\n"
            f"c, q = torch.rand(({N}, {D}), generator=g, device='cuda'), torch.rand(({Q}, {D}), generator=g, device='cuda')\n"
            "d, i = cuknns.search(c, q, 2)\nn = cuknns.last_stats()['workspace_bytes']\n"
            "d0, i0 = cuknns.search(c, q, 2, pilot=False)\nassert torch.equal(i, i0) and torch.equal(d, d0)\nprint(n)")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert int(r.stdout.split()[-1]) < most


@pytest.mark.parametrize("N,Q,D", [(9000, 3000, 40), (3000, 200, 90), (500, 20, 7)])
def test_infinite_queries_of_narrow_rows(engine, N, Q, D):
    # split keys of such a query are NaN: no results, whichever path the number of queries takes
    import torch
    g = torch.Generator(device="cuda").manual_seed(N)
    c, q = torch.randn((N, D), generator=g, device="cuda"), torch.randn((Q, D), generator=g, device="cuda")
    q[3, 1], q[4, 2], q[5, 0] = float("inf"), float("-inf"), float("nan")
    d, i, d0, i0, st = both(engine, c, q, 9)
    assert (i[3:6] == -1).all() and torch.isinf(d[3:6]).all()
    assert torch.equal(i, i0) and torch.equal(d, d0)


@pytest.mark.parametrize("N,Q,D,k", [(30, 140_000, 3, 10), (128, 131_073, 1, 5), (129, 131_073, 1, 5), (1, 300_000, 9, 1), (20, 32_769, 6, 3), (20, 32_768, 6, 3)])
def test_a_handful_of_values_and_very_many_queries(engine, N, Q, D, k):
    import torch
    g = torch.Generator(device="cuda").manual_seed(N)
    c, q = torch.rand((N, D), generator=g, device="cuda"), torch.rand((Q, D), generator=g, device="cuda")
    d, i, d0, i0, st = both(engine, c, q, k)
    assert torch.equal(i, i0) and torch.equal(d, d0)
