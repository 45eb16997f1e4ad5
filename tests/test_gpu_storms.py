"""Threshold scans in which some queries append whole tiles: most rows and most queries are zero, so a zero query's
threshold lets every zero row pass and its candidates overflow (the fix-up answers it).  Its warp spends long in
appends; the other queries of the warp must lose nothing by it.  Every kind of key, narrow and wide kernels:
each remaining query gets what it gets beside none of them, and in the exact form what FP64 distances say."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rows(g, n, D, ints):
    import torch
    x = torch.zeros((n, D), device="cuda")
    x[:, :5] = torch.randn((n, 5), generator=g, device="cuda")
    if ints:
        x = (x * 20).round()
    x[torch.rand(n, generator=g, device="cuda") < 0.6] = 0
    return x


@pytest.mark.parametrize("form,N,Q,D,k", [("fp16", 9000, 3000, 5, 20), ("fp16", 22159, 1765, 6, 45), ("fp16", 150_000, 3000, 96, 20),
                                          ("fp16 three chunks", 40_000, 2000, 190, 20), ("fp16 wide", 30_000, 2000, 300, 20),
                                          ("tf32", 30_000, 2000, 6, 64), ("tf32 wide", 30_000, 2000, 150, 64),
                                          ("int", 150_000, 3000, 40, 20), ("bf16", 140_000, 3000, 64, 20),
                                          ("fp8", 60_000, 3000, 100, 20), ("fp8", 60_000, 3000, 200, 20)])
def test_queries_beside_overflowing_ones(engine, form, N, Q, D, k):
    import torch
    g = torch.Generator(device="cuda").manual_seed(N + D)
    c, q = rows(g, N, D, form == "int"), rows(g, Q, D, form == "int")
    kw = {"tf32": {"kp": k}, "tf32 wide": {"kp": k}, "bf16": {"precision": engine.PREC_BF16, "shortlist": 4},
          "fp8": {"precision": engine.PREC_FP8, "shortlist": 8}}.get(form, {})
    nz = (q != 0).any(1)
    d0, i0 = engine.search(c, q[nz].contiguous(), k, **kw)
    assert engine.last_stats()["scan"] == 1 or N < 16384
    alone = engine.last_fixups()
    exact = torch.cat([torch.topk(((x[:, None].double() - c[None, :, :5].double()) ** 2).sum(2), k, largest=False).values
                       for x in q[nz][:, :5].split(30)])
    for _ in range(6):
        d, i = engine.search(c, q, k, **kw)
        assert engine.last_stats()["scan"] == 1
        # (a zero query sees more zero rows than its candidates can hold)
        assert engine.last_fixups() >= int((~nz).sum())
        d, i = d[nz], i[nz]
        if form in ("bf16", "fp8"):
            # (a query that fails over is ranked by other keys)
            assert (i != i0).any(1).sum().item() <= 2 * (engine.last_fixups() - int((~nz).sum()) + alone)
        else:
            assert (d.double() <= exact * (1 + 1e-4) + 1e-9).all()
