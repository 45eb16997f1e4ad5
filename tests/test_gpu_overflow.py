"""Small corpora whose squares leave the float range, on the direct kernel, against the shortlist and CUDA-core
kernels (pilot = False): rows whose norm or key ||c||^2 - 2 q.c overflows are no results, rows whose distance
alone does come back as (+inf, index)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,Q,D,k", [(24, 30, 1, 10), (20, 9, 7, 20), (600, 60, 200, 15), (30, 160, 4, 30), (900, 5, 140, 200)])
def test_squares_past_the_float_range(engine, N, Q, D, k):
    import torch
    g = torch.Generator(device="cuda").manual_seed(N + D)

    def rows(n):
        return torch.randn((n, D), generator=g, device="cuda") * 10.0 ** (torch.rand((n, 1), generator=g, device="cuda") * 2.4 + 17.2)

    c, q = rows(N), rows(Q)
    if D == 1:
        c[0], q[0] = 1e19, -1e19  # key 3e38, distance 4e38
        c[1], q[1] = 2e19, 1.9e19  # squared norm 4e38, distance 1e36
    d, i = engine.search(c, q, k)
    d0, i0 = engine.search(c, q, k, pilot=False)
    assert (torch.isinf(d0) & (i0 >= 0)).any()
    assert torch.equal(i, i0) and torch.equal(d, d0)
