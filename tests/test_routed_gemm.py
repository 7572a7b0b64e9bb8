"""The grouped GEMM (route plan + one decode per tile of pairs) against the routed GEMV, one decode per pair: the same float32 sums
up to the fp16 hi/lo split of the activations.  Sizes at the edges: an expert with more pairs than a tile holds, experts without
pairs, an absent expert, route entries outside the tables, a single 128-column block, rows of one and of many blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", (2, 3, 4, 5, 6, 8))
@pytest.mark.parametrize("m,n,E,T,k", ((128, 128, 3, 1, 1), (256, 384, 5, 7, 3), (384, 128, 4, 40, 2), (128, 2048, 70, 9, 4)))
def test_grouped_gemm_equals_routed_gemv(K, m, n, E, T, k):
    from htr_b200 import ops, wire

    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(K * m + n + T)
    experts = [wire.random_packed(m, n, K, seed=31 * e + K, device=dev) for e in range(E)]
    absent = E - 1 if E > 1 else -1
    tables = [torch.tensor([0 if e == absent else experts[e][i].data_ptr() for e in range(E)], dtype=torch.int64, device=dev) for i in range(4)]
    route = torch.randint(0, E, (T * k,), generator=g)
    if T * k > 20:
        route[:18] = 1                                            # more pairs than one tile holds
        route[-1], route[-2] = E, -3                              # outside the tables
    route = route.to(dev)
    plan = ops.route_plan(route, tables)
    for dtype, tol in ((torch.float32, 5e-5), (torch.bfloat16, 1e-3), (torch.float16, 3e-4)):
        x = (torch.randn(T, n, generator=g) * torch.where(torch.rand(n, generator=g) < 0.02, 3000.0, 1.0)).to(dtype).to(dev)
        want, got = (torch.full((T * k, m), 7.0, dtype=dtype, device=dev) for _ in range(2))
        ops.linear_routed(x, route, tables, m // 16, n // 16, K, x_div=k, out=want)
        assert ops.linear_routed_gemm(x, plan, T * k, tables, m // 16, n // 16, K, x_div=k, out=got) is got
        assert float((got.float() - want.float()).norm() / want.float().norm()) <= tol
        skipped = (route < 0) | (route >= E) | (route == absent)
        assert bool((got[skipped] == 7.0).all())                  # untouched, as the routed GEMV leaves them
        again = torch.empty_like(got)
        ops.linear_routed_gemm(x, plan, T * k, tables, m // 16, n // 16, K, x_div=k, out=again)
        assert torch.equal(again[~skipped], got[~skipped])
    gu = torch.randn(T * k, 2 * n, generator=g).bfloat16().to(dev)
    want = ops.linear_routed(gu, route, tables, m // 16, n // 16, K, prologue=ops.PROLOGUE_SWIGLU)
    got = ops.linear_routed_gemm(gu, plan, T * k, tables, m // 16, n // 16, K, prologue=ops.PROLOGUE_SWIGLU)
    if bool((~skipped).any()):
        assert float((got[~skipped].float() - want[~skipped].float()).norm() / want[~skipped].float().norm()) <= 1e-3
    assert all(c == 0 for c in ops.gemm_error_codes())
    assert ops.route_plan(torch.zeros(5000, dtype=torch.int64, device=dev), tables) is None
