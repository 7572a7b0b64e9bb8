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


@pytest.mark.parametrize("dtype,tol", ((torch.float32, 5e-5), (torch.bfloat16, 1e-3)))
def test_pairs_of_any_magnitude(dtype, tol):
    """Rows of every magnitude side by side in one tile, plain and behind SwiGLU (whose products are where small rows come from): each row as
    near to the routed GEMV, which stages float32 values, as ordinary rows are above."""
    from htr_b200 import ops, wire

    dev, m, n, E = torch.device("cuda:0"), 256, 384, 2
    experts = [wire.random_packed(m, n, 3, seed=7 + e, device=dev) for e in range(E)]
    tables = [torch.tensor([experts[e][i].data_ptr() for e in range(E)], dtype=torch.int64, device=dev) for i in range(4)]
    g = torch.Generator().manual_seed(3)
    scales = torch.tensor([10.0 ** p for p in (0, -3, -4, -5, -6, -8, -12, -20, -30, 4, 20, 30, -1, 0)], dtype=torch.float64)
    T = scales.numel()
    route = (torch.arange(T) % E).to(dev)
    plan = ops.route_plan(route, tables)
    x = (torch.randn(T, n, generator=g).double() * scales[:, None]).to(dtype).to(dev)

    def close(got, want):
        s = want.double().abs().amax(dim=1, keepdim=True)
        err = ((got.double() - want.double()) / s).norm(dim=1) / (want.double() / s).norm(dim=1)
        assert float(err.max()) <= tol, err.tolist()

    close(ops.linear_routed_gemm(x, plan, T, tables, m // 16, n // 16, 3), ops.linear_routed(x, route, tables, m // 16, n // 16, 3))
    if dtype == torch.bfloat16:
        gu = torch.cat([x * 0 + torch.randn(T, n, generator=g).to(dtype).to(dev), x], dim=1).contiguous()
        close(ops.linear_routed_gemm(gu, plan, T, tables, m // 16, n // 16, 3, prologue=ops.PROLOGUE_SWIGLU),
              ops.linear_routed(gu, route, tables, m // 16, n // 16, 3, prologue=ops.PROLOGUE_SWIGLU))
    assert all(c == 0 for c in ops.gemm_error_codes())


@pytest.mark.parametrize("m,n", ((128, 128), (256, 4096)))
def test_plans_without_a_pair_between_others(m, n):
    """Steps of which every pair goes to an expert outside the tables (an empty plan: no thread block has work) between ordinary ones that use
    the same scratch: the empty ones write nothing, the others give the bits that they give alone."""
    from htr_b200 import ops, wire

    dev, E, T = torch.device("cuda:0"), 4, 24
    experts = [wire.random_packed(m, n, 3, seed=5 + e, device=dev) for e in range(E)]
    tables = [torch.tensor([experts[e][i].data_ptr() for e in range(E)], dtype=torch.int64, device=dev) for i in range(4)]
    g = torch.Generator().manual_seed(n)
    x = torch.randn(T, n, generator=g).bfloat16().to(dev)
    some, none = (torch.arange(T) % E).to(dev), torch.full((T,), E, dtype=torch.int64, device=dev)

    def step(route, out):
        return ops.linear_routed_gemm(x, ops.route_plan(route, tables), T, tables, m // 16, n // 16, 3, out=out)

    want = step(some, torch.empty((T, m), dtype=torch.bfloat16, device=dev))
    torch.cuda.synchronize()
    outs = [(step(none, torch.full((T, m), 7.0, dtype=torch.bfloat16, device=dev)), step(some, torch.empty((T, m), dtype=torch.bfloat16, device=dev)))
            for _ in range(20)]
    for empty, full in outs:
        assert bool((empty == 7.0).all()) and torch.equal(full, want)
    assert all(c == 0 for c in ops.gemm_error_codes())


def test_pairs_of_an_expired_wait_are_nan():
    """One tile of activations is withheld: its row block of its experts' pairs comes out as NaN, and the row block behind it in the same thread
    block's run (13 blocks, more than there are stages, so that the decode warps' own waits run out as well); all others keep their bits."""
    from htr_b200 import _lib, ops, wire

    dev, m, n, E, T = torch.device("cuda:0"), 256, 4096, 32, 64
    experts = [wire.random_packed(m, n, 3, seed=60 + e, device=dev) for e in range(E)]
    tables = [torch.tensor([experts[e][i].data_ptr() for e in range(E)], dtype=torch.int64, device=dev) for i in range(4)]
    route = (torch.arange(T) % E).to(dev)                         # tile e holds the two pairs of expert e
    x = torch.randn(T, n, generator=torch.Generator().manual_seed(1)).bfloat16().to(dev)
    plan = ops.route_plan(route, tables)
    want = ops.linear_routed_gemm(x, plan, T, tables, m // 16, n // 16, 3)
    torch.cuda.synchronize()
    for block in (0, 19 * 64 + 3, 19 * 64 + 40):
        _lib.lib.htr_gemm_withhold_tile(block)
        try:
            got = ops.linear_routed_gemm(x, plan, T, tables, m // 16, n // 16, 3)
        finally:
            _lib.lib.htr_gemm_withhold_tile(-1)
        codes = ops.gemm_error_codes()
        assert any(c != 0 for c in codes)
        for ws in ops._GEMM_WS.values():
            ws.zero_()
        unit = block // (n // 128)                                # row block, counted through the tiles
        for at in range(E * 2):
            rows, cols = route == at // 2, slice(128 * (at % 2), 128 * (at % 2) + 128)
            lost = bool(torch.isnan(got[rows][:, cols]).all())
            assert lost or torch.equal(got[rows][:, cols], want[rows][:, cols])
            assert lost if at == unit else not lost or at == unit + 1
    assert torch.equal(ops.linear_routed_gemm(x, plan, T, tables, m // 16, n // 16, 3), want)
