"""The tensor-core GEMM at the sizes where its launch plan changes form (clusters of each size, one thread block per row block, even
runs across row blocks), its padded entry, and the route of small 16-bit batches, against the CPU oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a.astype(np.float64) - b.astype(np.float64)) / max(np.linalg.norm(b.astype(np.float64)), 1e-30))


@pytest.mark.parametrize("K,m,n,M", ((4, 2048, 2048, 8), (3, 640, 2176, 200), (5, 2944, 384, 37), (2, 6144, 256, 16), (6, 9472, 128, 130),
                                     (8, 19072, 128, 33), (4, 128, 1024, 256), (3, 4096, 1024, 2), (4, 2048, 2304, 3)))
def test_gemm_plans(coracle, K, m, n, M):
    from htr_b200 import ops, wire

    dev = torch.device("cuda:0")
    qw, sc, su, sv = wire.random_packed(m, n, K, seed=m + n + M)
    d = [t.to(dev) for t in (qw, sc, su, sv)]
    x = torch.randn(M, n, generator=torch.Generator().manual_seed(M)).bfloat16()
    rows = min(M, 40)
    ref = coracle.linear(x[:rows].float().numpy(), qw.numpy(), sc.numpy(), su.numpy(), sv.numpy())
    y = ops.linear(x.to(dev), *d)
    assert rel(y[:rows].float().cpu().numpy(), ref) <= 4e-3 and torch.equal(ops.linear(x.to(dev), *d), y)
    assert all(c == 0 for c in ops.gemm_error_codes())


@pytest.mark.parametrize("dtype,tol", ((torch.bfloat16, 3e-3), (torch.float16, 5e-4)))
@pytest.mark.parametrize("n_in,m_out,n_pad,m_pad,M", ((336, 328, 384, 384, 5), (8, 8, 128, 128, 17), (1000, 520, 1024, 640, 150), (4000, 4096, 4096, 4096, 11)))
def test_padded_gemm(coracle, dtype, tol, n_in, m_out, n_pad, m_pad, M):
    from htr_b200 import ops, wire

    dev = torch.device("cuda:0")
    qw, sc, su, sv = wire.random_packed(m_pad, n_pad, 3, seed=n_in + m_out)
    g = torch.Generator().manual_seed(M)
    x, bias = torch.randn(M, n_in, generator=g).to(dtype), torch.randn(m_out, generator=g).to(dtype)
    ref = coracle.linear(torch.nn.functional.pad(x, (0, n_pad - n_in)).float().numpy(), qw.numpy(), sc.numpy(), su.numpy(), sv.numpy())[:, :m_out] + bias.float().numpy()
    y = ops.linear_padded(x.to(dev), *[t.to(dev) for t in (qw, sc, su, sv)], bias=bias.to(dev), m_out=m_out)
    assert tuple(y.shape) == (M, m_out) and rel(y.float().cpu().numpy(), ref) <= tol
