"""The one-row GEMV of dependent launches (packed_gemv1.cuh) at the edges of its runs: fewer blocks than SMs, runs that cross one, two and
many row blocks, one block per row, ragged widths, all types and prologues, against the CPU oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a.astype(np.float64) - b.astype(np.float64)) / np.linalg.norm(b.astype(np.float64)))


@pytest.mark.parametrize("K", (2, 3, 4, 5, 6, 8))
@pytest.mark.parametrize("m,n", ((128, 16384), (16384, 128), (1024, 2048), (1536, 1408), (38144, 256), (2176, 5760)))
def test_one_row(coracle, K, m, n):
    from htr_b200 import ops, wire

    dev = torch.device("cuda:0")
    qw, sc, su, sv = wire.random_packed(m, n, K, seed=K + m + n)
    d = [t.to(dev) for t in (qw, sc, su, sv)]
    g = torch.Generator().manual_seed(m)
    x, bias = torch.randn(1, n, generator=g), torch.randn(m, generator=g)
    x[0, :: 131] *= 500.0
    ref = coracle.linear(x.numpy(), qw.numpy(), sc.numpy(), su.numpy(), sv.numpy(), bias=bias.numpy())
    y = ops.linear(x.to(dev), *d, bias.to(dev))
    assert rel(y.cpu().numpy(), ref) <= 5e-6 and torch.equal(ops.linear(x.to(dev), *d, bias.to(dev)), y)
    plain = coracle.linear(x.numpy(), qw.numpy(), sc.numpy(), su.numpy(), sv.numpy())
    for scale in (1e-12, 1e9):                                        # the subnormal products keep their bits at either end
        z = ops.linear((x * scale).to(dev), *d)
        assert rel(z.cpu().numpy() / scale, plain) <= 5e-6
    ones = torch.ones(1, n) * (1 - 2 * torch.from_numpy(np.unpackbits(su.numpy(), bitorder="little").astype(np.float32)))   # one spike per block
    assert rel(ops.linear(ones.to(dev), *d).cpu().numpy(), coracle.linear(ones.numpy(), qw.numpy(), sc.numpy(), su.numpy(), sv.numpy())) <= 5e-6
    for dt in (torch.bfloat16, torch.float16):
        xb = torch.randn(1, n, generator=g).to(dt)
        yb = ops.linear(xb.to(dev), *d)
        assert rel(yb.float().cpu().numpy(), coracle.linear(xb.float().numpy(), qw.numpy(), sc.numpy(), su.numpy(), sv.numpy())) <= 4e-3
