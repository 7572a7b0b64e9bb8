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


@pytest.mark.parametrize("dtype,tol", ((torch.float32, 5e-6), (torch.bfloat16, 4e-3)))
@pytest.mark.parametrize("m,n", ((128, 16384), (1024, 2048), (2176, 5760)))
def test_one_row_of_any_magnitude(coracle, m, n, dtype, tol):
    """Byte sums are multiplied as subnormal numbers with activations under a power-of-two factor, one per thread block: it must follow the
    range of float32 and bf16, also where thread blocks of one launch choose different ones (columns of different magnitude)."""
    from htr_b200 import ops, wire

    dev = torch.device("cuda:0")
    qw, sc, su, sv = wire.random_packed(m, n, 4, seed=m + n)
    d = [t.to(dev) for t in (qw, sc, su, sv)]
    g = torch.Generator().manual_seed(n)
    x = torch.randn(1, n, generator=g)
    for left, right in ((-36, -36), (-30, -30), (-20, -20), (-13, -11), (11, 13), (16, 16), (25, 25), (33, 33), (30, -30), (-25, 0), (0, 14), (13, 30), (-20, -36)):
        xs = x.double().clone()
        xs[:, :n // 2] *= 10.0 ** left
        xs[:, n // 2:] *= 10.0 ** right
        xs = xs.float().to(dtype)
        ref = coracle.linear(xs.float().numpy(), qw.numpy(), sc.numpy(), su.numpy(), sv.numpy())
        y = ops.linear(xs.to(dev), *d)
        assert bool(torch.isfinite(y).all()) and torch.equal(ops.linear(xs.to(dev), *d), y)
        s = float(np.abs(ref).max())                                  # (squares of the ends would leave float64's sums of float32)
        assert rel(y.float().cpu().numpy() / s, ref / s) <= tol, (left, right)
    zero = ops.linear(torch.zeros(1, n, dtype=dtype, device=dev), *d)
    assert not bool(zero.any())
    for bad in (float("inf"), float("nan")):
        xs = x.clone()
        xs[0, 17] = bad
        assert not bool(torch.isfinite(ops.linear(xs.to(dtype).to(dev), *d)).any())


@pytest.mark.parametrize("n", (512, 2560, 2688, 5120, 5248, 12800, 12928))
@pytest.mark.parametrize("m", (2048, 4864))
def test_one_row_at_the_widths_where_the_staging_changes(coracle, m, n):
    """A warp stages one, two, five or seven blocks of the row at most, and runs begin anywhere in a row block (their boundaries come from
    a multiplication with the reciprocal)."""
    from htr_b200 import ops, wire

    dev = torch.device("cuda:0")
    qw, sc, su, sv = wire.random_packed(m, n, 3, seed=m + n)
    d = [t.to(dev) for t in (qw, sc, su, sv)]
    x = torch.randn(1, n, generator=torch.Generator().manual_seed(n))
    ref = coracle.linear(x.numpy(), qw.numpy(), sc.numpy(), su.numpy(), sv.numpy())
    assert rel(ops.linear(x.to(dev), *d).cpu().numpy(), ref) <= 5e-6
