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


@pytest.mark.parametrize("dtype,M,tol", ((torch.bfloat16, 4, 4e-3), (torch.float16, 3, 4e-3), (torch.bfloat16, 14, 4e-3), (torch.float32, 14, 5e-5)))
@pytest.mark.parametrize("padded", (False, True))
def test_rows_of_any_magnitude(coracle, dtype, M, tol, padded):
    """The activations reach the MMA as fp16 numbers under a scale per row: each row of a call, however small or large, keeps the accuracy of
    rows near 1 (the tolerances of the tests above), next to rows of other magnitudes and a row of zeros.  float16 stays above its subnormals."""
    from htr_b200 import ops, wire

    dev = torch.device("cuda:0")
    m, n = 2048, 2048
    qw, sc, su, sv = wire.random_packed(m, n, 4, seed=M)
    x = torch.randn(M, n, generator=torch.Generator().manual_seed(M))
    x[:, ::97] *= 10.0
    powers = (0, -3, -4) if dtype == torch.float16 else (0, -8, 30, -3, -5, -6, -12, -20, -30, -36, 8, 2, 33, 0)
    for r in range(M):
        x[r] = (x[r].double() * 10.0 ** powers[r]).float()
    if M > 4:
        x[M - 1] = 0
    x = x.to(dtype)
    d = [t.to(dev) for t in (qw, sc, su, sv)]
    n_in, m_out = (n - 40, m - 8) if padded else (n, m)
    x[:, n_in:] = 0
    ref = coracle.linear(x.float().numpy(), qw.numpy(), sc.numpy(), su.numpy(), sv.numpy())[:, :m_out]
    if padded and dtype == torch.float32:
        y = torch.empty(M, m_out, device=dev)                     # (ops keeps float32 rows of padded linears on the GEMV)
        from htr_b200 import _lib

        ws = torch.zeros(_lib.lib.htr_linear_gemm_workspace_bytes(M, m, n, 4), dtype=torch.uint8, device=dev)
        xs = x[:, :n_in].contiguous().to(dev)
        rc = _lib.lib.htr_linear_gemm_padded(xs.data_ptr(), _lib.F32, M, n_in, d[0].data_ptr(), m // 16, n // 16, 4, d[1].data_ptr(), d[2].data_ptr(),
                                             d[3].data_ptr(), None, y.data_ptr(), m_out, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0
    else:
        y = ops.linear_padded(x[:, :n_in].contiguous().to(dev), *d, m_out=m_out) if padded else ops.linear(x.to(dev), *d)
    y = y.float().cpu().numpy()
    for r in range(M):
        if not x[r].any():
            assert not y[r].any()
        else:
            s = float(np.abs(ref[r]).max())                       # (norms of the smallest rows would underflow)
            assert rel(y[r] / s, ref[r] / s) <= tol, (r, powers[r])
    assert all(c == 0 for c in ops.gemm_error_codes())


@pytest.mark.parametrize("K,m,n,rows", ((3, 19072, 128, (9, 16, 17, 255, 256)), (4, 2048, 2048, (9, 15, 64, 65, 256)), (5, 640, 2176, (1, 33, 241, 256)),
                                        (8, 128, 1024, (5, 128, 129)), (2, 32768, 256, (8, 200))))
def test_rows_of_one_row_block(coracle, K, m, n, rows):
    """Thread blocks with one row block or a part of one: the decode warps finish rows 16 at a time (per member of a cluster), each with the
    sums and scales that its lane brought.  Row counts at the edges; every row has its own magnitude, so that a mixed-up scale shows."""
    from htr_b200 import ops, wire

    dev = torch.device("cuda:0")
    qw, sc, su, sv = wire.random_packed(m, n, K, seed=m + n)
    d = [t.to(dev) for t in (qw, sc, su, sv)]
    g = torch.Generator().manual_seed(K)
    x = (torch.randn(256, n, generator=g) + torch.randn(256, 1, generator=g)) * 2.0 ** torch.randint(-12, 12, (256, 1), generator=g)
    x, bias = x.bfloat16(), torch.randn(m, generator=g).bfloat16()
    few = slice(0, 640) if m > 4096 else slice(0, m)                     # (rows of the weight that the oracle computes)
    ref = coracle.linear(x.float().numpy(), qw[:few.stop // 16].numpy(), sc[few].numpy(), su.numpy(), sv[:few.stop // 8].numpy())
    for M in rows:
        y = ops.linear(x[:M].to(dev), *d, bias.to(dev)) if M > 1 else ops.linear_padded(x[:M].to(dev), *d, bias=bias.to(dev), m_out=m)
        want = ref[:M] + bias[few].float().numpy()
        err = np.linalg.norm(y[:, few].float().cpu().numpy() - want, axis=1) / np.linalg.norm(want, axis=1)
        assert err.max() <= 4e-3, (M, int(err.argmax()), float(err.max()))
    assert all(c == 0 for c in ops.gemm_error_codes())


def transform(dtype, M, m, n, K):
    """(thread blocks per row block, thread blocks of the GEMM, four blocks per warp, slices, warps of the transform)"""
    import ctypes

    from htr_b200 import _lib

    out = (ctypes.c_int * 5)()
    _lib.check(_lib.lib.htr_linear_gemm_shape({torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}[dtype], M, m, n, K, out), "htr_linear_gemm_shape")
    return tuple(out)


TRANSFORM_SIZES = ((128, 128), (128, 384), (128, 2176), (256, 2048), (4096, 4096), (128, 8320), (4096, 6144), (4096, 12288), (128, 16512), (128, 65664),
                   (19072, 4224), (19072, 12288))
TRANSFORM_ROWS = (3, 5, 8, 9, 16, 17, 24, 37, 48, 49, 64, 65, 100, 128, 129, 200, 256)


def test_every_form_of_the_transform_is_among_the_tested():
    """Form, warps, and slices where four blocks go to a warp, over the sizes that the rule looks at."""
    def form(shape):
        return (shape[2], shape[4], shape[3] if shape[2] else 0)

    tested = {form(transform(torch.bfloat16, M, m, n, 3)) for m, n in TRANSFORM_SIZES for M in TRANSFORM_ROWS}
    every = {form(transform(torch.bfloat16, M, m, n, 3)) for m in (128, 1024, 2048, 4096, 8192, 12288, 19072) for n in
             (*range(128, 4480, 128), 5120, 6144, 8192, 8320, 10240, 12288, 16384, 16512, 65664) for M in range(2, 257)}
    assert tested == every and len(every) >= 6, (tested, every)


@pytest.mark.parametrize("m,n", TRANSFORM_SIZES)
def test_activation_transform_shapes(coracle, m, n):
    """Form, slices and warps of the activation transform change with the rows, the columns and the SMs that the GEMM leaves free: rows at the
    edges, in two types; rows of their own magnitude, so that a scale of another row shows.
    float32: the tensor cores cut the accumulator towards zero at each of a block's eight MMAs, by 2^-24 of itself on average; it grows to 1534
    |sum of the activations|, for a row three deviations out 31 times the result (148 sqrt(n)), and is half of that on average:
    8 * 2^-24 * 31 / 2 = 7.4e-6 for every block that one accumulator takes."""
    from htr_b200 import ops, wire

    dev = torch.device("cuda:0")
    qw, sc, su, sv = wire.random_packed(m, n, 3, seed=m + n)
    d = [t.to(dev) for t in (qw, sc, su, sv)]
    g = torch.Generator().manual_seed(n)
    x = torch.randn(256, n, generator=g) * 2.0 ** torch.randint(-8, 8, (256, 1), generator=g)
    ref = {dt: coracle.linear(x.to(dt).float().numpy(), qw[:8].numpy(), sc[:128].numpy(), su.numpy(), sv[:16].numpy()) for dt in (torch.bfloat16, torch.float32)}
    for dt, tol, rows in ((torch.bfloat16, 4e-3, TRANSFORM_ROWS), (torch.float32, 5e-5, (5, 17, 49, 128))):
        for M in rows:
            split = transform(dt, M, m, n, 3)[0]
            most = max(tol, 7.4e-6 * -(-(n // 128) // max(split, 1))) if dt == torch.float32 else tol
            y = ops.linear(x[:M].to(dt).to(dev), *d)[:, :128].float().cpu().numpy()
            err = np.linalg.norm(y - ref[dt][:M], axis=1) / np.linalg.norm(ref[dt][:M], axis=1)
            assert err.max() <= most, (dt, M, int(err.argmax()), float(err.max()))
    assert all(c == 0 for c in ops.gemm_error_codes())


@pytest.mark.parametrize("m,n,dtype", ((256, 2048, torch.bfloat16), (4096, 4096, torch.bfloat16), (4096, 4096, torch.float32), (4096, 8192, torch.float16),
                                       (4096, 12288, torch.bfloat16), (19072, 12288, torch.bfloat16)))
def test_rows_do_not_depend_on_the_shape_of_the_transform(m, n, dtype):
    """One row more, so that the form, the slices or the warps of the activation transform change and the plan of the GEMM does not (in clusters, and,
    the last, in even runs over a full GPU): sums are formed in one order, so that not a bit of the other rows changes."""
    from htr_b200 import ops, wire

    def padded(M):
        return -(-M // 8) * 8 if dtype == torch.float32 or M <= 8 else -(-M // 16) * 16

    def addends(M):                                               # blocks that a lane adds up one after another
        return min(max(padded(M) // 48, 1), -(-n // 1024))

    dev = torch.device("cuda:0")
    w = [t.to(dev) for t in wire.random_packed(m, n, 3, seed=n)]
    x = torch.randn(256, n, generator=torch.Generator().manual_seed(n)).to(dtype).to(dev)
    found = 0
    for M in range(9, 128 if dtype == torch.float32 else 256):
        a, b = transform(dtype, M, m, n, 3), transform(dtype, M + 1, m, n, 3)
        if a[:2] == b[:2] and a[2:] != b[2:] and addends(M) == addends(M + 1):
            found += 1
            assert torch.equal(ops.linear(x[:M + 1], *w)[:M], ops.linear(x[:M], *w)), (M, a, b)
    assert found >= 1
