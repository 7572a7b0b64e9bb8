"""The native front of the operators (csrc/host_binding.cpp) against the general path in Python: the same kernels, so equal bits;
what it does not take (strided rows, wrong types, CPU tensors) must still work or raise as the general path does."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,dtype", ((1, torch.bfloat16), (4, torch.float32), (5, torch.float16), (129, torch.float32), (300, torch.bfloat16), (600, torch.bfloat16)))
def test_front_equals_general_path(M, dtype, monkeypatch):
    from htr_b200 import _lib, ops, wire

    dev = torch.device("cuda:0")
    m, n, K = 384, 256, 3
    w = wire.random_packed(m, n, K, seed=M, device=dev)
    x = torch.randn(M, n, generator=torch.Generator().manual_seed(M)).to(dtype).to(dev)
    bias = torch.randn(m, device=dev).to(dtype)
    ops.linear(x, *w, bias)                                              # the workspaces exist from here on
    got, padded = ops.linear(x.view(1, M, n), *w, bias), ops.linear_padded(x[:, :200].contiguous(), *w, bias[:136].contiguous(), m_out=136)
    assert got.shape == (1, M, m)
    strided = torch.zeros(M, 2 * n, dtype=dtype, device=dev)
    strided[:, :n] = x
    assert torch.equal(ops.linear(strided[:, :n], *w, bias), got[0])     # rows with a gap: copied by the general path
    with pytest.raises(_lib.HTRError):
        ops.linear(x, *w, bias.double())
    with pytest.raises(_lib.HTRError):
        ops.linear(x[:, :128].contiguous(), *w)
    side = torch.cuda.Stream()                                            # a stream without workspaces yet
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        other = ops.linear(x, *w, bias)
    side.synchronize()
    assert torch.equal(other, got[0])
    for name in ("linear", "linear_padded"):
        monkeypatch.setattr(ops._host, name, lambda *a: None)
    assert torch.equal(ops.linear(x, *w, bias), got[0])
    assert torch.equal(ops.linear_padded(x[:, :200].contiguous(), *w, bias[:136].contiguous(), m_out=136), padded)


@pytest.mark.parametrize("T,hidden,inter", ((1, 256, 128), (16, 2048, 1024)))    # the routed GEMV; pairs that share experts on the grouped GEMM
@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float32))
def test_moe_fronts_equal_general_path(T, hidden, inter, dtype, monkeypatch):
    from htr_b200 import ops, sharded, wire

    dev, E, k = torch.device("cuda:0"), 8, 4
    experts = [dict(gate_up=wire.random_packed(2 * inter, hidden, 3, seed=e, device=dev), down=wire.random_packed(hidden, inter, 3, seed=50 + e, device=dev))
               for e in range(E)]
    layer = sharded.ExpertParallelMoE(experts, device=dev)
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, hidden, generator=g).to(dtype).to(dev)
    score, ids = torch.randn(T, E, generator=g).to(dev).topk(k, dim=-1)
    gates = score.softmax(-1)
    layer(x, ids, gates)                                                 # the workspaces exist from here on
    got = layer(x, ids, gates)
    for name in ("linear_routed", "linear_routed_gemm", "route_plan", "moe_weighted_sum"):
        monkeypatch.setattr(ops._host, name, lambda *a: None)
    assert torch.equal(layer(x, ids, gates), got)


@pytest.mark.parametrize("T", (1, 2, 8, 9, 33))
def test_decoder_front_equals_general_path(T, monkeypatch):
    from htr_b200 import ops
    from htr_b200.decoder import DecoderConfig, PackedDecoder

    dev = torch.device("cuda:0")
    dec = PackedDecoder(DecoderConfig(layers=3, hidden=256, q_heads=4, kv_heads=2, intermediate=384, vocab=512, max_len=64), dev, seed=T)
    ids, pos = torch.arange(T, device=dev), torch.arange(5, 5 + T, device=dev)
    dec.forward(ids, pos)                                                # the workspace exists from here on
    took = []
    front = ops._host.decoder_step
    monkeypatch.setattr(ops._host, "decoder_step", lambda *a: took.append(front(*a)) or took[-1])
    got, k, v = dec.forward(ids, pos), dec.k_cache.clone(), dec.v_cache.clone()
    assert took[0] is not None
    monkeypatch.setattr(ops._host, "decoder_step", lambda *a: None)
    assert torch.equal(dec.forward(ids, pos), got) and torch.equal(dec.k_cache, k) and torch.equal(dec.v_cache, v)
    monkeypatch.setattr(ops._host, "decoder_step", front)
    dec.layers[1]["o"] = dec.layers[1]["qkv"]                            # another shape: refused as the general path refuses it
    with pytest.raises(Exception):
        dec.forward(ids, pos)


def test_integers_beyond_their_range_are_refused(monkeypatch):
    """Sizes that do not fit a C integer: the error or the result of the general path, never a Python error left set by the front."""
    from htr_b200 import _lib, ops, wire

    dev = torch.device("cuda:0")
    w = wire.random_packed(384, 256, 4, seed=1, device=dev)
    x = torch.randn(3, 256, device=dev).bfloat16()
    want = ops.linear(x, *w)
    for m_out in (2 ** 31, 2 ** 40, 2 ** 63, 2 ** 70, -(2 ** 70), 0, 385):
        with pytest.raises(_lib.HTRError):
            ops.linear_padded(x, *w, m_out=m_out)
    with pytest.raises(_lib.HTRError):
        ops.linear_fused(x, *w, prologue=3)
    monkeypatch.setattr(ops, "GEMM_ROUTE_MAX", 2 ** 70)
    assert torch.equal(ops.linear(x, *w), want)
    for bad in (2 ** 31, 2 ** 70, -(2 ** 70), "1", None):                # the front itself: None, no exception
        assert ops._host.linear(x, *w, None, 0, 4, bad) is None
        assert ops._host.linear_padded(x, *w, None, bad, 4) is None and ops._host.linear_padded(x, *w, None, 384, bad) is None
        assert ops._host.linear_fused(x, *w, None, bad, None, 1e-6, False) is None


@pytest.mark.parametrize("T", (1, 3, 9, 300))
def test_a_refused_decoder_step_leaves_nothing_behind(T):
    """None from the native loop means that nothing was enqueued, also where only a late linear is the reason: the residual stream and the
    caches are as they were.  Reasons: a weight that is not 16-byte aligned, a workspace that is too small for one of the linears."""
    from htr_b200 import _lib, ops
    from htr_b200.decoder import DecoderConfig, PackedDecoder

    dev = torch.device("cuda:0")
    dec = PackedDecoder(DecoderConfig(layers=2, hidden=256, q_heads=4, kv_heads=2, intermediate=384, vocab=65536, max_len=512), dev, seed=T)
    ids, pos = torch.arange(T, device=dev), torch.arange(5, 5 + T, device=dev)
    want = dec.forward(ids, pos)                                         # the workspaces exist from here on
    c, gemm_rows = dec.cfg, 0 if T <= ops.GEMV_MAX_M else ops.GEMM_ROUTE_MAX
    dec.k_cache.zero_(), dec.v_cache.zero_()

    def step():
        x = dec.embed.index_select(0, ids)
        y = ops._host.decoder_step(x, dec.layers, dec.head, dec.ln_f, dec.k_cache, dec.v_cache, pos, dec.cos, dec.sin, dec.status, c.q_heads, c.kv_heads,
                                   c.eps, gemm_rows)
        if y is None:
            assert torch.equal(x, dec.embed.index_select(0, ids)) and not bool(dec.k_cache.any()) and not bool(dec.v_cache.any())
        return y

    qw = dec.layers[1]["down"][0]
    shifted = torch.zeros(qw.numel() + 1, dtype=qw.dtype, device=dev)[1:].view_as(qw)
    shifted.copy_(qw)
    good = dec.layers[1]["down"]
    dec.layers[1]["down"] = (shifted, *good[1:])
    assert step() is None
    with pytest.raises(_lib.HTRError):
        dec.forward(ids, pos)
    dec.layers[1]["down"] = good
    dec.k_cache.zero_(), dec.v_cache.zero_()
    kind, stream = (0 if gemm_rows == 0 else 1), torch.cuda.current_stream().cuda_stream
    rows = min(T, ops.GEMM_MAX_M)
    size = _lib.lib.htr_linear_workspace_bytes if kind == 0 else _lib.lib.htr_linear_gemm_workspace_bytes
    need = max(size(rows, t[0].shape[0] * 16, t[0].shape[1] * 16, t[0].shape[2] // 8) for t in (*(dec.layers[0][k] for k in ("qkv", "o", "gate_up", "down")), dec.head))
    small = torch.zeros(need - 1, dtype=torch.uint8, device=dev)         # too little for one of them
    ops._host.set_workspace(kind, dev.index, stream, small)
    try:
        assert step() is None
    finally:
        ops._host.set_workspace(kind, dev.index, stream, (ops._WORKSPACES if kind == 0 else ops._GEMM_WS)[(dev.index, stream)])
    assert torch.equal(step(), want)
