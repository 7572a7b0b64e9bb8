"""The single-token attention kernel where its work split can go wrong: positions around the cluster size and the rows held in flight,
groups of one to six query heads, the last row of the caches, against the two separate kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rep", (1, 2, 3, 6))
@pytest.mark.parametrize("p", (0, 3, 4, 127, 128, 255, 256, 257, 1023))
def test_positions_and_groups(rep, p):
    from htr_b200 import _lib

    dev, L, hkv, D, max_len = torch.device("cuda:0"), _lib.lib, 2, 128, 1024
    hq, st = hkv * rep, torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device=dev).manual_seed(p + rep)
    ang = torch.arange(max_len, device=dev).float()[:, None] / 1.0e6 ** (torch.arange(0, D, 2, device=dev).float() / D)
    cos, sin, status = ang.cos(), ang.sin(), torch.zeros(1, dtype=torch.int32, device=dev)
    k1, v1 = (torch.randn(max_len, hkv, D, device=dev, generator=g).bfloat16() for _ in range(2))
    k1[p + 1:], v1[p + 1:] = float("nan"), float("nan")                      # rows of later positions must not matter
    qkv = torch.randn(1, (hq + 2 * hkv) * D, device=dev, generator=g).bfloat16()
    pos, k2, v2, q = torch.full((1,), p, dtype=torch.long, device=dev), k1.clone(), v1.clone(), torch.empty(1, hq, D, dtype=torch.bfloat16, device=dev)
    want, got = torch.empty_like(q), torch.empty_like(q)
    _lib.check(L.htr_dec_rope_cache(qkv.data_ptr(), pos.data_ptr(), cos.data_ptr(), sin.data_ptr(), q.data_ptr(), k1.data_ptr(), v1.data_ptr(), 1, hq, hkv,
                                    D, max_len, status.data_ptr(), st), "htr_dec_rope_cache")
    _lib.check(L.htr_dec_attention(q.data_ptr(), k1.data_ptr(), v1.data_ptr(), pos.data_ptr(), want.data_ptr(), 1, hq, hkv, D, max_len, status.data_ptr(),
                                   st), "htr_dec_attention")
    _lib.check(L.htr_dec_rope_attention(qkv.data_ptr(), pos.data_ptr(), cos.data_ptr(), sin.data_ptr(), k2.data_ptr(), v2.data_ptr(), got.data_ptr(), hq, hkv,
                                        D, max_len, status.data_ptr(), st), "htr_dec_rope_attention")
    assert torch.equal(k1[:p + 1], k2[:p + 1]) and torch.equal(v1[:p + 1], v2[:p + 1]) and int(status.item()) == 0
    assert float((got.float() - want.float()).abs().max()) <= 1e-2 * float(want.float().abs().max())
