"""The workloads by which the speed of the package is judged, each through the public call that a user's program makes.

Five kinds of work, all from what the package is for:

  linear    `ops.linear`: one packed linear, from a single decode row to a prefill batch
  padded    `ops.linear_padded`: a packed linear whose widths are not multiples of 128
  moe       `sharded.ExpertParallelMoE` on one GPU: routed experts of a decode step
  decoder   `decoder.PackedDecoder.forward`: one step of a whole decoder (a token of decoding, or a prompt)
  encode    `encoder.viterbi`: the trellis search behind the encoder, on the tiles of one 16-column block

Inputs are synthetic and made on the GPU from the seed: every bit pattern is a valid circular stream, so packed words are
uniform; scales, signs and activations (1 % of the channels ten times larger) follow `wire.random_packed` and the benchmark.
"""
import math

import torch

from htr_b200 import encoder, ops, sharded, wire
from htr_b200.decoder import DecoderConfig, PackedDecoder

DEV = torch.device("cuda:0")
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
WIDTHS = (2, 3, 4, 5, 6, 8)


def listed():
    return [
        # the key or value projection of a grouped-query layer for one token: the smallest call, all latency
        {"name": "kv_proj_m1", "kind": "linear", "m": 1024, "n": 4096, "K": 4, "M": 1, "dtype": "bf16", "bias": False},
        # the MLP up-projection at batch 1: the headline case of the benchmark
        {"name": "mlp_up_m1", "kind": "linear", "m": 12288, "n": 4096, "K": 4, "M": 1, "dtype": "bf16", "bias": False},
        # the MLP down-projection at the small batches of the bitrate sweep, one decode step of 4 and of 16 sequences
        {"name": "mlp_down_m4", "kind": "linear", "m": 4096, "n": 12288, "K": 3, "M": 4, "dtype": "bf16", "bias": False},
        {"name": "mlp_down_m16", "kind": "linear", "m": 4096, "n": 12288, "K": 5, "M": 16, "dtype": "bf16", "bias": False},
        # a large decode batch or a short prompt, in fp16 and at the narrowest stream
        {"name": "mlp_up_m64", "kind": "linear", "m": 12288, "n": 4096, "K": 2, "M": 64, "dtype": "fp16", "bias": False},
        # odd sizes with a bias, in float32: 23 x 13 blocks, a row count that fills no tile, a wide stream
        {"name": "ragged_m37", "kind": "linear", "m": 2944, "n": 1664, "K": 6, "M": 37, "dtype": "fp32", "bias": True},
        # the prefill of 2048 tokens
        {"name": "prefill_m2048", "kind": "linear", "m": 4096, "n": 12288, "K": 4, "M": 2048, "dtype": "bf16", "bias": False},
        # the LM head for 8 sequences
        {"name": "lm_head_m8", "kind": "linear", "m": 151936, "n": 4096, "K": 4, "M": 8, "dtype": "bf16", "bias": False},
        # a projection whose widths are padded to the block size, a few rows
        {"name": "padded_m11", "kind": "padded", "m": 4096, "n": 4096, "m_out": 4096, "n_in": 4000, "K": 3, "M": 11, "dtype": "bf16", "bias": True},
        # the experts of one decode step of 16 sequences
        {"name": "moe_t16", "kind": "moe", "hidden": 4096, "inter": 1536, "experts": 64, "top_k": 8, "K": 3, "T": 16},
        # one token of the 9B-class decoder, a few hundred positions into its sequence
        {"name": "decoder_step", "kind": "decoder", "layers": 36, "hidden": 4096, "q_heads": 32, "kv_heads": 8, "inter": 12288, "vocab": 151936,
         "K": 4, "K_head": 4, "max_len": 512, "T": 1, "pos": 200},
        # the tiles of one 16-column block of a 4096-row matrix
        {"name": "encode_256", "kind": "encode", "tiles": 256, "K": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _blocks(rng, lo, hi):
    return 128 * max(1, _log(rng, lo, hi) // 128)


def draw(rng):
    kind = rng.choices(("linear", "padded", "moe", "decoder", "encode"), (10, 2, 3, 3, 2))[0]
    if kind == "linear":
        dtype = rng.choices(("bf16", "fp16", "fp32"), (6, 3, 2))[0]
        most = 2048 * 12288 * 4096
        while True:
            c = {"kind": kind, "m": _blocks(rng, 256, 32768), "n": _blocks(rng, 256, 16384), "K": rng.choice(WIDTHS),
                 "M": _log(rng, 1, 256 if dtype == "fp32" else 2048), "dtype": dtype, "bias": rng.random() < 0.3}
            if c["M"] * c["m"] * c["n"] <= most:
                return c
    if kind == "padded":
        m_out, n_in = 8 * _log(rng, 16, 1024), 8 * _log(rng, 16, 1024)
        return {"kind": kind, "m": -(-m_out // 128) * 128, "n": -(-n_in // 128) * 128, "m_out": m_out, "n_in": n_in, "K": rng.choice((2, 3, 4, 5)),
                "M": _log(rng, 1, 64), "dtype": rng.choice(("bf16", "fp16")), "bias": rng.random() < 0.5}
    if kind == "moe":
        return {"kind": kind, "hidden": 128 * rng.randint(8, 32), "inter": 128 * rng.randint(4, 12), "experts": rng.choice((16, 32, 64)),
                "top_k": rng.choice((2, 4, 8)), "K": rng.choice((2, 3, 4)), "T": _log(rng, 1, 32)}
    if kind == "decoder":
        kv = rng.choice((2, 4, 8))
        c = {"kind": kind, "layers": _log(rng, 2, 24), "hidden": 128 * rng.randint(8, 32), "q_heads": kv * rng.choice((2, 4)), "kv_heads": kv,
             "inter": 128 * rng.randint(16, 96), "vocab": 128 * _log(rng, 64, 1024), "K": rng.choice((2, 3, 4, 5)), "K_head": rng.choice((4, 5, 6)),
             "max_len": 1024, "T": 1, "pos": _log(rng, 1, 1000)}
        if rng.random() < 0.4:                                   # a prompt instead of a token
            c.update(T=_log(rng, 2, 64), pos=0)
        return c
    return {"kind": kind, "tiles": _log(rng, 16, 256), "K": rng.choice(WIDTHS)}


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _packed(m, n, K, g):
    qw = torch.randint(-(2 ** 31), 2 ** 31, (m // 16, n // 16, 8 * K), dtype=torch.int32, device=DEV, generator=g)
    sc = (torch.randn(m, device=DEV, generator=g).abs() * 0.01 + 0.01).half()
    su = torch.randint(0, 256, (n // 8,), dtype=torch.uint8, device=DEV, generator=g)
    sv = torch.randint(0, 256, (m // 8,), dtype=torch.uint8, device=DEV, generator=g)
    return qw, sc, su, sv


def _activations(M, n, dtype, g):
    x = torch.randn(M, n, device=DEV, generator=g)
    x *= torch.where(torch.rand(n, device=DEV, generator=g) < 0.01, 10.0, 1.0)
    return x.to(dtype)


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind in ("linear", "padded"):
        dt = DTYPES[case["dtype"]]
        w = _packed(case["m"], case["n"], case["K"], g)
        x = _activations(case["M"], case.get("n_in", case["n"]), dt, g)
        bias = torch.randn(case.get("m_out", case["m"]), device=DEV, generator=g).to(dt) if case["bias"] else None
        return {"kind": kind, "x": x, "w": w, "bias": bias, "m_out": case.get("m_out")}
    if kind == "moe":
        h, inter, K, E, T, k = (case[s] for s in ("hidden", "inter", "K", "experts", "T", "top_k"))
        experts = [dict(gate_up=_packed(2 * inter, h, K, g), down=_packed(h, inter, K, g)) for _ in range(E)]
        layer = sharded.ExpertParallelMoE(experts, device=DEV)
        score, ids = torch.randn(T, E, device=DEV, generator=g).topk(k, dim=-1)
        return {"kind": kind, "layer": layer, "x": _activations(T, h, torch.bfloat16, g), "ids": ids, "gates": score.softmax(-1)}
    if kind == "decoder":
        cfg = DecoderConfig(layers=case["layers"], hidden=case["hidden"], q_heads=case["q_heads"], kv_heads=case["kv_heads"], head_dim=128,
                            intermediate=case["inter"], vocab=case["vocab"], K=case["K"], K_head=case["K_head"], max_len=case["max_len"])
        h, att = cfg.hidden, cfg.q_heads * 128

        def norm():
            return (1.0 + 0.05 * torch.randn(h, device=DEV, generator=g)).bfloat16()

        layers = [dict(qkv=_packed(att + 2 * cfg.kv_heads * 128, h, cfg.K, g), o=_packed(h, att, cfg.K, g), gate_up=_packed(2 * cfg.intermediate, h, cfg.K, g),
                       down=_packed(h, cfg.intermediate, cfg.K, g), ln1=norm(), ln2=norm()) for _ in range(cfg.layers)]
        weights = dict(layers=layers, head=_packed(cfg.vocab, h, cfg.K_head, g), ln_f=norm(),
                       embed=(torch.randn(cfg.vocab, h, device=DEV, dtype=torch.bfloat16, generator=g) * 0.02))
        model = PackedDecoder(cfg, DEV, weights=weights)
        pos = case["pos"]
        for cache in (model.k_cache, model.v_cache):             # the sequence so far
            cache[:, :pos].normal_(generator=g)
        return {"kind": kind, "model": model, "ids": torch.randint(0, cfg.vocab, (case["T"],), device=DEV, generator=g),
                "pos": torch.arange(pos, pos + case["T"], device=DEV)}
    B = case["tiles"]
    x = torch.randn(B, 256, device=DEV, generator=g)
    rs = (torch.rand(B, 16, device=DEV, generator=g) + 0.5).repeat_interleave(16, dim=1) ** 2       # squared row scales of a tile's rows
    return {"kind": kind, "x": x, "w": rs / rs.mean(dim=1, keepdim=True), "K": case["K"]}


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return ops.linear(state["x"], *state["w"], state["bias"])
    if kind == "padded":
        return ops.linear_padded(state["x"], *state["w"], bias=state["bias"], m_out=state["m_out"])
    if kind == "moe":
        return state["layer"](state["x"], state["ids"], state["gates"])
    if kind == "decoder":
        model = state["model"]
        return {"logits": model.forward(state["ids"], state["pos"]), "k_cache": model.k_cache, "v_cache": model.v_cache}
    return encoder.viterbi(state["x"], state["w"], None, state["K"])


def work(case):
    kind = case["kind"]
    if kind in ("linear", "padded"):
        m, n, M = case.get("m_out", case["m"]), case.get("n_in", case["n"]), case["M"]
        size = 4 if case["dtype"] == "fp32" else 2
        return {"bytes": wire.payload_bytes(case["m"], case["n"], case["K"]) + size * (M * (m + n) + (m if case["bias"] else 0)), "flops": 2 * M * m * n}
    if kind == "moe":
        h, inter, K, E, T, k = (case[s] for s in ("hidden", "inter", "K", "experts", "T", "top_k"))
        hit = E * (1.0 - (1.0 - k / E) ** T)                      # experts that T tokens are expected to meet: each read once
        return {"bytes": hit * (wire.payload_bytes(2 * inter, h, K) + wire.payload_bytes(h, inter, K)) + 4 * T * h, "flops": 2 * T * k * 3 * h * inter}
    if kind == "decoder":
        h, L, T, inter, att, kv = case["hidden"], case["layers"], case["T"], case["inter"], 128 * case["q_heads"], 128 * case["kv_heads"]
        shapes = ((att + 2 * kv, h), (h, att), (2 * inter, h), (h, inter))
        weights = L * sum(wire.payload_bytes(m, n, case["K"]) for m, n in shapes) + wire.payload_bytes(case["vocab"], h, case["K_head"])
        seen = case["pos"] + T                                   # positions whose keys and values are read; the new ones are written too
        return {"bytes": weights + L * 4 * kv * (seen + T) + 2 * T * (h + case["vocab"]),
                "flops": 2 * T * (L * sum(m * n for m, n in shapes) + case["vocab"] * h) + 4 * T * L * att * seen}
    # two passes over 65536 candidates a step, each: the distance to its value, squared, weighted, added to the path, compared
    return {"bytes": case["tiles"] * 256 * (4 + 4 + 8), "flops": case["tiles"] * 256 * 65536 * 2 * 5}


def tolerance(case):
    kind = case["kind"]
    if kind == "encode":
        return "exact"
    if kind == "decoder":                                        # dozens of bf16 layers one after another
        return {"rel": 0.03, "max": 0.5}
    if kind == "moe":                                            # two bf16 linears and a bf16 activation between them
        return {"rel": 1e-2}
    if case["dtype"] == "fp32":                                  # batches travel through the tensor cores as two fp16 halves
        return {"rel": 1e-5 if case["M"] <= 4 else 1e-4}
    return {"rel": 6e-3 if case["dtype"] == "bf16" or case["M"] > 512 else 2e-3}
