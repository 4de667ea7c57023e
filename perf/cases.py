"""What a user of this package has it do, as timed cases over the range of sizes that such programs meet.

Four kinds of work, each through the package's public entry points:

  linear  y = x W^T of a block-quantized weight (`QMatMul.forward`), from one decoded token to a 2048-token prompt chunk.
          A model's next linear has other weights, so a pass takes the next of several copies of the matrix, enough of
          them that the weights come from HBM and not from the L2 cache of the pass before.
  host    the same product for a caller whose activations and results live in pinned host memory (`ops.qmatmul_host`), which
          waits for its stream because it reads the result next.
  moe     a sparse mixture-of-experts block (`QMoeBlock.forward`): routing, grouped products, combine.
  decode  one token of a LLaMA-architecture model at a position of its context (`QLlama.run_step`, captured as serving loops do).
  codec   weights to blocks and back (`ops.quantize_weights`, `ops.dequantize`): converting a checkpoint, checking it.
"""
from __future__ import annotations

import math

import torch

from fuel_b200 import GgmlDType as T
from fuel_b200 import _lib, ops
from fuel_b200.llama import LlamaConfig, QLlama, q4km_mix
from fuel_b200.moe import QMoeBlock
from fuel_b200.quantized import QMatMul, QTensor

_L2_BYTES = 126 << 20
_FORMATS = {t.name: t for t in (T.Q4_0, T.Q4_1, T.Q5_0, T.Q5_1, T.Q8_0, T.Q2K, T.Q3K, T.Q4K, T.Q5K, T.Q6K)}
_FLOATS = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def listed():
    return [
        # one token through an attention projection of a 7B-class model: the smallest call, latency and launches count
        dict(name="linear_q4k_m1", kind="linear", fmt="Q4K", m=1, n=4096, k=4096, operands="f16"),
        # one token through its feed-forward down projection, kept at 6 bits as mixed checkpoints do
        dict(name="linear_q6k_m1_down", kind="linear", fmt="Q6K", m=1, n=4096, k=11008, operands="f16"),
        # a few sequences decoded together on a small 3-bit checkpoint; the vocabulary-like width is odd
        dict(name="linear_q3k_m7", kind="linear", fmt="Q3K", m=7, n=5003, k=4096, operands="f16"),
        # a serving batch of 16 through the down projection
        dict(name="linear_q4k_m16_down", kind="linear", fmt="Q4K", m=16, n=4096, k=11008, operands="f16"),
        # a ragged batch between decoding and prompt processing
        dict(name="linear_q6k_m45", kind="linear", fmt="Q6K", m=45, n=11008, k=4096, operands="f16"),
        # a prompt of a few hundred tokens, 8-bit weights
        dict(name="linear_q8_0_m333", kind="linear", fmt="Q8_0", m=333, n=4096, k=4096, operands="f16"),
        # a long prompt chunk through a wide feed-forward projection: the dense contraction
        dict(name="linear_q4k_m2048", kind="linear", fmt="Q4K", m=2048, n=14336, k=4096, operands="f16"),
        # a runtime that keeps activations on the host: one token, up projection
        dict(name="host_q4k_m1", kind="host", fmt="Q4K", m=1, n=11008, k=4096),
        # 256 tokens through a 128-expert block, top 8: some sixteen rows an expert
        dict(name="moe_q4k_t256", kind="moe", fmt="Q4K", tokens=256, experts=128, top_k=8, hidden=2048, ffn=768),
        # the same block while three sequences decode: a couple of dozen experts with one row each
        dict(name="moe_q4k_t3", kind="moe", fmt="Q4K", tokens=3, experts=128, top_k=8, hidden=2048, ffn=768),
        # one token of a 7B-architecture model after a 512-token prompt
        dict(name="decode_7b", kind="decode", mix="q4km", layers=32, dim=4096, heads=32, kv_heads=32, ffn=11008, vocab=32000,
             pos=512, max_seq=640),
        # converting a feed-forward matrix to 4 bits and reading it back as f16
        dict(name="codec_q4k_f16", kind="codec", fmt="Q4K", n=11008, k=4096, out="f16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _k_of(rng, fmt, lo, hi):
    """Row lengths: whole 256-element blocks for the k-quants; the 32-element formats are what models with other widths use."""
    unit = 256 if fmt.endswith("K") or rng.random() < 0.7 else 64
    return max(1, round(_log_int(rng, lo, hi) / unit)) * unit


def _n_of(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    return n if rng.random() < 0.4 else max(64, n // 64 * 64)


def draw(rng):
    kind = rng.choices(("linear", "host", "moe", "decode", "codec"), (11, 1, 3, 2, 2))[0]
    # most checkpoints are Q4_K, Q6_K and Q8_0; the other formats share the rest
    fmt = rng.choice(("Q4K", "Q6K", "Q8_0")) if rng.random() < 0.6 else rng.choice(sorted(_FORMATS))
    if kind == "linear":
        m = _log_int(rng, 1, 2048) if rng.random() < 0.8 else 1
        return dict(kind=kind, fmt=fmt, m=m, n=_n_of(rng, 1024, 14336), k=_k_of(rng, fmt, 1024, 4096 if m > 512 else 14336),
                    operands="bf16" if m > 64 and rng.random() < 0.25 else "f16")
    if kind == "host":
        return dict(kind=kind, fmt=rng.choice(("Q4K", "Q6K", "Q8_0")), m=_log_int(rng, 1, 4), n=_n_of(rng, 1024, 14336),
                    k=_k_of(rng, "Q4K", 1024, 14336))
    if kind == "moe":
        e = rng.choice((8, 16, 60, 64, 128))
        return dict(kind=kind, fmt="Q4K" if rng.random() < 0.75 else "Q6K", tokens=_log_int(rng, 1, 256), experts=e,
                    top_k=rng.choice((1, 2, 4, 8)), hidden=256 * rng.randint(2, 8), ffn=256 * rng.randint(2, 6))
    if kind == "decode":
        heads = rng.choice((8, 12, 16, 20, 24, 32))
        max_seq = rng.choice((640, 2048, 4096))
        return dict(kind=kind, mix="q4km" if rng.random() < 0.75 else "q8_0", layers=rng.randint(2, 16), dim=128 * heads,
                    heads=heads, kv_heads=heads // rng.choice((1, 2, 4)), ffn=256 * rng.randint(heads, 43 * heads // 32),
                    vocab=_n_of(rng, 8000, 32000), pos=_log_int(rng, 1, max_seq - 1), max_seq=max_seq)
    return dict(kind=kind, fmt=fmt, n=_n_of(rng, 512, 11008), k=_k_of(rng, fmt, 512, 4096), out=rng.choice(sorted(_FLOATS)))


def _normal(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * scale


def _copies(nbytes):
    """Copies of a matrix that, together with another set of them, exceed the L2 cache."""
    return max(2, min(64, math.ceil(0.75 * _L2_BYTES / nbytes)))


def _prepare_decode(case, seed):
    mixes = {"q4km": q4km_mix, "q8_0": lambda name, layer: T.Q8_0}
    cfg = LlamaConfig(dim=case["dim"], n_layers=case["layers"], n_heads=case["heads"], n_kv_heads=case["kv_heads"],
                      ffn_dim=case["ffn"], vocab=case["vocab"], max_seq=case["max_seq"])
    model = QLlama(cfg, torch.device("cuda", torch.cuda.current_device()), seed=seed, mix=mixes[case["mix"]])
    pos = case["pos"]
    for li, layer in enumerate(model.layers):      # the context so far
        layer["kc"][:, :pos] = _normal((case["kv_heads"], pos, cfg.head_dim), 7 * seed + 2 * li)
        layer["vc"][:, :pos] = _normal((case["kv_heads"], pos, cfg.head_dim), 7 * seed + 2 * li + 1)
    g = torch.Generator().manual_seed(seed)
    token = torch.randint(0, cfg.vocab, (1,), generator=g, dtype=torch.int32).cuda()
    at = torch.tensor([pos], dtype=torch.int32, device="cuda")
    model.token.copy_(token)
    model.pos.copy_(at)
    _lib.lib.fuelq_set_option(_lib.OPT_PDL, 1)     # as the package recommends for captured loops; the graph keeps it
    model.capture()
    _lib.lib.fuelq_set_option(_lib.OPT_PDL, 0)
    return dict(model=model, token=token, at=at)


def prepare(case, seed):
    kind, fmt = case["kind"], _FORMATS.get(case.get("fmt"))
    _lib.lib.fuelq_set_option(_lib.OPT_PDL, 0)
    _lib.lib.fuelq_set_option(_lib.OPT_PREFILL_BF16, 1 if case.get("operands") == "bf16" else 0)
    state = dict(kind=kind, next=0)
    if kind == "decode":
        state.update(_prepare_decode(case, seed))
    elif kind == "moe":
        e, h, f = case["experts"], case["hidden"], case["ffn"]
        gate_up = ops.quantize_weights(fmt, _normal((e * 2 * f, h), seed, 0.02))
        down = ops.quantize_weights(fmt, _normal((e * h, f), seed + 1_000_003, 0.02))
        state.update(block=QMoeBlock(e, h, f, case["top_k"], gate_up, down, dtype=fmt, max_tokens=case["tokens"]),
                     x=_normal((case["tokens"], h), seed + 2_000_003), logits=_normal((case["tokens"], e), seed + 3_000_017))
    elif kind == "codec":
        state.update(fmt=fmt, w=_normal((case["n"], case["k"]), seed, 0.02), out=_FLOATS[case["out"]])
    else:
        m, n, k = case["m"], case["n"], case["k"]
        w = _normal((n, k), seed, 0.02)
        copies = _copies(ops.storage_bytes(fmt, n * k))
        x = _normal((m, k), seed + 1_000_003)
        if kind == "linear":
            state.update(linears=[QMatMul.from_qtensor(QTensor.quantize(w, fmt)) for _ in range(copies)], x=x)
        else:
            blocks = ops.quantize_weights(fmt, w)
            ws = _lib.lib.fuelq_qmatmul_host_workspace_bytes(int(fmt), m, n, k)
            state.update(fmt=fmt, n=n, blocks=[blocks.clone() for _ in range(copies)], x=x.cpu().pin_memory(),
                         y=torch.empty(m, n, dtype=torch.float32, pin_memory=True),
                         workspace=torch.empty(ws, dtype=torch.uint8, device="cuda"))
    return state


def run(state):
    kind = state["kind"]
    if kind == "linear":
        i = state["next"]
        state["next"] = (i + 1) % len(state["linears"])
        return state["linears"][i].forward(state["x"])
    if kind == "host":
        i = state["next"]
        state["next"] = (i + 1) % len(state["blocks"])
        y = ops.qmatmul_host(state["fmt"], state["blocks"][i], state["n"], state["x"], state["y"], state["workspace"])
        torch.cuda.current_stream().synchronize()
        return y
    if kind == "moe":
        return state["block"].forward(state["x"], state["logits"])
    if kind == "decode":
        model = state["model"]
        model.token.copy_(state["token"])
        model.pos.copy_(state["at"])
        model.run_step()
        return model.logits
    blocks = ops.quantize_weights(state["fmt"], state["w"])
    return blocks, ops.dequantize(state["fmt"], blocks, state["w"].numel(), state["out"])


def _bytes(fmt, count):
    return ops.storage_bytes(_FORMATS[fmt], count)


def _experts_hit(case):
    """Experts that at least one of the tokens goes to, on average."""
    e = case["experts"]
    return e * (1.0 - (1.0 - case["top_k"] / e) ** case["tokens"])


def work(case):
    kind = case["kind"]
    if kind in ("linear", "host"):
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": _bytes(case["fmt"], n * k) + 4 * m * (n + k), "flops": 2 * m * n * k}
    if kind == "moe":
        e, h, f, t, top = case["experts"], case["hidden"], case["ffn"], case["tokens"], case["top_k"]
        per = _bytes(case["fmt"], 2 * f * h) + _bytes(case["fmt"], h * f)
        return {"bytes": int(_experts_hit(case) * per) + 4 * t * (2 * h + e), "flops": 2 * t * top * 3 * h * f}
    if kind == "decode":
        d, f, kv, v, n_l = case["dim"], case["ffn"], 128 * case["kv_heads"], case["vocab"], case["layers"]
        shapes = dict(attn_q=d * d, attn_k=kv * d, attn_v=kv * d, attn_output=d * d, ffn_gate=f * d, ffn_up=f * d, ffn_down=f * d)
        fmt = (lambda name, li: q4km_mix(name, li).name) if case["mix"] == "q4km" else (lambda name, li: "Q8_0")
        nbytes = _bytes(fmt("output", -1), v * d) + 4 * v
        for li in range(n_l):
            nbytes += sum(_bytes(fmt(name, li), count) for name, count in shapes.items()) + 2 * 4 * kv * (case["pos"] + 1)
        return {"bytes": nbytes, "flops": 2 * (v * d + n_l * (sum(shapes.values()) + 2 * d * (case["pos"] + 1)))}
    count = case["n"] * case["k"]
    out = 4 if case["out"] == "f32" else 2
    return {"bytes": 4 * count + 2 * _bytes(case["fmt"], count) + out * count, "flops": 2 * count}


def tolerance(case):
    """Integer kernels: 8-bit activations times block integers are exact, the sums over blocks are 32-bit floats. Above the
    batch size at which the product becomes a tensor-core contraction: operands of 11 (f16) or 8 (bf16) significant bits."""
    kind = case["kind"]
    if kind == "codec":
        return "exact"
    if kind == "moe":
        return {"rel": 1e-3}       # integer products, re-quantized to 8 bits in between: a rounding tie may fall the other way
    if kind == "decode":
        return {"rel": 0.03}       # the same at four places of every layer
    if kind == "linear":
        main = case["fmt"] in ("Q4K", "Q5K", "Q6K", "Q8_0") and case["k"] % 256 == 0
        if case["m"] > (64 if main else 16):
            return {"rel": 1e-2 if case["operands"] == "bf16" else 1e-3}
    return {"rel": 1e-5}
