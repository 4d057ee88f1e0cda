"""Performance cases: the work that users of this framework have it do, through its public entry points.

A case is a dict of plain values.  Its `kind` says which part of the path it is:

  gemv      one quantized matrix x vector (`GemvQuant.launch`): the op that a host with its own model code calls
  gemm      n vectors through one quantized matrix (`GemmQuant.launch`)
  layer     decoder layers composed from the op objects in the order of a token (`RmsNorm`, `GemvQuant`, `RoPE`,
            `FusedAttention`, `Silu`, `add_assign`): many small launches
  attention one decode query over a long cache (`FusedAttention.launch`)
  sample    temperature / top-p / greedy choice of a token from logits on the device (`Sampler.sample`, `argmax`)
  decode    the model's own token loop from a filled context (`Llama2.generate`), greedy or sampled
  forward   the loop of a host that samples by itself: one token in, all logits out, once per token (`Llama2.forward`)
  prefill   a prompt, from an empty or a filled context (`Llama2.prefill`)
  turn      a chat turn: a prompt and the answer that follows it (`Llama2.prefill`, then `Llama2.generate_until`)

Model sizes are the two configurations of `inferi_b200.llama2` (1B and 8B architectures) and generic ones between them.

Weights are random blocks made on the GPU: every quant value with the scales that a round-to-nearest quantizer gives to
matrices of the wanted deviation.  Token t's classifier row is the embedding row of another token (a permutation), and
the embeddings are large enough to be still visible in the residual stream behind the last layer: as in a trained model the next
token's distribution then has a peak, and the greedy token does not hang on the last bits of the logits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from inferi_b200 import quant
from inferi_b200.llama2 import LAYER_MATS, LLAMA_3_2_1B, LLAMA_3_8B, Llama2, Llama2Config, Llama2Weights, Q4_K_M
from inferi_b200.ops import (AttnParams, Backend, FusedAttention, GemmQuant, GemvQuant, GpuQuantTensor, RmsNorm, RmsNormConfig, RoPE, RoPEConfig, Sampler,
                             Silu, add_assign, argmax)

TYPES = {quant.NAMES[t]: t for t in (quant.Q8_0, quant.Q4_K, quant.Q5_K, quant.Q6_K, quant.Q4_0)}
# matrix types of a file: the mixes that GGUF files commonly come in (embedding and classifier share the rows' values here, hence one type)
RECIPES = {
    "Q4_K_M": dict(Q4_K_M, token_embd=quant.Q6_K),
    "Q5_K_M": dict({n: quant.Q5_K for n in LAYER_MATS}, attn_v=quant.Q6_K, ffn_down=quant.Q6_K, token_embd=quant.Q6_K, output=quant.Q6_K),
    "Q8_0": dict({n: quant.Q8_0 for n in LAYER_MATS}, token_embd=quant.Q8_0, output=quant.Q8_0),
}
WEIGHT_STD, EMBEDDING_STD = 0.02, 4.0
F16, F32 = "f16", "f32"

_backend = None


def backend() -> Backend:
    """One context per process, as a host program keeps it."""
    global _backend
    if _backend is None:
        _backend = Backend(torch.cuda.current_device())
    return _backend


# ---------------------------------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------------------------------
def model_fields(cfg: Llama2Config, **more) -> dict:
    return dict(hidden=cfg.hidden_size, ffn=cfg.intermediate_size, layers=cfg.num_hidden_layers, heads=cfg.num_attention_heads,
                kv_heads=cfg.num_key_value_heads, vocab=cfg.vocab_size, context=cfg.max_position_embeddings, **more)


def listed() -> list[dict]:
    m1, m8 = LLAMA_3_2_1B, LLAMA_3_8B
    return [
        # a host's own model code calls the op once per matrix: the smallest call, bound by its launch
        dict(name="gemv_q8_0_4096", kind="gemv", type="Q8_0", rows=4096, cols=4096),
        # the classifier of the 8B architecture, alone: the largest single matrix
        dict(name="gemv_q6_k_lm_head", kind="gemv", type="Q6_K", rows=128256, cols=4096),
        # two 1B-architecture layers called op by op, with the f32 cache that the op API was first made for
        dict(name="layer_ops_1b", kind="layer", recipe="Q4_K_M", hidden=2048, ffn=8192, heads=32, kv_heads=8, layers=2, context=1024, pos=300, kv=F32),
        # attention over a long document
        dict(name="attention_16k", kind="attention", context=16384, heads=32, kv_heads=8, head_size=128, kv=F16),
        # nucleus sampling over a Llama-3 vocabulary
        dict(name="sample_top_p", kind="sample", vocab=128256, temperature=0.8, topp=0.95, zipf=1.5),
        # the 1B architecture early in an answer, greedy
        dict(name="decode_1b", kind="decode", recipe="Q4_K_M", kv=F16, pos=32, tokens=32, temperature=0.0, topp=0.0, **model_fields(m1)),
        # the same architecture with 8-bit weights, deep in a conversation, sampled
        dict(name="decode_1b_q8_0_sampled", kind="decode", recipe="Q8_0", kv=F16, pos=3000, tokens=16, temperature=0.8, topp=0.95, **model_fields(m1)),
        # the 8B architecture behind a 128-token prompt: what the benchmark is quoted on
        dict(name="decode_8b", kind="decode", recipe="Q4_K_M", kv=F16, pos=128, tokens=16, temperature=0.0, topp=0.0, **model_fields(m8)),
        # ... driven token by token by a host that reads the logits, further into the context
        dict(name="forward_8b_logits", kind="forward", recipe="Q4_K_M", kv=F16, pos=1900, tokens=4, **model_fields(m8)),
        # prompts: the benchmark's, and a page of text whose length is no round number
        dict(name="prefill_8b_128", kind="prefill", recipe="Q4_K_M", pos=0, tokens=128, **model_fields(m8)),
        dict(name="prefill_8b_1021", kind="prefill", recipe="Q4_K_M", pos=0, tokens=1021, **model_fields(m8)),
        # a short question in a running conversation and a short answer
        dict(name="turn_1b", kind="turn", recipe="Q4_K_M", pos=171, prompt=45, tokens=24, **model_fields(m1)),
    ]


def log_uniform(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw_model(rng, heads_per_kv=(4, 4, 4, 2, 8, 1)) -> dict:
    pick = rng.random()
    if pick < 0.25:
        m = model_fields(LLAMA_3_2_1B)
    elif pick < 0.4:
        m = model_fields(LLAMA_3_8B)
    else:
        hidden = rng.choice([2048, 2048, 4096])
        heads = hidden // rng.choice([64, 128])
        m = dict(hidden=hidden, ffn=2048 * rng.randint(hidden // 2048, 7 if hidden == 4096 else 5), layers=rng.randint(3, 24), heads=heads,
                 kv_heads=heads // rng.choice(heads_per_kv), vocab=4 * rng.randint(8000, 32064), context=rng.choice([2048, 4096]))
    m["recipe"] = rng.choice(["Q4_K_M", "Q4_K_M", "Q4_K_M", "Q5_K_M", "Q8_0"])
    return m


def draw(rng) -> dict:
    kind = rng.choice(["gemv", "gemv", "gemm", "layer", "attention", "sample", "decode", "decode", "forward", "prefill", "prefill", "turn"])
    if kind in ("gemv", "gemm"):
        t = rng.choice(["Q8_0", "Q4_K", "Q4_K", "Q5_K", "Q6_K", "Q6_K"] + (["Q4_0"] if kind == "gemv" else []))
        step = 2048 if t == "Q6_K" else 256
        cols = max(1, round(log_uniform(rng, 1024, 14336) / step)) * step
        most = 128256 * 4096 / cols          # no larger than the classifier
        rows = log_uniform(rng, 256, min(131072, most))
        if kind == "gemv":
            return dict(kind=kind, type=t, rows=4 * round(rows / 4), cols=cols)
        return dict(kind=kind, type=t, rows=128 * max(1, round(min(rows, 16384) / 128)), cols=cols, tokens=round(log_uniform(rng, 8, 1000)))
    if kind == "attention":
        hs = rng.choice([64, 128, 128])
        kv_heads = rng.choice([4, 8, 8, 16])
        return dict(kind=kind, context=round(log_uniform(rng, 40, 32768)), heads=kv_heads * rng.choice([4, 4, 4, 8, 2, 1]), kv_heads=kv_heads, head_size=hs,
                    kv=rng.choice([F16, F16, F32]))
    if kind == "sample":
        return dict(kind=kind, vocab=round(log_uniform(rng, 32000, 152000)), temperature=rng.choice([0.0, 0.6, 0.8, 1.0, 1.2]),
                    topp=rng.choice([0.0, 0.8, 0.9, 0.95, 0.98]), zipf=round(rng.uniform(1.2, 2.0), 3))
    if kind == "layer":
        hidden = rng.choice([2048, 2048, 4096])
        heads = hidden // rng.choice([64, 128])
        context = rng.choice([512, 1024, 2048])
        return dict(kind=kind, recipe=rng.choice(["Q4_K_M", "Q5_K_M", "Q8_0"]), hidden=hidden, ffn=2048 * rng.randint(hidden // 2048, 7), heads=heads,
                    kv_heads=heads // rng.choice([4, 4, 2, 8, 1]), layers=rng.randint(1, 4), context=context, pos=round(log_uniform(rng, 8, context - 1)),
                    kv=rng.choice([F32, F32, F16]))
    # the tensor-core prefill takes four query heads per kv head (the decode loop takes any group)
    m = draw_model(rng, (4,) if kind in ("prefill", "turn") else (4, 4, 4, 2, 8, 1))
    weights = m["layers"] * (2 * m["hidden"] ** 2 * (1 + m["kv_heads"] / m["heads"]) + 3 * m["hidden"] * m["ffn"])
    if kind in ("decode", "forward"):
        group4 = m["heads"] == 4 * m["kv_heads"]
        kv = rng.choice([F16, F16, F16, F32]) if kind == "decode" else F16
        # a context that the prefill cannot fill is fed token by token in prepare(): a shorter one
        pos = round(log_uniform(rng, 1, m["context"] - 40 if group4 and kv == F16 else 400))
        tokens = rng.randint(3, 32 if kind == "decode" else 8)
        if kind == "forward":
            return dict(kind=kind, kv=kv, pos=pos, tokens=tokens, **m)
        temperature = rng.choice([0.0, 0.0, 0.7, 1.0])
        return dict(kind=kind, kv=kv, pos=pos, tokens=tokens, temperature=temperature, topp=rng.choice([0.0, 0.9, 0.95]) if temperature else 0.0, **m)
    most = min(1021.0 * (7.0e9 / weights) ** 0.8, m["context"] / 2)      # no dearer than the largest listed prompt
    if kind == "prefill":
        return dict(kind=kind, pos=rng.choice([0, 0, rng.randint(1, m["context"] // 4)]), tokens=round(log_uniform(rng, 9, min(most, 1200))), **m)
    return dict(kind=kind, pos=rng.randint(0, m["context"] // 2 - 1), prompt=round(log_uniform(rng, 9, min(most, 300))), tokens=rng.randint(8, 32), **m)


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def random_matrix(g: torch.Generator, qtype: int, rows: int, cols: int, std: float) -> torch.Tensor:
    """[rows, row bytes] blocks on the GPU: uniform quants, scales such that the weights have deviation `std` and mean 0."""
    be, bb = quant.BLOCK_ELEMS[qtype], quant.BLOCK_BYTES[qtype]
    n = rows * (cols // be)
    words = torch.randint(-2**63, 2**63 - 1, ((n * bb + 7) // 8,), dtype=torch.int64, device="cuda", generator=g)
    b = words.view(torch.uint8)[: n * bb].view(n, bb)
    spread = 0.75 + 0.5 * torch.rand(n, device="cuda", generator=g)

    def put(at: int, scale: float):
        b[:, at:at + 2] = (spread * scale).to(torch.float16).view(torch.uint8).view(n, 2)

    if qtype == quant.Q8_0:            # quants -128 .. 127
        put(0, std / 73.9)
    elif qtype == quant.Q4_0:          # quants 0 .. 15, -8: half a step off the mean
        put(0, std / 4.61)
    elif qtype in (quant.Q4_K, quant.Q5_K):
        # 6-bit sub-block scales 32 .. 63 and minimums of the same size (the header's packed bytes), quants 0 .. 15 or 0 .. 31
        mid, dev = (7.5, 4.61) if qtype == quant.Q4_K else (15.5, 9.23)
        b[:, 4:8] |= 0xA0
        b[:, 8:12] = b[:, 4:8]
        low = b[:, 12:16] & 0x0F
        b[:, 12:16] = low | (low << 4)
        put(0, std / (48.4 * dev))
        put(2, mid * std / (48.4 * dev))
    elif qtype == quant.Q6_K:          # scales of either sign, 64 .. 127 in size; quants -32 .. 31
        s = b[:, 192:208]
        b[:, 192:208] = torch.where(s >= 128, (s & 0x3F) + 129, (s & 0x3F) | 0x40)
        put(208, std / (97.2 * 18.5))
    return b.view(rows, -1)


def with_scale(blocks: torch.Tensor, qtype: int, factor: float) -> torch.Tensor:
    """The same blocks (Q6_K or Q8_0) with every scale multiplied."""
    at = 208 if qtype == quant.Q6_K else 0
    b = blocks.clone().view(-1, quant.BLOCK_BYTES[qtype])
    d = b[:, at:at + 2].contiguous().view(torch.float16).to(torch.float32) * factor
    b[:, at:at + 2] = d.to(torch.float16).view(torch.uint8).view(-1, 2)
    return b.view(blocks.shape)


def config_of(case: dict) -> Llama2Config:
    return Llama2Config(case["hidden"], case["ffn"], case["layers"], case["heads"], case["kv_heads"], case["vocab"], case["context"], 500000.0, 1e-5)


def norm_weight(g: torch.Generator, n: int) -> torch.Tensor:
    return 1.0 + WEIGHT_STD * torch.randn(n, device="cuda", generator=g)


def make_model(case: dict, g: torch.Generator, kv: str) -> tuple[Llama2, Llama2Weights]:
    cfg, recipe = config_of(case), RECIPES[case["recipe"]]
    shapes = cfg.shapes()
    layers = []
    for _ in range(cfg.num_hidden_layers):
        lw = {n: (recipe[n], random_matrix(g, recipe[n], *shapes[n], WEIGHT_STD)) for n in LAYER_MATS}
        lw["attn_norm"], lw["ffn_norm"] = norm_weight(g, cfg.hidden_size), norm_weight(g, cfg.hidden_size)
        layers.append(lw)
    qt = recipe["output"]
    embd = random_matrix(g, qt, cfg.vocab_size, cfg.hidden_size, EMBEDDING_STD)
    successor = torch.randperm(cfg.vocab_size, device="cuda", generator=g)
    weights = {"layers": layers, "token_embd": (qt, embd), "output": (qt, with_scale(embd[successor], qt, WEIGHT_STD / EMBEDDING_STD)),
               "output_norm": norm_weight(g, cfg.hidden_size)}
    dev = Llama2Weights(backend(), cfg, weights)
    return Llama2(backend(), cfg, dev, kv_f16=kv == F16), dev


def prepare(case: dict, seed: int):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("gemv", "gemm"):
        t, rows, cols = TYPES[case["type"]], case["rows"], case["cols"]
        s["m"] = GpuQuantTensor(backend(), t, rows, cols, random_matrix(g, t, rows, cols, WEIGHT_STD))
        n = case.get("tokens")
        s["x"] = torch.randn((n, cols) if n else (cols,), device="cuda", generator=g)
        s["out"] = torch.empty((n, rows) if n else (rows,), device="cuda")
        s["op"] = (GemmQuant if n else GemvQuant)(backend())
    elif kind == "attention":
        nh, nkv, hs, ctx = case["heads"], case["kv_heads"], case["head_size"], case["context"]
        dtype = torch.float16 if case["kv"] == F16 else torch.float32
        s["k"], s["v"] = (torch.randn(ctx, nkv * hs, device="cuda", generator=g).to(dtype) for _ in range(2))
        s["q"], s["out"] = torch.randn(nh * hs, device="cuda", generator=g), torch.empty(nh * hs, device="cuda")
        s["params"], s["op"] = AttnParams(ctx, nkv * hs, nh // nkv, nh, hs, ctx - 1), FusedAttention(backend())
    elif kind == "sample":
        # a ranked distribution over a shuffled vocabulary, with some noise on every logit
        n = case["vocab"]
        rank = torch.randperm(n, device="cuda", generator=g).to(torch.float32) + 1.0
        s["logits"] = -case["zipf"] * max(case["temperature"], 0.6) * torch.log(rank) + 0.05 * torch.randn(n, device="cuda", generator=g) + 15.0
        s["coin"] = float(rng.random())
        s["sampler"] = Sampler(backend(), n, case["temperature"], case["topp"])
        s["out"] = torch.empty(1, dtype=torch.int32, device="cuda")
    elif kind == "layer":
        h, f, nh, nkv, ctx = case["hidden"], case["ffn"], case["heads"], case["kv_heads"], case["context"]
        cfg, recipe = Llama2Config(h, f, case["layers"], nh, nkv, 32000, ctx, 500000.0, 1e-5), RECIPES[case["recipe"]]
        shapes, dtype = cfg.shapes(), torch.float16 if case["kv"] == F16 else torch.float32
        s["layers"] = []
        for _ in range(case["layers"]):
            lw = {n: GpuQuantTensor(backend(), recipe[n], *shapes[n], random_matrix(g, recipe[n], *shapes[n], WEIGHT_STD)) for n in LAYER_MATS}
            lw["attn_norm"], lw["ffn_norm"] = norm_weight(g, h), norm_weight(g, h)
            lw["k"], lw["v"] = (torch.randn(ctx, cfg.kv_dim, device="cuda", generator=g).to(dtype) for _ in range(2))
            s["layers"].append(lw)
        s["embedding"] = torch.randn(h, device="cuda", generator=g)
        s.update({n: torch.empty(w, device="cuda") for n, w in dict(x=h, xb=h, xb2=h, q=h, k=cfg.kv_dim, v=cfg.kv_dim, hb=f, hb2=f).items()})
        b = backend()
        s["ops"] = RmsNorm(b), GemvQuant(b), RoPE(b), FusedAttention(b), Silu(b)
        s["params"] = AttnParams(ctx, cfg.kv_dim, cfg.kv_mul, nh, cfg.head_size, case["pos"])
        s["rope"], s["norm"] = RoPEConfig(cfg.head_size, cfg.kv_dim, case["pos"], 500000.0), RmsNormConfig(1e-5)
    else:
        s["model"], s["weights"] = m, _ = make_model(case, g, case.get("kv", F16))
        pos = case["pos"]
        if pos:        # the conversation so far
            earlier = rng.integers(0, case["vocab"], pos).astype(np.uint32)
            if case.get("kv", F16) == F16 and case["heads"] == 4 * case["kv_heads"]:
                m.prefill(earlier)
            else:
                m.generate(earlier, 0)
        if case.get("temperature"):
            m.set_sampler(case["temperature"], case["topp"], seed=seed)
        n = case["prompt"] if kind == "turn" else (case["tokens"] if kind == "prefill" else 1)
        s["tokens"] = rng.integers(0, case["vocab"], n).astype(np.uint32)
        s["eos"] = 128001 if case["vocab"] > 128001 else 2
    return s


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------
def run_layers(s):
    """One token through the decoder layers, op by op, in the order of a token (q, k and v land where the cache wants them)."""
    rms, gemv, rope, attention, silu = s["ops"]
    b, pos, x, xb, xb2, q, hb, hb2 = backend(), s["case"]["pos"], s["x"], s["xb"], s["xb2"], s["q"], s["hb"], s["hb2"]
    f32 = s["case"]["kv"] == F32
    x.copy_(s["embedding"])
    for lw in s["layers"]:
        k, v = (lw["k"][pos], lw["v"][pos]) if f32 else (s["k"], s["v"])
        rms.launch(s["norm"], xb, x, lw["attn_norm"])
        gemv.launch(q, lw["attn_q"], xb)
        gemv.launch(k, lw["attn_k"], xb)
        gemv.launch(v, lw["attn_v"], xb)
        rope.launch(0, s["rope"], q, k)
        if not f32:
            lw["k"][pos].copy_(k)
            lw["v"][pos].copy_(v)
        attention.launch(s["params"], q, lw["k"], lw["v"], xb)
        gemv.launch(xb2, lw["attn_output"], xb)
        add_assign(b, x, xb2)
        rms.launch(s["norm"], xb, x, lw["ffn_norm"])
        gemv.launch(hb, lw["ffn_gate"], xb)
        gemv.launch(hb2, lw["ffn_up"], xb)
        silu.launch(hb, hb2)
        gemv.launch(xb, lw["ffn_down"], hb)
        add_assign(b, x, xb)
    return {"x": x, "k": [lw["k"][pos] for lw in s["layers"]], "v": [lw["v"][pos] for lw in s["layers"]]}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("gemv", "gemm"):
        s["op"].launch(s["out"], s["m"], s["x"])
        return s["out"]
    if kind == "attention":
        s["op"].launch(s["params"], s["q"], s["k"], s["v"], s["out"])
        return s["out"]
    if kind == "sample":
        if case["temperature"] == 0.0:
            argmax(backend(), s["logits"], s["out"])
            return s["out"]
        return s["sampler"].sample(s["logits"], s["coin"], s["out"])
    if kind == "layer":
        return run_layers(s)
    m, pos, tokens = s["model"], case["pos"], s["tokens"]
    if kind == "decode":
        return {"tokens": m.generate(tokens, case["tokens"], start_pos=pos), "logits": m.last_logits()}
    if kind == "forward":
        out, tok = [], int(tokens[0])
        for i in range(case["tokens"]):
            tok, logits = m.forward(tok, pos + i, want_logits=True)
            out.append(logits)
        return {"logits": out, "token": tok}
    if kind == "prefill":
        return {"token": m.prefill(tokens, start_pos=pos), "logits": m.last_logits()}
    first = m.prefill(tokens, start_pos=pos)
    rest = m.generate_until([first], case["tokens"] - 1, s["eos"], start_pos=pos + len(tokens))
    return {"first": first, "rest": rest, "logits": m.last_logits()}


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how near its results are defined
# ---------------------------------------------------------------------------------------------------------------------
def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("gemv", "gemm"):
        n, rows, cols = case.get("tokens", 1), case["rows"], case["cols"]
        return {"bytes": quant.matrix_bytes(TYPES[case["type"]], rows, cols) + 4 * n * (rows + cols), "flops": 2 * n * rows * cols}
    if kind == "attention":
        kv_dim, elem = case["kv_heads"] * case["head_size"], 2 if case["kv"] == F16 else 4
        return {"bytes": 2 * case["context"] * kv_dim * elem + 8 * case["heads"] * case["head_size"], "flops": 4 * case["context"] * case["heads"] * case["head_size"]}
    if kind == "sample":
        return {"bytes": 4 * case["vocab"], "flops": 4 * case["vocab"]}
    if kind == "layer":
        cfg, recipe = Llama2Config(case["hidden"], case["ffn"], case["layers"], case["heads"], case["kv_heads"], 32000, case["context"]), RECIPES[case["recipe"]]
        n, first, logits = 1, case["pos"], 0
    else:
        cfg, recipe, first = config_of(case), RECIPES[case["recipe"]], case["pos"]
        n = {"turn": case.get("prompt", 0)}.get(kind, case["tokens"])
        logits = 1 if kind in ("prefill", "turn") else n
    sh, layers = cfg.shapes(), cfg.num_hidden_layers
    layer_bytes = layers * (sum(quant.matrix_bytes(recipe[m], *sh[m]) for m in LAYER_MATS) + 8 * cfg.hidden_size)
    head_bytes = quant.matrix_bytes(recipe["output"], *sh["output"]) + 4 * cfg.vocab_size
    kv_row = cfg.kv_bytes_per_position(case.get("kv", F16) == F16)

    def tokens_at(at: int, count: int, passes: int) -> dict:
        """`count` tokens from position `at` in `passes` readings of the layers' weights; each reading reads the cache before it."""
        seen = sum(at + i + 1 for i in range(count))
        return {"bytes": passes * (layer_bytes + kv_row * at) + kv_row * (count if passes == 1 else sum(range(count)) + count),
                "flops": count * 2 * cfg.matrix_params() + 4 * seen * layers * cfg.hidden_size}

    w = tokens_at(first, n, 1 if kind in ("prefill", "turn", "layer") else n)
    if kind != "layer":
        w["bytes"] += logits * head_bytes
        w["flops"] += logits * 2 * cfg.hidden_size * cfg.vocab_size
    if kind == "turn":
        more = tokens_at(first + n, case["tokens"] - 1, case["tokens"] - 1)
        w["bytes"] += more["bytes"] + (case["tokens"] - 1) * head_bytes
        w["flops"] += more["flops"] + (case["tokens"] - 1) * 2 * cfg.hidden_size * cfg.vocab_size
    return w


def tolerance(case: dict):
    """Decode activations are 16-bit block fixed point (2^-15 of a group's largest value, ~1e-4 of a product's norm), the cache
    is f16 (2^-11), the sums are f32; prompt inputs are split into two f16.  Through a whole model these differences add up over
    its layers.  A token is a whole number and stays the same, but for a sampled one's coin at a boundary."""
    kind = case["kind"]
    if kind == "gemv":
        return {"rel": 5e-5 if case["type"] == "Q4_0" else 3e-4}
    if kind == "gemm":
        return {"rel": 5e-5}
    if kind == "attention":
        return {"rel": 2e-5, "max": 1e-3}
    if kind == "sample":
        return "exact"
    if kind == "layer":
        return {"rel": 2e-3}
    return {"rel": 5e-3, "max": 0.1}
