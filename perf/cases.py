"""The work this library is timed on: its ops and its decoder through the public entry points, over the ranges users run.

The sizes are those of the repository's own configurations: the projections of a Llama-3-8B-architecture decoder
(d 4096, 32 query / 8 KV heads of 128, FFN 14336) and the small 896 -> 896 / 4864 layers, batches of 1 to 64 at
decode, prompts of hundreds to thousands of tokens, caches of 1 to 32768 keys, bf16 / fp16 / fp32, packed 4- and
8-bit weights in groups of 32, 64 and 128.
"""

import math

import torch

import mlx_batch_invariant_b200 as bi
from mlx_batch_invariant_b200.runner import LLAMA3_8B, GraphedDecoder, ShardedDecoder
from mlx_batch_invariant_b200.runner.decoder import quantize_rows

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}
EPS = 1e-5
FFN, D_MODEL = 14336, 4096


def listed():
    return [
        # one token's hidden state through a norm: the smallest call a decode loop makes
        {"name": "norm_token", "op": "rms_norm", "rows": 1, "dim": 4096, "dtype": "bf16"},
        # the hidden states of a long (odd) prompt batch
        {"name": "norm_prompt", "op": "rms_norm", "rows": 4093, "dim": 4096, "dtype": "bf16"},
        # a single sequence decoding: one row against a square projection
        {"name": "linear_token", "op": "linear", "rows": 1, "in": 4096, "out": 4096, "dtype": "bf16", "bias": False},
        # a full decode batch through the FFN's down projection
        {"name": "linear_batch", "op": "linear", "rows": 64, "in": FFN, "out": 4096, "dtype": "bf16", "bias": False},
        # a ragged prompt through the FFN's up projection, in the other 16-bit type
        {"name": "linear_prompt", "op": "linear", "rows": 1900, "in": 4096, "out": FFN, "dtype": "fp16", "bias": False},
        # full-precision users (evaluation, small models): no tensor cores
        {"name": "linear_fp32", "op": "linear", "rows": 100, "in": 4096, "out": 4096, "dtype": "fp32", "bias": False},
        # a single sequence decoding with 4-bit weights
        {"name": "packed_token", "op": "packed", "rows": 1, "in": 4096, "out": FFN, "bits": 4, "group": 64, "dtype": "bf16"},
        # a short ragged prompt on 8-bit weights with fine groups
        {"name": "packed_prompt", "op": "packed", "rows": 300, "in": 4096, "out": 4096, "bits": 8, "group": 32, "dtype": "bf16"},
        # a decode batch of mixed ages reading a shared, partly filled cache
        {"name": "decode_mixed", "op": "decode", "batch": 64, "keys": 4096, "mixed": True, "heads": 32, "kv_heads": 8,
         "dim": 128, "dtype": "bf16"},
        # one-shot causal prefill of a 2048-token prompt
        {"name": "prefill", "op": "prefill", "batch": 1, "tokens": 2048, "cached": 0, "heads": 32, "kv_heads": 8,
         "dim": 128, "dtype": "bf16"},
        # the serving step of the whole decoder: 64 sequences, one greedy token each, replayed from a CUDA graph
        {"name": "model_step", "op": "model_step", "batch": 64, "position": 560, "bits": 16},
        # time to first token of two 512-token prompts on the 4-bit decoder
        {"name": "model_prompt", "op": "model_prompt", "batch": 2, "tokens": 512, "bits": 4},
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], uniform in its logarithm."""
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    op = rng.choice(["rms_norm", "linear", "linear", "linear", "packed", "packed", "decode", "decode", "prefill", "model"])
    half = rng.choice(["bf16", "bf16", "fp16"])
    shapes = [(896, 896), (896, 4864), (4864, 896), (4096, 4096), (4096, 6144), (4096, FFN), (FFN, 4096), (4096, 2 * FFN)]
    if op == "rms_norm":
        return {"op": op, "rows": _log(rng, 1, 8192), "dim": rng.choice([896, 4096, 4096, _log(rng, 100, 8192)]),
                "dtype": rng.choice([half, half, "fp32"])}
    if op == "linear":
        k, n = rng.choice(shapes + [(8 * _log(rng, 32, 1024), _log(rng, 100, 8192))] * 2)
        if rng.random() < 0.2:
            return {"op": op, "rows": _log(rng, 1, 256), "in": k, "out": n, "dtype": "fp32", "bias": rng.random() < 0.25}
        return {"op": op, "rows": _log(rng, 1, 2048), "in": k, "out": n, "dtype": half, "bias": rng.random() < 0.25}
    if op == "packed":
        k, n = rng.choice(shapes + [(128 * _log(rng, 2, 64), _log(rng, 100, 8192))] * 2)
        return {"op": op, "rows": _log(rng, 1, 2048), "in": k, "out": n, "bits": rng.choice([4, 4, 8]),
                "group": rng.choice([g for g in (32, 64, 64, 128) if k % g == 0]), "dtype": half}
    heads, kv, dim = rng.choice([(32, 8, 128), (32, 8, 128), (8, 2, 128), (14, 2, 64)])
    half = rng.choice([half] * 7 + ["fp32"])
    if op == "decode":
        batch = _log(rng, 1, 64)
        return {"op": op, "batch": batch, "keys": _log(rng, 1, min(32768, 64 * 4096 // batch)), "mixed": rng.random() < 0.5,
                "heads": heads, "kv_heads": kv, "dim": dim, "dtype": half}
    if op == "prefill":
        tokens = _log(rng, 16, 2048)
        return {"op": op, "batch": _log(rng, 1, max(1, 2048 // tokens)), "tokens": tokens, "cached": rng.choice([0, 0, _log(rng, 1, 1024)]),
                "heads": heads, "kv_heads": kv, "dim": dim, "dtype": half}
    if rng.random() < 0.7:
        return {"op": "model_step", "batch": _log(rng, 1, 64), "position": rng.randint(32, 560), "bits": rng.choice([16, 4])}
    batch = rng.randint(1, 2)
    return {"op": "model_prompt", "batch": batch, "tokens": _log(rng, 32, 512), "bits": rng.choice([16, 4])}


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(g, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=g, device="cuda") * std).to(dtype)


def prepare(case, seed):
    g, op = _gen(seed), case["op"]
    s = {"op": op, "case": case}
    if op.startswith("model"):
        return _prepare_model(case, seed, g, s)
    dt = DTYPES[case["dtype"]]
    if op == "rms_norm":
        s["x"] = _normal(g, case["rows"], case["dim"], std=3.0, dtype=dt)
        s["w"] = (1 + _normal(g, case["dim"], std=0.1)).to(dt)
    elif op in ("linear", "packed"):
        m, k, n = case["rows"], case["in"], case["out"]
        s["x"] = _normal(g, m, k, dtype=dt)
        if op == "linear":
            s["w"] = _normal(g, n, k, std=k ** -0.5, dtype=dt)
            s["bias"] = _normal(g, n, dtype=dt) if case["bias"] else None
        else:
            s["w"] = quantize_rows(_normal(g, n, k, std=0.02, dtype=dt), case["group"], case["bits"])
    elif op == "decode":
        b, n, d = case["batch"], case["keys"], case["dim"]
        s["q"] = _normal(g, b, case["heads"], 1, d, dtype=dt)
        s["k"], s["v"] = (_normal(g, b, case["kv_heads"], n, d, dtype=dt) for _ in range(2))
        # mixed: every sequence has its own age, from one key to the whole cache, most of them in between
        lens = torch.randint(1, n + 1, (b,), generator=g, device="cuda", dtype=torch.int32)
        s["lens"] = lens if case["mixed"] else None
    else:
        b, t, d = case["batch"], case["tokens"], case["dim"]
        s["q"] = _normal(g, b, case["heads"], t, d, dtype=dt)
        s["k"], s["v"] = (_normal(g, b, case["kv_heads"], case["cached"] + t, d, dtype=dt) for _ in range(2))
    return s


def _prepare_model(case, seed, g, s):
    """A decoder with random weights. For a step, the caches hold random keys and values of the size the random weights
    would produce (a prompt's worth of prefill is not part of the path), and the step is captured once."""
    b = case["batch"]
    step = case["op"] == "model_step"
    length = case["position"] + 1 if step else case["tokens"]
    m = ShardedDecoder(LLAMA3_8B, quant=None if case["bits"] == 16 else (case["bits"], 64), seed=seed, max_batch=b, max_len=(length + 63) // 64 * 64)
    s["model"] = m
    if step:
        std = LLAMA3_8B.init_std * LLAMA3_8B.d_model ** 0.5
        for c in m.kc + m.vc:
            c[:, :, :case["position"]].normal_(0.0, std, generator=g)
        s["first"] = torch.randint(0, LLAMA3_8B.vocab, (b,), generator=g, device="cuda")
        s["decoder"] = GraphedDecoder(m, b)
        s["decoder"].start(s["first"], case["position"])
        s["decoder"].capture()
    else:
        s["tokens"] = torch.randint(0, LLAMA3_8B.vocab, (b, case["tokens"]), generator=g, device="cuda")
    return s


def run(state):
    op, c = state["op"], state["case"]
    if op == "rms_norm":
        return bi.batch_invariant_rms_norm(state["x"], state["w"], EPS)
    if op == "linear":
        if state["bias"] is None:
            return bi.batch_invariant_matmul(state["x"], state["w"].T)
        return bi.batch_invariant_matmul(state["x"], state["w"].T, bias=state["bias"])
    if op == "packed":
        codes, scales, biases = state["w"]
        return bi.batch_invariant_quantized_matmul(state["x"], codes, scales, biases, group_size=c["group"], bits=c["bits"])
    if op == "decode":
        return bi.batch_invariant_decode_attention(state["q"], state["k"], state["v"], scale=c["dim"] ** -0.5, kv_lens=state["lens"])
    if op == "prefill":
        return bi.batch_invariant_attention(state["q"], state["k"], state["v"], scale=c["dim"] ** -0.5, mask="causal")
    if op == "model_step":
        d = state["decoder"]
        d.start(state["first"], c["position"])
        logits = d.step()
        return {"logits": logits, "tokens": d.tokens, "position": d.pos, "lengths": d.lens}
    return state["model"].forward(state["tokens"], 0)


def _attention(batch_pairs, heads, dim):
    return 4.0 * heads * dim * batch_pairs


def work(case):
    op = case["op"]
    if op.startswith("model"):
        m = LLAMA3_8B
        head = m.vocab * m.d_model
        layer = m.d_model * (m.n_heads + 2 * m.n_kv_heads) * m.head_dim + m.n_heads * m.head_dim * m.d_model + 3 * m.ffn * m.d_model
        per_weight = 2.0 if case["bits"] == 16 else case["bits"] / 8 + 4 / 64
        b = case["batch"]
        kv_row = 2 * m.n_kv_heads * m.head_dim * 2 * m.n_layers          # bytes a token takes in the caches
        if op == "model_step":
            tokens, pairs, kv = b, b * (case["position"] + 1), b * (case["position"] + 1) * kv_row
        else:
            t = case["tokens"]
            tokens, pairs, kv = b * t, b * t * (t + 1) // 2, b * t * kv_row
        weights = m.n_layers * layer + head
        return {"bytes": weights * per_weight + kv + tokens * m.d_model * 2 + b * m.vocab * 2,
                "flops": 2.0 * (m.n_layers * layer * tokens + head * b) + m.n_layers * _attention(pairs, m.n_heads, m.head_dim)}
    e = SIZE[case["dtype"]]
    if op == "rms_norm":
        n = case["rows"] * case["dim"]
        return {"bytes": e * (2.0 * n + case["dim"]), "flops": 4.0 * n}
    if op in ("linear", "packed"):
        m, k, n = case["rows"], case["in"], case["out"]
        weight = e * n * k if op == "linear" else n * k * (case["bits"] / 8 + 2 * e / case["group"])
        return {"bytes": float(weight + e * m * (k + n)), "flops": 2.0 * m * n * k}
    q = 2.0 * e * case["batch"] * case["heads"] * case["dim"]            # queries in, outputs out, per query position
    kv = 2.0 * e * case["batch"] * case["kv_heads"] * case["dim"]        # a key and a value of every sequence
    if op == "decode":
        keys = (case["keys"] + 1) / 2 if case["mixed"] else case["keys"]  # mixed: the mean of the lengths drawn
        return {"bytes": q + kv * keys, "flops": _attention(case["batch"] * keys, case["heads"], case["dim"])}
    t, l = case["tokens"], case["cached"] + case["tokens"]
    pairs = case["batch"] * (t * case["cached"] + t * (t + 1) // 2)
    return {"bytes": q * t + kv * l, "flops": _attention(pairs, case["heads"], case["dim"])}


def tolerance(case):
    """What the types give: one rounding of an fp32 sum to a 16-bit output, or fp32 sums in another order."""
    if case["op"].startswith("model"):
        return {"rel": 0.02, "max": 0.3, "differ": 0.01}                 # bf16 roundings carried through 32 layers; argmax ties
    if case["dtype"] == "fp32":
        return {"rel": 1e-5}
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3}
