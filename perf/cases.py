"""The work whose time counts: what a program that generates with this library has it do.

Every case is one pass through public entry points: a whole step loop through ``tb.Engine``, or one layer's work through
``trapetum_b200.csrc.ops`` as the parts of a layer (and programs that register parts of their own) call it.  Sizes are
those of the Gemma-2 shapes and of the medium models of the other architectures in ``bench.py``; lengths are ragged as
requests are.  ``draw`` spreads each kind over the sizes that it stands for.
"""
import math

import torch

import trapetum_b200 as tb
from trapetum_b200.csrc import ops

DEV = "cuda:0"
BF, F32, F64, I32 = torch.bfloat16, torch.float32, torch.float64, torch.int32
PAGE = ops.PAGE_ROWS
EPS = 1e-6

# heads, kv heads, head size, hidden size, intermediate size of the Gemma-2 shapes and of a medium model
SHAPES = {"2b": (8, 4, 256, 2304, 9216), "9b": (16, 8, 256, 3584, 14336), "27b": (32, 16, 128, 4608, 36864),
          "medium": (16, 4, 128, 2048, 8192)}
VOCAB = 256000


def listed():
    return [
        # Token-by-token generation for a batch of chat requests of unequal length: short prompts, then eight decode
        # steps.  Latency and launches count.
        {"name": "model_decode", "kind": "model", "lens": "17,64,5,131,40,96,23,8", "steps": 8},
        # Time to the first token of one long request.
        {"name": "model_prompt", "kind": "model", "lens": "2048", "steps": 0},
        # Decode attention of a layer with all keys, eight requests in long contexts of unequal length.
        {"name": "attn_decode", "kind": "attn_decode", "shape": "2b", "lens": "8192,7900,8000,6500,8100,7333,8191,7001", "cap": 50.0},
        # Prompt attention of a larger model's layer, an odd length with the soft cap.
        {"name": "attn_prompt", "kind": "attn_prompt", "shape": "9b", "lens": "2999", "window": 4096, "cap": 50.0},
        # The gated feed-forward of a 9B layer over the packed prompts of a small batch.
        {"name": "mlp_prompt", "kind": "mlp", "shape": "9b", "tokens": 1000, "dtype": "bfloat16"},
        # The true 32-bit path, with which results are checked, on a 2B layer's feed-forward.
        {"name": "mlp_float32", "kind": "mlp", "shape": "2b", "tokens": 300, "dtype": "float32"},
        # Output head and nucleus sampling of a batch of 64 requests over the whole vocabulary.
        {"name": "head_sample", "kind": "head", "rows": 64, "hidden": 2304, "vocab": VOCAB, "top_p": 0.95, "penalty": 1.1},
        # A state-space layer (Divanex, Sezanex) over one long prompt.
        {"name": "mamba2_prompt", "kind": "mamba2", "lens": "2048", "heads": 64, "state": 128},
        # Gated linear attention (Lofirax) over two prompts of unequal length.
        {"name": "gla_prompt", "kind": "gla", "lens": "1500,548", "heads": 8},
        # Decode attention over cached latents with a sink (Lofirax, Fibelix): 64 requests.
        {"name": "latent_decode", "kind": "latent", "batch": 64, "context": 2048, "heads": 16},
        # Attention with scores mixed across heads (Fibelix) over one prompt, blocks of 1,024 positions.
        {"name": "mixed_prompt", "kind": "mixed", "lens": "2048", "heads": 16, "kv_heads": 4, "block": 1024},
        # Routing and experts of a decode step of eight requests (the weights are what is read).
        {"name": "moe_decode", "kind": "moe", "tokens": 8, "gated": True, "width": 2048, "ff": 1024},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lens(rng, n, total):
    """n unequal lengths that add up to about ``total``."""
    w = [rng.uniform(0.2, 1.0) for _ in range(n)]
    return ",".join(str(max(1, int(total * x / sum(w)))) for x in w)


def draw(rng):
    kind = rng.choice(["model", "attn_decode", "attn_prompt", "mlp", "mlp32", "head", "mamba2", "gla", "latent", "mixed", "moe"])
    if kind == "model":
        if rng.random() < 0.5:
            return {"kind": kind, "lens": _lens(rng, rng.randint(1, 4), _log(rng, 100, 2000)), "steps": 0}
        n = rng.randint(1, 8)
        return {"kind": kind, "lens": _lens(rng, n, _log(rng, 8 * n, 384)), "steps": rng.randint(2, 8)}
    if kind == "attn_decode":
        n = rng.randint(1, 16)
        return {"kind": kind, "shape": rng.choice(["2b", "9b", "27b", "medium"]), "cap": rng.choice([0.0, 50.0]),
                "lens": ",".join(str(_log(rng, 300, 8192)) for _ in range(n))}
    if kind == "attn_prompt":
        return {"kind": kind, "shape": rng.choice(["2b", "9b", "27b", "medium"]), "cap": rng.choice([0.0, 50.0]),
                "window": rng.choice([0, 1024, 4096]), "lens": _lens(rng, rng.randint(1, 4), _log(rng, 200, 4000))}
    if kind == "mlp":
        return {"kind": kind, "shape": rng.choice(["2b", "9b", "medium"]), "tokens": _log(rng, 1, 2048), "dtype": "bfloat16"}
    if kind == "mlp32":
        return {"kind": "mlp", "shape": rng.choice(["2b", "medium"]), "tokens": _log(rng, 1, 400), "dtype": "float32"}
    if kind == "head":
        return {"kind": kind, "rows": _log(rng, 1, 64), "hidden": rng.choice([2048, 2304, 3584]), "vocab": rng.choice([65536, VOCAB]),
                "top_p": rng.choice([0.9, 0.95, 1.0]), "penalty": rng.choice([1.0, 1.1])}
    if kind == "mamba2":
        return {"kind": kind, "lens": _lens(rng, rng.randint(1, 4), _log(rng, 100, 3000)), "heads": rng.choice([32, 48, 64]),
                "state": rng.choice([64, 128])}
    if kind == "gla":
        return {"kind": kind, "lens": _lens(rng, rng.randint(1, 4), _log(rng, 100, 3000)), "heads": rng.choice([4, 8, 16])}
    if kind == "latent":
        return {"kind": kind, "batch": _log(rng, 1, 64), "context": _log(rng, 300, 4096), "heads": rng.choice([16, 32])}
    if kind == "mixed":
        return {"kind": kind, "lens": _lens(rng, rng.randint(1, 3), _log(rng, 100, 2500)), "heads": rng.choice([8, 16]),
                "kv_heads": rng.choice([2, 4]), "block": rng.choice([512, 1024])}
    return {"kind": "moe", "tokens": _log(rng, 1, 512), "gated": rng.choice([True, False]), "width": rng.choice([1024, 2048]),
            "ff": rng.choice([512, 1024])}


# ---------------------------------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------------------------------
class _Rand:
    """Seeded tensors on the device."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(seed)
        self.host = torch.Generator().manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=F32):
        out = torch.empty(shape, dtype=dtype, device=DEV)
        out.normal_(0.0, std, generator=self.g)
        return out

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(shape, device=DEV, generator=self.g) * (hi - lo) + lo

    def perm(self, n):
        return torch.randperm(n, generator=self.host)

    def ids(self, n, hi):
        return torch.randint(0, hi, (n,), generator=self.host).tolist()


def _ints(case, key="lens"):
    return [int(x) for x in case[key].split(",")]


def _packed(lens):
    """Index tensors of a step of whole prompts packed back to back."""
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    i32 = dict(dtype=I32, device=DEV)
    return {"starts": starts, "seq_start": torch.tensor(starts, **i32), "slots": torch.arange(len(lens), **i32),
            "token_seq": torch.cat([torch.full((n,), b) for b, n in enumerate(lens)]).to(**i32)}


def _tables(r, lens):
    """A page table over a pool whose pages are handed out in no order, as they are after some use of a cache."""
    pages = [(n + PAGE - 1) // PAGE for n in lens]
    perm = r.perm(sum(pages)).tolist()
    table = torch.zeros(len(lens), max(pages), dtype=I32)
    at = 0
    for b, n in enumerate(pages):
        table[b, :n] = torch.tensor(perm[at:at + n], dtype=I32)
        at += n
    return sum(pages), table.to(DEV)


def _bucket(n):
    """The engine's bucket of a context length: launch shapes depend on it alone."""
    b = 256
    while b < n:
        b *= 2
    return b


def _uneven(lens):
    """How much the contexts differ, in quarters, as the engine hands it to decode attention."""
    return max(0, min(3, 3 - 4 * sum(lens) // (len(lens) * max(lens)))) if len(lens) > 1 else 0


def _config():
    h, g, d, hidden, ff = SHAPES["2b"]
    return {"architectures": ["Gemma2ForCausalLM"], "model_type": "gemma2", "num_hidden_layers": 26, "hidden_size": hidden,
            "num_attention_heads": h, "num_key_value_heads": g, "head_dim": d, "intermediate_size": ff, "vocab_size": VOCAB,
            "rope_theta": 10000.0, "sliding_window": 4096, "query_pre_attn_scalar": 256, "attn_logit_softcapping": 50.0,
            "final_logit_softcapping": 30.0, "rms_norm_eps": EPS, "hidden_activation": "gelu_pytorch_tanh",
            "tie_word_embeddings": True, "max_position_embeddings": 8192}


def prepare(case, seed):
    r = _Rand(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "model":
        lens = _ints(case)
        model = tb.random_model(_config(), seed=seed)
        s["engine"] = tb.Engine(model, max_tokens=sum((n + case["steps"] + PAGE) // PAGE * PAGE for n in lens) + PAGE, max_slots=len(lens))
        s["prompts"] = [r.ids(n, VOCAB) for n in lens]
        s["tokens"] = [r.ids(len(lens), VOCAB) for _ in range(case["steps"])]
    elif kind == "attn_decode":
        h, g, d = SHAPES[case["shape"]][:3]
        lens = _ints(case)
        n, s["table"] = _tables(r, lens)
        s["q"] = r.normal(len(lens), h * d, dtype=BF)
        s["k"], s["v"] = r.normal(n, g, PAGE, d, dtype=BF), r.normal(n, g, PAGE, d, dtype=BF)
        s["lens"] = torch.tensor(lens, dtype=I32, device=DEV)
        s["bucket"], s["uneven"] = _bucket(max(lens)), _uneven(lens)
    elif kind == "attn_prompt":
        h, g, d = SHAPES[case["shape"]][:3]
        s.update(_packed(_ints(case)))
        qkv = r.normal(s["starts"][-1], (h + 2 * g) * d, dtype=BF)          # the fused product's rows, sliced as the part does
        s["q"], s["k"], s["v"] = qkv[:, :h * d], qkv[:, h * d:(h + g) * d], qkv[:, (h + g) * d:]
    elif kind == "mlp":
        hidden, ff = SHAPES[case["shape"]][3:]
        dt = BF if case["dtype"] == "bfloat16" else F32
        s["x"] = r.normal(case["tokens"], hidden, dtype=dt)
        s["gate"], s["up"] = r.normal(ff, hidden, std=0.02, dtype=dt), r.normal(ff, hidden, std=0.02, dtype=dt)
        s["down"] = r.normal(hidden, ff, std=0.02, dtype=dt)
        s["gate_up"] = ops.interleave_gate_up(s["gate"], s["up"]) if dt == BF else torch.cat([s["gate"], s["up"]])
        del s["gate"], s["up"]
    elif kind == "head":
        rows = case["rows"]
        s["x"] = r.normal(rows, case["hidden"], dtype=BF)
        s["w"] = r.normal(case["vocab"], case["hidden"], std=0.05, dtype=BF)
        s["temperature"] = torch.full((rows,), 0.8, device=DEV)
        s["top_p"] = torch.full((rows,), case["top_p"], device=DEV)
        s["penalty"] = torch.full((rows,), case["penalty"], device=DEV)
        s["draw"] = r.uniform(rows)
        s["recent"] = torch.randint(0, case["vocab"], (rows, 128), device=DEV, dtype=I32, generator=r.g) if case["penalty"] != 1.0 else None
    elif kind == "mamba2":
        H, P, N = case["heads"], 64, case["state"]
        lens = _ints(case)
        s.update(_packed(lens))
        T, inner, ch = s["starts"][-1], H * P, H * P + 2 * N
        s["proj"], s["dt"] = r.normal(T, inner + ch, dtype=BF), r.normal(T, H)
        s["conv_w"], s["conv_b"] = r.normal(ch, 4, std=0.3), r.normal(ch, std=0.1)
        s["dt_bias"], s["A_log"], s["D"] = r.normal(H) - 2.0, r.normal(H, std=0.5), r.normal(H)
        s["norm"] = r.normal(inner, std=0.1) + 1.0
        s["state"] = torch.zeros(len(lens), ops.mamba2_state_size(H, P, N, 1, 4), device=DEV)
    elif kind == "gla":
        H, D, V, rank = case["heads"], 128, 256, 16
        lens = _ints(case)
        s.update(_packed(lens))
        T = s["starts"][-1]
        s["proj"], s["low"] = r.normal(T, 2 * H * (D + V), dtype=BF), r.normal(1, T, rank)
        s["a2"], s["a2_bias"] = r.normal(H * D, rank, std=0.3), r.normal(H * D) + 2.0
        s["norm"] = r.normal(V, std=0.1) + 1.0
        s["state"] = torch.zeros(len(lens), H * D * V, device=DEV)
    elif kind == "latent":
        C, R, B = 448, 64, case["batch"]
        lens = [max(1, case["context"] - (37 * b) % (case["context"] // 4)) for b in range(B)]
        n, s["table"] = _tables(r, lens)
        s["pool"] = r.normal(n, 1, PAGE, C + R, dtype=BF)
        s["q"] = r.normal(B, case["heads"] * (C + R), dtype=BF)
        s["sink"] = r.normal(case["heads"])
        s["lens"], s["host_lens"] = torch.tensor(lens, dtype=I32, device=DEV), lens
        s["bucket"] = _bucket(max(lens))
    elif kind == "mixed":
        H, G, d = case["heads"], case["kv_heads"], 128
        s.update(_packed(_ints(case)))
        T = s["starts"][-1]
        s["q"], s["k"], s["v"] = (r.normal(T, n * d, dtype=BF) for n in (H, G, G))
        s["mix"] = (torch.eye(H, device=DEV) + r.normal(H, H, std=0.1)) * d ** -0.5
    elif kind == "moe":
        E, W, ff = 32, case["width"], case["ff"]
        s["x"] = r.normal(case["tokens"], W, dtype=BF)
        s["logits"] = r.normal(1, case["tokens"], E)
        s["gate"] = r.normal(E, ff, W, std=0.02, dtype=BF) if case["gated"] else None
        s["up"], s["down"] = r.normal(E, ff, W, std=0.02, dtype=BF), r.normal(E, W, ff, std=0.02, dtype=BF)
        s["gate_up"] = torch.stack([ops.interleave_gate_up(s["gate"][e], s["up"][e]) for e in range(E)]) if case["gated"] else None
    return s


# ---------------------------------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "model":
        e, out = s["engine"], []
        slots = e.start(len(s["prompts"]))
        out.append(e.step(slots, s["prompts"]))
        for tokens in s["tokens"]:
            out.append(e.step(slots, [[t] for t in tokens]))
        e.release(slots)
        return out
    if kind == "attn_decode":
        h, g, d = SHAPES[case["shape"]][:3]
        return ops.attn_decode(s["q"], s["k"], s["v"], s["table"], s["lens"], h, g, d, d ** -0.5, case["cap"], 0, 0, s["bucket"], s["uneven"])
    if kind == "attn_prompt":
        h, g, d = SHAPES[case["shape"]][:3]
        lens = _ints(case)
        return ops.attn_prefill(s["q"], s["k"], s["v"], s["seq_start"], s["token_seq"], h, g, d, d ** -0.5, case["cap"], case["window"],
                                max(lens), lens)
    if kind == "mlp":
        if case["dtype"] == "bfloat16":
            act = ops.gemm_tc(s["x"], s["gate_up"], BF, gated_act="gelu_tanh")
            return ops.gemm_tc(act, s["down"], F32)
        act = ops.gated_act(ops.gemm_simt(s["x"], s["gate_up"], F32), "gelu_tanh", F32)
        return ops.gemm_simt(act, s["down"], F32)
    if kind == "head":
        logits = ops.gemm_tc(s["x"], s["w"], F32, softcap=30.0)
        tokens = ops.sample(logits, s["temperature"], s["top_p"], s["penalty"], s["draw"], s["recent"], nucleus=case["top_p"] < 1.0)
        return {"logits": logits, "tokens": tokens}
    if kind == "mamba2":
        s["state"].zero_()                                               # a slot's state when a sequence claims it
        lens = _ints(case)
        out = ops.mamba2(s["proj"], s["dt"], case["heads"], 64, case["state"], 1, 4, 1, s["conv_w"], s["conv_b"], s["dt_bias"], s["A_log"],
                         s["D"], s["norm"], EPS, s["state"], s["seq_start"], s["token_seq"], s["slots"], len(lens), False, max(lens))
        return {"out": out, "state": s["state"]}
    if kind == "gla":
        s["state"].zero_()
        lens = _ints(case)
        out = ops.gla(s["proj"], s["low"], s["a2"], s["a2_bias"], 8.0, 128 ** -0.5, s["norm"], EPS, case["heads"], 128, 256, s["state"],
                      s["seq_start"], s["token_seq"], s["slots"], len(lens), max(lens))
        return {"out": out, "state": s["state"]}
    if kind == "latent":
        return ops.latent_decode(s["q"], s["pool"], s["table"], s["lens"], s["sink"], case["heads"], 448, 64, 0.07, s["bucket"])
    if kind == "mixed":
        return ops.attn_mixed_prefill(s["q"], s["k"], s["v"], s["seq_start"], s["token_seq"], case["heads"], case["kv_heads"], 128, s["mix"],
                                      -case["block"], True, max(_ints(case)))
    idx, weight, _ = ops.moe_route(s["logits"], 32, None, False, 4, 1, 1, 1, 1e-20, "softmax")
    return {"out": ops.moe_experts(s["x"], s["gate"], s["up"], s["down"], idx, weight, gate_up_w=s["gate_up"]), "idx": idx, "weight": weight}


# ---------------------------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def _pairs(n, window=0):
    """(query, key) pairs of a causal sequence of n tokens; window W: the last W keys."""
    return n * (n + 1) // 2 if not window or n <= window else window * (window + 1) // 2 + (n - window) * window


def work(case):
    kind = case["kind"]
    if kind == "model":
        h, g, d, hidden, ff = SHAPES["2b"]
        lens, steps, layers = _ints(case), case["steps"], 26
        matrices = layers * hidden * ((h + 2 * g) * d + h * d + 3 * ff)
        per_step = 2 * (matrices + VOCAB * hidden)
        kv = 4 * layers * g * d                                          # bytes a token leaves in the cache
        tokens = sum(lens) + steps * len(lens)
        read = sum(kv * (n + i) for n in lens for i in range(1, steps + 1))
        att = 4 * layers * h * d * (sum(_pairs(n, 0) for n in lens) + sum(n + i for n in lens for i in range(1, steps + 1)))
        rows = (steps + 1) * len(lens)
        return {"bytes": per_step * (steps + 1) + kv * tokens + read + rows * VOCAB * 4,
                "flops": 2 * matrices * tokens + att + 2 * VOCAB * hidden * rows}
    if kind == "attn_decode":
        h, g, d = SHAPES[case["shape"]][:3]
        lens = _ints(case)
        return {"bytes": sum(lens) * g * d * 4 + 4 * len(lens) * h * d, "flops": 4 * h * d * sum(lens)}
    if kind == "attn_prompt":
        h, g, d = SHAPES[case["shape"]][:3]
        lens = _ints(case)
        return {"bytes": sum(lens) * (2 * h + 2 * g) * d * 2, "flops": 4 * h * d * sum(_pairs(n, case["window"]) for n in lens)}
    if kind == "mlp":
        hidden, ff = SHAPES[case["shape"]][3:]
        size, T = (2 if case["dtype"] == "bfloat16" else 4), case["tokens"]
        return {"bytes": 3 * hidden * ff * size + T * hidden * (size + 4), "flops": 6 * T * hidden * ff}
    if kind == "head":
        rows, hidden, vocab = case["rows"], case["hidden"], case["vocab"]
        return {"bytes": vocab * hidden * 2 + rows * hidden * 2 + rows * vocab * 4 + rows * 4, "flops": 2 * rows * hidden * vocab}
    if kind == "mamba2":
        T, inner, N = sum(_ints(case)), case["heads"] * 64, case["state"]
        state = len(_ints(case)) * 4 * (inner * N + 3 * (inner + 2 * N))
        return {"bytes": T * (2 * (2 * inner + 2 * N) + 4 * case["heads"] + 2 * inner) + 2 * state, "flops": 5 * T * inner * N}
    if kind == "gla":
        T, H = sum(_ints(case)), case["heads"]
        return {"bytes": T * (2 * H * 768 + 4 * 16 + 2 * H * 256) + 2 * len(_ints(case)) * 4 * H * 128 * 256, "flops": 5 * T * H * 128 * 256}
    if kind == "latent":
        B, H, ctx = case["batch"], case["heads"], case["context"]
        rows = sum(max(1, ctx - (37 * b) % (ctx // 4)) for b in range(B))
        return {"bytes": rows * 512 * 2 + B * H * (512 + 448) * 2, "flops": 2 * H * (512 + 448) * rows}
    if kind == "mixed":
        H, G, blk, lens = case["heads"], case["kv_heads"], case["block"], _ints(case)
        pairs = sum((n // blk) * _pairs(blk) + _pairs(n % blk) for n in lens)
        return {"bytes": sum(lens) * (2 * H + 2 * G) * 128 * 2, "flops": pairs * (4 * H * 128 + 2 * H * H)}
    T, W, ff, mats = case["tokens"], case["width"], case["ff"], 3 if case["gated"] else 2
    used = 32 * (1 - (1 - 4 / 32) ** T)                                  # experts that some token chooses
    return {"bytes": used * mats * W * ff * 2 + T * W * 6 + T * 4 * 36, "flops": 2 * T * 4 * mats * W * ff}


def tolerance(case):
    kind = case["kind"]
    if kind == "model":
        return {"rel": 0.035}                    # 26 layers of bfloat16 activations: 0.007 to 0.009 from 64 bits
    if kind == "mlp" and case["dtype"] == "float32":
        return {"rel": 3e-6}                     # 6e-7 from 64 bits
    if kind == "head":
        return {"rel": 1e-5, "differ": 0.05}     # 2e-6 from 64 bits; a draw may fall on another token where a sum's last bit decides
    if kind == "moe":
        return {"rel": 1e-2, "differ": 0.0}
    return {"rel": 1e-2}                         # bfloat16 in and out, 32-bit between: 0.0017 to 0.0027 from 64 bits


# ---------------------------------------------------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------------------------------------------------
def _gelu_tanh(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _cap(x, cap):
    return cap * torch.tanh(x / cap) if cap else x


def _attention(q, k, v, scale, cap, window):
    """One causal sequence: q [T, h, d], k and v [T, g, d] in 64 bits."""
    T, h = q.shape[:2]
    at = torch.arange(T, device=q.device)
    back = at[:, None] - at[None, :]
    hidden = (back < 0) | (back >= window) if window else back < 0
    out = torch.empty_like(q)
    for i in range(h):
        j = i // (h // k.shape[1])
        sc = _cap(q[:, i] @ k[:, j].T * scale, cap).masked_fill(hidden, -math.inf)
        out[:, i] = torch.softmax(sc, -1) @ v[:, j]
    return out


def _rms(x, w):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS) * w


def _model_exact(case, seed, s):
    """Every sequence's prompt and given tokens as one causal pass; logits at the places that the steps return."""
    from trapetum_b200.engine.model import tensor_specs_for_config
    from trapetum_b200.weights.loader import random_tensors
    cfg = _config()
    specs = tensor_specs_for_config(cfg)

    def weight(name):                                                    # the seed's weights, one tensor at a time
        return dict(random_tensors({name: specs[name]}, seed, 0.02, 0.1, device=DEV))[name].double()

    h, g, d, hidden = SHAPES["2b"][:4]
    seqs = [p + [t[b] for t in s["tokens"]] for b, p in enumerate(s["prompts"])]
    lens = [len(q) for q in seqs]
    ids = torch.tensor([t for q in seqs for t in q], device=DEV)
    table = weight("model.embed_tokens.weight")
    x = table[ids] * math.sqrt(hidden)
    ang = torch.cat([torch.arange(n, device=DEV) for n in lens]).double()[:, None] \
        * 10000.0 ** (-torch.arange(0, d, 2, device=DEV).double() / d)
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]

    def turn(u):
        a, b = u[..., :d // 2], u[..., d // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    for i in range(cfg["num_hidden_layers"]):
        def w(name):
            return weight(f"model.layers.{i}.{name}.weight")
        y = _rms(x, 1.0 + w("input_layernorm"))
        q, k, v = (y @ w(f"self_attn.{n}_proj").T for n in "qkv")
        q, k, v = turn(q.view(-1, h, d)), turn(k.view(-1, g, d)), v.view(-1, g, d)
        parts = [_attention(a, b, c, 256 ** -0.5, 50.0, 4096 if i % 2 == 0 else 0)
                 for a, b, c in zip(q.split(lens), k.split(lens), v.split(lens))]
        x = x + _rms(torch.cat(parts).reshape(-1, h * d) @ w("self_attn.o_proj").T, 1.0 + w("post_attention_layernorm"))
        y = _rms(x, 1.0 + w("pre_feedforward_layernorm"))
        y = (_gelu_tanh(y @ w("mlp.gate_proj").T) * (y @ w("mlp.up_proj").T)) @ w("mlp.down_proj").T
        x = x + _rms(y, 1.0 + w("post_feedforward_layernorm"))
    x = _rms(x, 1.0 + weight("model.norm.weight"))
    first = [sum(lens[:b]) + len(p) - 1 for b, p in enumerate(s["prompts"])]
    return [_cap(x[torch.tensor([f + i for f in first], device=DEV)] @ table.T, 30.0) for i in range(case["steps"] + 1)]


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "model":
        del s["engine"]
        return _model_exact(case, seed, s)
    if kind == "attn_decode":
        h, g, d = SHAPES[case["shape"]][:3]
        out = []
        for b, n in enumerate(_ints(case)):
            pages = s["table"][b, :(n + PAGE - 1) // PAGE].long()
            k, v = (s[x][pages].transpose(0, 1).reshape(g, -1, d)[:, :n].double() for x in "kv")
            q = s["q"][b].double().view(g, h // g, d)
            p = torch.softmax(_cap(q @ k.transpose(1, 2) * d ** -0.5, case["cap"]), -1)
            out.append((p @ v).reshape(-1))
        return torch.stack(out)
    if kind == "attn_prompt":
        h, g, d = SHAPES[case["shape"]][:3]
        lens = _ints(case)
        q, k, v = (s[x].double().reshape(-1, n, d).split(lens) for x, n in (("q", h), ("k", g), ("v", g)))
        return torch.cat([_attention(a, b, c, d ** -0.5, case["cap"], case["window"]).reshape(-1, h * d) for a, b, c in zip(q, k, v)])
    if kind == "mlp":
        hidden, ff = SHAPES[case["shape"]][3:]
        x, gu = s["x"].double(), s["gate_up"]
        gate, up = (gu.view(-1, 2, 16, hidden)[:, i].reshape(ff, hidden) for i in (0, 1)) if case["dtype"] == "bfloat16" else (gu[:ff], gu[ff:])
        return (_gelu_tanh(x @ gate.double().T) * (x @ up.double().T)) @ s["down"].double().T
    if kind == "head":
        logits = torch.cat([_cap(s["x"].double() @ w.double().T, 30.0) for w in s["w"].split(32768)], -1)
        if s["recent"] is not None:
            at = torch.zeros_like(logits, dtype=torch.bool).scatter_(1, s["recent"].long(), True)
            pen = s["penalty"].double()[:, None]
            logits = torch.where(at, torch.where(logits > 0, logits / pen, logits * pen), logits)
        return {"logits": logits, "tokens": None}
    if kind == "mamba2":
        return _mamba2_exact(case, s)
    if kind == "gla":
        return _gla_exact(case, s)
    if kind == "latent":
        H, out = case["heads"], []
        for b, n in enumerate(s["host_lens"]):
            rows = s["pool"][s["table"][b, :(n + PAGE - 1) // PAGE].long()].reshape(-1, 512)[:n].double()
            sc = s["q"][b].double().view(H, 512) @ rows.T * 0.07
            p = torch.softmax(torch.cat([sc, s["sink"].double()[:, None]], -1), -1)[:, :n]
            out.append((p @ rows[:, :448]).reshape(-1))
        return torch.stack(out)
    if kind == "mixed":
        H, G, blk, out = case["heads"], case["kv_heads"], case["block"], []
        for a, b in zip(s["starts"], s["starts"][1:]):
            for t0 in range(a, b, blk):
                t1 = min(b, t0 + blk)
                q = s["q"][t0:t1].double().view(-1, H, 128).transpose(0, 1)
                k, v = (s[x][t0:t1].double().view(-1, G, 128).transpose(0, 1).repeat_interleave(H // G, 0) for x in "kv")
                sc = torch.einsum("hg,gij->hij", s["mix"].double(), q @ k.transpose(1, 2))
                n = t1 - t0
                sc = sc.masked_fill(torch.ones(n, n, device=DEV, dtype=torch.bool).triu(1), -math.inf)
                p = torch.softmax(torch.cat([sc, torch.zeros(H, n, 1, device=DEV, dtype=F64)], -1), -1)[..., :n]
                out.append((p @ v).transpose(0, 1).reshape(n, -1))
        return torch.cat(out)
    x = s["x"].double()
    p = torch.softmax(s["logits"][0].double(), -1)
    weight, idx = torch.topk(p, 4, dim=-1)
    weight = weight / weight.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(32):
        t, k = torch.nonzero(idx == e, as_tuple=True)
        if len(t):
            u = x[t] @ s["up"][e].double().T
            act = torch.nn.functional.silu(x[t] @ s["gate"][e].double().T) * u if case["gated"] else torch.relu(u) ** 2
            out.index_add_(0, t, weight[t, k][:, None] * (act @ s["down"][e].double().T))
    return {"out": out, "idx": idx, "weight": weight}


def _mamba2_exact(case, s):
    H, P, N = case["heads"], 64, case["state"]
    inner, ch = H * P, H * P + 2 * N
    proj = s["proj"].double()
    z, raw = proj[:, :inner], proj[:, inner:]
    dt = torch.nn.functional.softplus(s["dt"].double() + s["dt_bias"].double())
    decay = torch.exp(-torch.exp(s["A_log"].double()) * dt)
    y, states = [], []
    for a, b in zip(s["starts"], s["starts"][1:]):
        rows = torch.cat([torch.zeros(3, ch, device=DEV, dtype=F64), raw[a:b]])
        u = s["conv_b"].double() + sum(rows[j:j + b - a] * s["conv_w"][:, j].double() for j in range(4))
        u = torch.nn.functional.silu(u)
        x, B, C = u[:, :inner].view(-1, H, P), u[:, inner:inner + N], u[:, inner + N:]
        dx = dt[a:b, :, None] * x
        S = torch.zeros(H, P, N, device=DEV, dtype=F64)
        for t in range(b - a):
            S = decay[a + t, :, None, None] * S + dx[t, :, :, None] * B[t]
            y.append((S @ C[t] + s["D"].double()[:, None] * x[t]).reshape(-1))
        states.append(torch.cat([S.reshape(-1), rows[-3:].reshape(-1)]))
    return {"out": _rms(torch.stack(y) * torch.nn.functional.silu(z), s["norm"].double()), "state": torch.stack(states)}


def _gla_exact(case, s):
    H, D, V = case["heads"], 128, 256
    proj = s["proj"].double()
    q, k = proj[:, :H * D].view(-1, H, D) * D ** -0.5, proj[:, H * D:2 * H * D].view(-1, H, D)
    v, g = proj[:, 2 * H * D:2 * H * D + H * V].view(-1, H, V), proj[:, 2 * H * D + H * V:].view(-1, H, V)
    decay = torch.exp(torch.nn.functional.logsigmoid(s["low"][0].double() @ s["a2"].double().T + s["a2_bias"].double()) / 8.0).view(-1, H, D)
    y, states = [], []
    for a, b in zip(s["starts"], s["starts"][1:]):
        S = torch.zeros(H, D, V, device=DEV, dtype=F64)
        for t in range(a, b):
            S = decay[t, :, :, None] * S + k[t, :, :, None] * v[t, :, None, :]
            y.append((q[t, :, None, :] @ S)[:, 0])
        states.append(S.reshape(-1))
    out = _rms(torch.stack(y), s["norm"].double()) * torch.nn.functional.silu(g)
    return {"out": out.reshape(-1, H * V), "state": torch.stack(states)}
