"""The work that serving with this framework consists of, as measurable cases.

`listed()` holds one case per path that a request takes -- prompt attention, paged decode attention, the mixture of
experts, the recurrences of the hybrid decoders, a whole prompt step -- at sizes of the presets in
nanovllm/config.py and of bench.py; `draw()` gives further cases of the same ranges. `prepare()` makes what a
program has in hand before the call (inputs, caches, weights), `run()` is one pass through the public entry points,
`exact()` the same result in 64-bit torch, `work()` the bytes and operations that cannot be avoided and
`tolerance()` what another correct implementation at the same precision may differ by.
"""
from __future__ import annotations

import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nano-vllm-ascend_b200"))

from nanovllm import ops  # noqa: E402
from nanovllm.layers.seq_mixers import DeltaRule, LinearRecurrence, VarSizeAttention  # noqa: E402
from nanovllm.models.decoder import DecoderForCausalLM, DecoderSpec  # noqa: E402
from nanovllm.utils.context import set_context  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
F64 = torch.float64


def listed():
    return [
        # one user waiting for the next token: the smallest call of the service
        {"name": "decode_one", "kind": "decode", "seqs": 1, "lo": 1500, "hi": 1500, "heads": 16, "kv": 8, "dim": 128,
         "block": 16, "dtype": "bf16"},
        # a full decode batch of bench.py's serving workload (prompts of 100-1024 tokens, 100-1024 generated)
        {"name": "decode_batch", "kind": "decode", "seqs": 256, "lo": 100, "hi": 2048, "heads": 16, "kv": 8, "dim": 128,
         "block": 16, "dtype": "bf16"},
        # the same service with the e4m3 cache, a middling batch
        {"name": "decode_fp8", "kind": "decode_fp8", "seqs": 64, "lo": 100, "hi": 2048, "heads": 16, "kv": 8, "dim": 128,
         "block": 16, "dtype": "bf16"},
        # a prompt step of equal prompts: attention of one dense layer, K and V packed
        {"name": "prompt_attention", "kind": "prompt", "seqs": 16, "lo": 1024, "hi": 1024, "heads": 16, "kv": 8,
         "dim": 128, "dtype": "bf16", "softcap": 0.0, "sink": False},
        # ragged prompts through an attention layer with capped scores and a sink, heads of 64
        {"name": "prompt_capped_ragged", "kind": "prompt", "seqs": 12, "lo": 37, "hi": 1501, "heads": 32, "kv": 8,
         "dim": 64, "dtype": "bf16", "softcap": 30.0, "sink": True},
        # a prefix hit: few new tokens against a long cached prompt, fp16, heads of 64
        {"name": "prompt_prefix_hit", "kind": "prefix", "seqs": 1, "new": 256, "cached": 7936, "heads": 32, "kv": 8,
         "dim": 64, "block": 16, "dtype": "f16"},
        # a sparse mixture layer in a decode step (weight streaming) and in a prompt step (tensor-bound)
        {"name": "moe_decode", "kind": "moe", "tokens": 64, "width": 2048, "inter": 768, "experts": 128, "top": 8},
        {"name": "moe_prompt", "kind": "moe", "tokens": 4096, "width": 2048, "inter": 768, "experts": 128, "top": 8},
        # a selective recurrence of a hybrid decoder over a prompt step
        {"name": "recurrence_prompt", "kind": "recurrence", "seqs": 16, "lo": 1024, "hi": 1024, "heads": 32, "groups": 8,
         "kdim": 128, "vdim": 64, "mode": "selective"},
        # a gated delta rule (one decay per key channel) over ragged prompts: preparation and recurrence
        {"name": "delta_prompt", "kind": "delta", "seqs": 16, "lo": 500, "hi": 1300, "heads": 8, "groups": 4, "dim": 128,
         "per_head": False},
        # attention of a model served in 32 bits, prompt step over the paged cache
        {"name": "attention_f32", "kind": "attention_f32", "seqs": 4, "lo": 700, "hi": 1024, "heads": 8, "kv": 2,
         "dim": 128, "block": 16},
        # a whole prompt step of the dense decoder qwen3-0.6b, up to the logits
        {"name": "model_prompt", "kind": "model", "seqs": 6, "lo": 300, "hi": 1000, "layers": 28},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["decode", "decode", "decode_fp8", "prompt", "prompt", "prefix", "moe", "moe", "recurrence",
                       "delta", "attention_f32", "model"])
    heads, kv, dim = rng.choice([(16, 8, 128), (32, 8, 64), (8, 2, 128), (32, 4, 128), (8, 8, 64)])
    lo = log(16, 600)
    if kind in ("decode", "decode_fp8"):
        if kind == "decode_fp8":
            heads, kv, dim = rng.choice([(16, 8, 128), (32, 8, 64)])
        return {"kind": kind, "seqs": log(1, 256), "lo": lo, "hi": lo + log(16, 1400), "heads": heads, "kv": kv,
                "dim": dim, "block": rng.choice([16, 64, 256]), "dtype": rng.choice(["bf16", "f16"])}
    if kind == "prompt":
        capped = rng.random() < 0.4
        return {"kind": kind, "seqs": log(1, 16), "lo": lo, "hi": lo + log(16, 400), "heads": heads, "kv": kv, "dim": dim,
                "dtype": rng.choice(["bf16", "f16"]), "softcap": 30.0 if capped else 0.0, "sink": capped}
    if kind == "prefix":
        return {"kind": kind, "seqs": rng.randint(1, 4), "new": log(17, 512), "cached": log(64, 7000), "heads": heads,
                "kv": kv, "dim": dim, "block": rng.choice([16, 64]), "dtype": rng.choice(["bf16", "f16"])}
    if kind == "moe":
        width, inter, experts, top = rng.choice([(2048, 768, 128, 8), (1024, 512, 16, 2), (2048, 1024, 16, 2)])
        return {"kind": kind, "tokens": log(1, 4096), "width": width, "inter": inter, "experts": experts, "top": top}
    if kind == "recurrence":
        mode = rng.choice(["selective", "decay"])
        h, g, kd, vd = rng.choice([(32, 8, 128, 64), (64, 8, 128, 64)] if mode == "selective" else [(8, 8, 128, 128), (32, 32, 64, 64)])
        return {"kind": kind, "seqs": log(1, 8), "lo": lo, "hi": lo + log(16, 400), "heads": h, "groups": g, "kdim": kd,
                "vdim": vd, "mode": mode}
    if kind == "delta":
        h, dim = rng.choice([(8, 128), (32, 64)])
        return {"kind": kind, "seqs": log(1, 16), "lo": lo, "hi": lo + log(16, 700), "heads": h, "groups": h // 2,
                "dim": dim, "per_head": rng.random() < 0.5}
    if kind == "attention_f32":
        heads, kv, dim = rng.choice([(8, 2, 128), (32, 8, 64), (8, 8, 48)])
        return {"kind": kind, "seqs": rng.randint(1, 4), "lo": lo, "hi": lo + log(16, 400), "heads": heads, "kv": kv,
                "dim": dim, "block": rng.choice([16, 64])}
    return {"kind": kind, "seqs": log(1, 5), "lo": lo, "hi": lo + log(16, 400), "layers": 28}


# ------------------------------------------------------------------ sizes and inputs
def _lens(c):
    """The lengths of a case's sequences: spread over lo .. hi in an order that looks random, fixed by the case."""
    n, lo, hi = c["seqs"], c["lo"], c["hi"]
    return [lo + int((hi - lo) * ((0.37 + i * 0.6180339887498949) % 1.0)) for i in range(n)]


def _spans(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return cu


class _Random:
    """Normal tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def __call__(self, *shape, dtype=torch.float32, scale=1.0):
        x = torch.randn(*shape, device="cuda", dtype=dtype, generator=self.g)
        return x if scale == 1.0 else x.mul_(scale)

    def perm(self, n):
        return torch.randperm(n, device="cuda", generator=self.g)


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def _blocks(r, lens, block):
    """Block tables [seqs, most] over a pool in random order, and the pool's size."""
    need = [-(-n // block) for n in lens]
    pool = sum(need) + 3
    order = r.perm(pool).to(torch.int32)
    bt = torch.full((len(lens), max(need)), -1, dtype=torch.int32, device="cuda")
    at = 0
    for i, n in enumerate(need):
        bt[i, :n] = order[at:at + n]
        at += n
    return bt, pool


def _inputs(c, seed):
    """Everything that is random or laid out: used by prepare() and by exact()."""
    r, kind, s = _Random(seed), c["kind"], {}
    if kind in ("decode", "decode_fp8"):
        dt, lens, row = DTYPES[c["dtype"]], _lens(c), c["kv"] * c["dim"]
        s["tables"], pool = _blocks(r, lens, c["block"])
        s["lens"] = _i32(lens)
        s["q"] = r(c["seqs"], c["heads"], c["dim"], dtype=dt)
        s["k"], s["v"] = (r(pool, c["block"], row, dtype=dt) for _ in range(2))
        if kind == "decode_fp8":
            s["k"], s["v"] = (t.to(torch.float8_e4m3fn) for t in (s["k"], s["v"]))
    elif kind == "prompt":
        dt, lens = DTYPES[c["dtype"]], _lens(c)
        T, H, G, D = sum(lens), c["heads"], c["kv"], c["dim"]
        s["qkv"] = r(T, (H + 2 * G) * D, dtype=dt)             # as the projection leaves it
        s["cu"], s["most"] = _i32(_spans(lens)), max(lens)
        s["sink"] = torch.zeros(H, device="cuda") if c["sink"] else None
    elif kind == "prefix":
        dt, n = DTYPES[c["dtype"]], c["new"] + c["cached"]
        s["tables"], pool = _blocks(r, [n] * c["seqs"], c["block"])
        s["q"] = r(c["seqs"] * c["new"], c["heads"], c["dim"], dtype=dt)
        s["k"], s["v"] = (r(pool, c["block"], c["kv"] * c["dim"], dtype=dt) for _ in range(2))
        s["cu_q"], s["cu_k"] = _i32(_spans([c["new"]] * c["seqs"])), _i32(_spans([n] * c["seqs"]))
    elif kind == "moe":
        E, W, I, bf = c["experts"], c["width"], c["inter"], torch.bfloat16
        s["x"] = r(c["tokens"], W, dtype=bf)
        s["router"] = r(c["tokens"], E, dtype=bf)
        s["w13"], s["w2"] = r(E, 2 * I, W, dtype=bf, scale=W ** -0.5), r(E, W, I, dtype=bf, scale=I ** -0.5)
    elif kind == "recurrence":
        lens, bf = _lens(c), torch.bfloat16
        T, H, G, N, V = sum(lens), c["heads"], c["groups"], c["kdim"], c["vdim"]
        s["cu"], s["most"] = _i32(_spans(lens)), max(lens)
        if c["mode"] == "selective":                           # x | B | C as the convolution leaves them, dt projected
            s["xbc"] = torch.nn.functional.silu(r(T, H * V + 2 * G * N, dtype=bf))
            s["dt"] = r(T, H, dtype=bf)
            s["dt_bias"], s["a_log"], s["d"] = r(H, scale=0.5), -2 * torch.rand(H, device="cuda", generator=r.g), torch.ones(H, device="cuda")
        else:                                                  # q | k | v | gate, one projection
            s["p"] = r(T, 2 * H * N + 2 * H * V, dtype=bf)
    elif kind == "delta":
        lens, bf = _lens(c), torch.bfloat16
        T, H, G, D = sum(lens), c["heads"], c["groups"], c["dim"]
        s["cu"], s["most"] = _i32(_spans(lens)), max(lens)
        s["qkv"] = r(T, (2 * G + H) * D, dtype=bf)
        s["a"], s["b"] = r(T, H * (1 if c["per_head"] else D), dtype=bf), r(T, H, dtype=bf)
        s["dt_bias"] = r(H * (1 if c["per_head"] else D))
        s["a_log"] = -1 - 2 * torch.rand(H, device="cuda", generator=r.g)
    elif kind == "attention_f32":
        lens, H, G, D = _lens(c), c["heads"], c["kv"], c["dim"]
        s["tables"], pool = _blocks(r, lens, c["block"])
        s["q"] = r(sum(lens), H, D)
        s["k"], s["v"] = (r(pool, c["block"], G * D) for _ in range(2))
        s["cu"], s["most"] = _i32(_spans(lens)), max(lens)
    elif kind == "model":
        lens = _lens(c)
        s["ids"] = torch.randint(0, SPEC["vocab_size"], (sum(lens),), device="cuda", generator=r.g)
        s["cu"], s["most"] = _i32(_spans(lens)), max(lens)
        s["positions"] = torch.cat([torch.arange(n, device="cuda") for n in lens])
        s["weights"] = r
    return s


# qwen3-0.6b of nanovllm/config.py
SPEC = dict(vocab_size=151936, hidden_size=1024, num_heads=16, num_kv_heads=8, head_dim=128, intermediate_size=3072,
            rms_eps=1e-6, rope_theta=1000000.0, max_position=4096, qkv_bias=False, o_bias=False, mlp_bias=False, qk_norm=True,
            tie_embeddings=True, shared_rope=True, explicit_scale=False)


def _fill(model, r):
    """Random weights of a trained model's size (norm weights near one), made from the seed in the modules' order."""
    with torch.no_grad():
        for name, p in model.named_parameters():
            if name == "lm_head.weight":
                continue                                       # tied to the embedding
            p.normal_(1.0 if p.dim() == 1 else 0.0, 0.1 if p.dim() == 1 else p.shape[1] ** -0.5, generator=r.g)


def prepare(case, seed):
    c, s = case, _inputs(case, seed)
    kind, s["case"] = c["kind"], case
    if kind == "recurrence":
        H, V, N = c["heads"], c["vdim"], c["kdim"]
        decay = None if c["mode"] == "selective" else [1.0 - 2.0 ** (-3 - 5 * i / max(1, H - 1)) for i in range(H)]
        m = LinearRecurrence(H, c["groups"], N, V, decay=decay, act_silu=decay is not None).cuda().requires_grad_(False)
        if decay is None:
            for p, x in ((m.dt_bias, s["dt_bias"]), (m.A_log, s["a_log"]), (m.D, s["d"])):
                p.copy_(x)
        m.state = torch.zeros(c["seqs"], H, N, V, device="cuda")
        s["layer"], s["slots"] = m, _i32(list(range(c["seqs"])))
    elif kind == "delta":
        m = DeltaRule(c["heads"], c["groups"], c["dim"], c["dim"], per_head=c["per_head"]).cuda().requires_grad_(False)
        m.dt_bias.copy_(s["dt_bias"])
        m.A_log.copy_(s["a_log"])
        m.state = torch.zeros(c["seqs"], c["heads"], c["dim"], c["dim"], device="cuda")
        s["layer"], s["slots"] = m, _i32(list(range(c["seqs"])))
    elif kind == "attention_f32":
        m = VarSizeAttention(c["heads"], c["kv"], c["dim"], c["dim"], c["dim"] ** -0.5)
        m.k_cache, m.v_cache = s["k"], s["v"]
        s["layer"] = m
    elif kind == "model":
        old = torch.get_default_dtype()
        torch.set_default_dtype(torch.bfloat16)
        try:
            with torch.device("cuda"):
                m = DecoderForCausalLM(DecoderSpec(num_layers=c["layers"], **SPEC)).requires_grad_(False)
        finally:
            torch.set_default_dtype(old)
        _fill(m, s.pop("weights"))
        lens = _lens(c)
        s["tables"], pool = _blocks(_Random(seed), lens, 16)
        kv = torch.zeros(2, c["layers"], pool, 16, SPEC["num_kv_heads"] * SPEC["head_dim"], dtype=torch.bfloat16, device="cuda")
        for i, layer in enumerate(m.model.layers):
            layer.self_attn.attn.k_cache, layer.self_attn.attn.v_cache = kv[0, i], kv[1, i]
        s["slots"] = torch.cat([s["tables"][i].repeat_interleave(16)[:n] * 16 + torch.arange(n, device="cuda") % 16
                                for i, n in enumerate(lens)]).to(torch.int32)
        s["model"] = m
    return s


@torch.inference_mode()
def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "decode":
        return ops.paged_decode_attn(s["q"], s["k"], s["v"], s["tables"], s["lens"], c["dim"] ** -0.5, c["kv"])
    if kind == "decode_fp8":
        return ops.paged_decode_attn_fp8(s["q"], s["k"], s["v"], s["tables"], s["lens"], c["dim"] ** -0.5, c["kv"])
    if kind == "prompt":
        H, G, D = c["heads"], c["kv"], c["dim"]
        q, k, v = s["qkv"].split([H * D, G * D, G * D], dim=1)
        return ops.prefill_varlen_attn(q.unflatten(1, (H, D)), k.unflatten(1, (G, D)), v.unflatten(1, (G, D)), s["cu"],
                                       s["cu"], s["most"], s["most"], D ** -0.5, G, softcap=c["softcap"], sink=s["sink"])
    if kind == "prefix":
        return ops.prefill_varlen_attn(s["q"], s["k"], s["v"], s["cu_q"], s["cu_k"], c["new"], c["new"] + c["cached"],
                                       c["dim"] ** -0.5, c["kv"], block_tables=s["tables"])
    if kind == "moe":
        ids, weights = ops.moe_route(s["router"], c["top"])
        plan = ops.moe_align(ids, 0, c["experts"])
        return ops.moe_experts(s["x"], s["w13"], s["w2"], ids, weights, plan)
    if kind == "recurrence":
        set_context(True, s["cu"], s["cu"], s["most"], s["most"], state_slots=s["slots"])
        H, G, N, V = c["heads"], c["groups"], c["kdim"], c["vdim"]
        if c["mode"] == "selective":
            x, b, q = s["xbc"].split([H * V, G * N, G * N], dim=1)
            return s["layer"](q, b, x, dt=s["dt"]), s["layer"].state
        q, k, v, _ = s["p"].split([H * N, H * N, H * V, H * V], dim=1)
        return s["layer"](q, k, v), s["layer"].state
    if kind == "delta":
        set_context(True, s["cu"], s["cu"], s["most"], s["most"], state_slots=s["slots"])
        n = 2 * c["groups"] * c["dim"]
        return s["layer"](s["qkv"][:, :n], s["qkv"][:, n:], s["a"], s["b"]), s["layer"].state
    if kind == "attention_f32":
        set_context(True, s["cu"], s["cu"], s["most"], s["most"], block_tables=s["tables"], block_size=c["block"])
        return s["layer"](s["q"], None, None)
    set_context(True, s["cu"], s["cu"], s["most"], s["most"], slot_mapping=s["slots"], block_tables=s["tables"], block_size=16)
    return s["model"].compute_logits(s["model"](s["ids"], s["positions"]))


# ------------------------------------------------------------------ what cannot be avoided
def work(case):
    c = case
    kind = c["kind"]
    if kind in ("decode", "decode_fp8"):
        keys, size = sum(_lens(c)), 1 if kind == "decode_fp8" else 2
        return {"bytes": keys * 2 * c["kv"] * c["dim"] * size + 4 * c["seqs"] * c["heads"] * c["dim"],
                "flops": 4 * keys * c["heads"] * c["dim"]}
    if kind in ("prompt", "attention_f32"):
        lens, size = _lens(c), 4 if kind == "attention_f32" else 2
        return {"bytes": sum(lens) * 2 * (c["heads"] + c["kv"]) * c["dim"] * size,
                "flops": 4 * c["heads"] * c["dim"] * sum(n * (n + 1) // 2 for n in lens)}
    if kind == "prefix":
        n, m = c["new"], c["cached"]
        return {"bytes": c["seqs"] * 4 * (n * c["heads"] + (n + m) * c["kv"]) * c["dim"],
                "flops": 4 * c["seqs"] * c["heads"] * c["dim"] * (n * m + n * (n + 1) // 2)}
    if kind == "moe":
        hit = c["experts"] * (1 - (1 - c["top"] / c["experts"]) ** c["tokens"])
        return {"bytes": hit * 6 * c["width"] * c["inter"] + c["tokens"] * (4 * c["width"] + 2 * c["experts"]),
                "flops": 6 * c["tokens"] * c["top"] * c["width"] * c["inter"]}
    if kind == "recurrence":
        T, H, N, V = sum(_lens(c)), c["heads"], c["kdim"], c["vdim"]
        return {"bytes": T * (4 * c["groups"] * N + 6 * H * V) + 4 * c["seqs"] * H * N * V, "flops": 4 * T * H * N * V}
    if kind == "delta":
        T, H, D = sum(_lens(c)), c["heads"], c["dim"]
        return {"bytes": T * (4 * c["groups"] * D + 6 * H * D + 2 * H * (1 if c["per_head"] else D)) + 4 * c["seqs"] * H * D * D,
                "flops": 8 * T * H * D * D}
    lens = _lens(c)
    per_layer = 1024 * (4096 + 2048 + 3 * 3072)
    return {"bytes": 2 * (c["layers"] * (per_layer + sum(lens) * 2048) + 151936 * (1024 + len(lens))),
            "flops": 2 * c["layers"] * (sum(lens) * per_layer + 2 * 16 * 128 * sum(n * (n + 1) // 2 for n in lens))
            + 2 * len(lens) * 151936 * 1024}


def tolerance(case):
    """Against the 64-bit result the present code is off by (relative 2-norm): 32-bit paths 2e-7 to 4e-7, attention with
    bf16 inputs 2e-3 and with fp16 inputs 3e-4, the mixture 6e-3, the logits of the whole decoder 2e-2."""
    kind = case["kind"]
    if kind in ("recurrence", "delta", "attention_f32"):
        return {"rel": 5e-6}
    if kind == "model":                      # 16-bit roundings of 28 layers, each of which moves all that follow
        return {"rel": 3e-2}
    return {"rel": 1.5e-3 if case.get("dtype") == "f16" else 1e-2}


# ------------------------------------------------------------------ 64-bit results
def _attend(q, k, v, rep, scale, softcap=0.0, sink=None):
    """q [n, H, D] (the last n positions), k, v [m, G, D] -> [n, H * D], causal."""
    n, m = q.shape[0], k.shape[0]
    q, k, v = q.to(F64).transpose(0, 1), k.to(F64).transpose(0, 1), v.to(F64).transpose(0, 1)
    hidden = torch.arange(m, device="cuda")[None, :] > torch.arange(m - n, m, device="cuda")[:, None]
    out = []
    for g in range(k.shape[0]):
        s = torch.matmul(q[g * rep:(g + 1) * rep], k[g].T) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[g * rep:(g + 1) * rep].to(F64)[:, None, None].expand(-1, n, 1)], 2)
        out.append(torch.matmul(torch.softmax(s, -1)[..., :m], v[g]))
    return torch.cat(out).transpose(0, 1).reshape(n, -1)


def _rows(cache, table, n, G, D):
    b = cache.shape[1]
    return cache[table[:-(-n // b)].long()].reshape(-1, G, D)[:n]


def _recur(lens, T, H, N, V, step):
    """Runs step(t, rows, S) -> (S, o) over all sequences at once, longest first: o [T, H * V], S [seqs, H, N, V]."""
    cu = torch.tensor(_spans(lens), device="cuda")
    o = torch.empty(T, H, V, dtype=F64, device="cuda")
    S = torch.zeros(len(lens), H, N, V, dtype=F64, device="cuda")
    order = sorted(range(len(lens)), key=lambda i: -lens[i])
    idx, sizes = torch.tensor(order, device="cuda"), [lens[i] for i in order]
    S_sorted = S[idx]
    live = len(lens)
    for t in range(sizes[0]):
        while sizes[live - 1] <= t:
            live -= 1
        rows = cu[idx[:live]] + t
        S_sorted[:live], o[rows] = step(rows, S_sorted[:live])
    S[idx] = S_sorted
    return o.reshape(T, H * V), S


def exact(case, seed):
    c, s = case, _inputs(case, seed)
    kind = c["kind"]
    if kind in ("decode", "decode_fp8"):
        G, D = c["kv"], c["dim"]
        return torch.cat([_attend(s["q"][i:i + 1], _rows(s["k"], s["tables"][i], n, G, D), _rows(s["v"], s["tables"][i], n, G, D),
                                  c["heads"] // G, D ** -0.5) for i, n in enumerate(_lens(c))])
    if kind in ("prompt", "attention_f32"):
        H, G, D, lens, out, at = c["heads"], c["kv"], c["dim"], _lens(c), [], 0
        for i, n in enumerate(lens):
            if kind == "prompt":
                q, k, v = s["qkv"][at:at + n].split([H * D, G * D, G * D], dim=1)
                q, k, v = q.unflatten(1, (H, D)), k.unflatten(1, (G, D)), v.unflatten(1, (G, D))
            else:
                q, k, v = s["q"][at:at + n], _rows(s["k"], s["tables"][i], n, G, D), _rows(s["v"], s["tables"][i], n, G, D)
            out.append(_attend(q, k, v, H // G, D ** -0.5, c.get("softcap", 0.0), s.get("sink")))
            at += n
        return torch.cat(out)
    if kind == "prefix":
        G, D, n, m = c["kv"], c["dim"], c["new"], c["new"] + c["cached"]
        return torch.cat([_attend(s["q"][i * n:(i + 1) * n], _rows(s["k"], s["tables"][i], m, G, D),
                                  _rows(s["v"], s["tables"][i], m, G, D), c["heads"] // G, D ** -0.5) for i in range(c["seqs"])])
    if kind == "moe":
        p = torch.softmax(s["router"].to(F64), -1)
        w, ids = torch.sort(p, dim=-1, descending=True, stable=True)
        w, ids = w[:, :c["top"]], ids[:, :c["top"]]
        w = w / w.sum(-1, keepdim=True)
        out, I = torch.zeros(c["tokens"], c["width"], dtype=F64, device="cuda"), c["inter"]
        for e in range(c["experts"]):
            rows, j = (ids == e).nonzero(as_tuple=True)
            if rows.numel():
                h = s["x"][rows].to(F64) @ s["w13"][e].to(F64).T
                y = (torch.nn.functional.silu(h[:, :I]) * h[:, I:]) @ s["w2"][e].to(F64).T
                out.index_add_(0, rows, y * w[rows, j, None])
        return out
    if kind == "recurrence":
        H, G, N, V, lens = c["heads"], c["groups"], c["kdim"], c["vdim"], _lens(c)
        T = sum(lens)
        if c["mode"] == "selective":
            x, k, q = (t.to(F64) for t in s["xbc"].split([H * V, G * N, G * N], dim=1))
            step = torch.nn.functional.softplus(s["dt"].to(F64) + s["dt_bias"].to(F64))
            a, d = torch.exp(-torch.exp(s["a_log"].to(F64)) * step), s["d"].to(F64)
        else:
            q, k, x, _ = (torch.nn.functional.silu(t.float()).to(torch.bfloat16).to(F64) for t in s["p"].split([H * N, H * N, H * V, H * V], dim=1))
            decay = torch.tensor([1.0 - 2.0 ** (-3 - 5 * i / max(1, H - 1)) for i in range(H)], device="cuda", dtype=torch.float32)
            step, a, d = torch.ones(T, H, dtype=F64, device="cuda"), decay.to(F64).expand(T, H), torch.zeros(H, dtype=F64, device="cuda")
        q, k, x = q.view(T, G, N).repeat_interleave(H // G, 1), k.view(T, G, N).repeat_interleave(H // G, 1), x.view(T, H, V)

        def token(rows, S):
            S = a[rows][..., None, None] * S + k[rows][..., None] * (step[rows][..., None] * x[rows])[:, :, None, :]
            return S, torch.matmul(q[rows][:, :, None, :], S).squeeze(2) + d[:, None] * x[rows]
        return _recur(lens, T, H, N, V, token)
    if kind == "delta":
        H, G, D, lens = c["heads"], c["groups"], c["dim"], _lens(c)
        T = sum(lens)
        q, k, v = (t.to(F64) for t in s["qkv"].split([G * D, G * D, H * D], dim=1))
        q, k = ((t.view(T, G, D) / torch.sqrt((t.view(T, G, D) ** 2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1) for t in (q, k))
        q, v, beta = q * D ** -0.5, v.view(T, H, D), torch.sigmoid(s["b"].to(F64))
        soft = torch.nn.functional.softplus(s["a"].to(F64) + s["dt_bias"].to(F64)).view(T, H, -1)
        g = torch.exp(-torch.exp(s["a_log"].to(F64))[:, None] * soft)

        def token(rows, S):
            S = g[rows][..., None] * S
            w = beta[rows][..., None] * (v[rows] - torch.matmul(k[rows][:, :, None, :], S).squeeze(2))
            S = S + k[rows][..., None] * w[:, :, None, :]
            return S, torch.matmul(q[rows][:, :, None, :], S).squeeze(2)
        return _recur(lens, T, H, D, D, token)
    return _exact_model(c, s)


def _exact_model(c, s):
    """The decoder in 64 bits, weights drawn as prepare() draws them, one layer's at a time."""
    W, H, G, D, F, eps, r = 1024, 16, 8, 128, 3072, SPEC["rms_eps"], s["weights"]

    def matrix(n, m):
        return torch.empty(n, m, dtype=torch.bfloat16, device="cuda").normal_(0.0, m ** -0.5, generator=r.g).to(F64)

    def vector(n):
        return torch.empty(n, dtype=torch.bfloat16, device="cuda").normal_(1.0, 0.1, generator=r.g).to(F64)

    def norm(x, w):
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w

    embed = torch.empty(SPEC["vocab_size"], W, dtype=torch.bfloat16, device="cuda").normal_(0.0, W ** -0.5, generator=r.g)
    x = embed[s["ids"]].to(F64)
    angle = s["positions"].to(F64)[:, None] / SPEC["rope_theta"] ** (torch.arange(0, D, 2, device="cuda", dtype=F64) / D)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def rotate(t):
        a, b = t[..., :D // 2], t[..., D // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    lens = _lens(c)
    for _ in range(c["layers"]):
        wqkv, wo = matrix((H + 2 * G) * D, W), matrix(W, H * D)
        qn, kn = vector(D), vector(D)
        gate_up, down = matrix(2 * F, W), matrix(W, F)
        n1, n2 = vector(W), vector(W)
        q, k, v = (norm(x, n1) @ wqkv.T).split([H * D, G * D, G * D], dim=1)
        q, k = rotate(norm(q.unflatten(1, (H, D)), qn)), rotate(norm(k.unflatten(1, (G, D)), kn))
        v, parts, at = v.unflatten(1, (G, D)), [], 0
        for n in lens:
            parts.append(_attend(q[at:at + n], k[at:at + n], v[at:at + n], H // G, D ** -0.5))
            at += n
        x = x + torch.cat(parts) @ wo.T
        a, b = (norm(x, n2) @ gate_up.T).split([F, F], dim=1)
        x = x + (torch.nn.functional.silu(a) * b) @ down.T
    last = s["cu"][1:].long() - 1
    return norm(x[last], vector(W)) @ embed.to(F64).T
