"""What the performance of this framework is measured on: requests through the public entry points of its model runtimes.

* `qwen`: the native engine on the FP8 hybrid decoder at the 27B shape's widths (hidden 5120, SwiGLU 17408, 40 / 8 heads, 16 / 32
  DeltaNet heads), one period of its layers (three DeltaNet, one attention), loaded from a checkpoint: prompts, greedy decoding
  behind a short or a long context, rows of a speculative verification.
* `minimax`: MiniMax-M2 on raw GGUF blocks at the full widths (hidden 3072, 256 experts, IQ2_XXS experts, Q5_K attention), four
  layers: prompts and single-token decoding.
* `zemozen`: a mixer decoder of windowed attention, a state-space recurrence and routed experts at the "4k" size of its
  benchmark, four layers, under the batch step function: prompts and batches of requests.

Every model has fewer layers than it has in use, and a smaller vocabulary so that the output matrix keeps its share. The weights
are random, with two traits of trained ones: the next token follows from the present one (so that a greedy pick does not hang on
the last bit) and a token's experts stand out (so that a choice does not either).
"""
from __future__ import annotations

import json
import math
import os
import tempfile
from functools import lru_cache

import numpy as np
import torch

F64 = torch.float64
QWEN_VOCAB, MINIMAX_VOCAB, ZEMOZEN_VOCAB = 16384, 32768, 32000
QWEN_LAYERS = MINIMAX_LAYERS = 4
ROUTER_GAIN, ROUTER_SIGNAL = 0.3, 8.0


def listed() -> list[dict]:
    q, m, z = {"model": "qwen", "kv": "bf16"}, {"model": "minimax"}, {"model": "zemozen"}
    return [
        # a short question: latency and the number of launches count
        {"name": "qwen_prompt_13", "op": "prompt", "tokens": 13, **q},
        # the benchmark's prompt: one chunk of the tensor-core path
        {"name": "qwen_prompt_512", "op": "prompt", "tokens": 512, **q},
        # a document: several chunks, the last one ragged, attention over what came before
        {"name": "qwen_prompt_3001", "op": "prompt", "tokens": 3001, **q},
        # an answer to one user, token by token: the weights stream once per token
        {"name": "qwen_decode_500", "op": "decode", "context": 500, "steps": 24, **q},
        # the same behind a long document with the smaller cache
        {"name": "qwen_decode_6000_fp8kv", "op": "decode", "context": 6000, "steps": 16, "model": "qwen", "kv": "fp8"},
        # a drafter's proposals checked in one pass
        {"name": "qwen_verify_5", "op": "verify", "context": 300, "rows": 5, **q},
        # a short question to the routed-expert model: fewer than four routes per expert
        {"name": "minimax_prompt_23", "op": "prompt", "tokens": 23, **m},
        # the benchmark's prompt: every expert has a few rows
        {"name": "minimax_prompt_256", "op": "prompt", "tokens": 256, **m},
        # a document
        {"name": "minimax_prompt_1500", "op": "prompt", "tokens": 1500, **m},
        # an answer to one user
        {"name": "minimax_decode_200", "op": "decode", "context": 200, "steps": 16, **m},
        # a document to the mixer decoder
        {"name": "zemozen_prompt_1900", "op": "prompt", "tokens": 1900, **z},
        # a server's work: eight requests of different lengths admitted together, then decoded together
        {"name": "zemozen_batch_8", "op": "batch", "requests": 8, "tokens": 21, "steps": 12, **z},
    ]


def _log(rng, a: int, b: int) -> int:
    return min(b, max(a, round(math.exp(rng.uniform(math.log(a), math.log(b + 1))))))


def draw(rng) -> dict:
    model, op = rng.choice([("qwen", "prompt"), ("qwen", "prompt"), ("qwen", "decode"), ("qwen", "verify"), ("minimax", "prompt"), ("minimax", "prompt"),
                            ("minimax", "decode"), ("zemozen", "prompt"), ("zemozen", "batch")])
    case = {"model": model, "op": op}
    if model == "qwen":
        case["kv"] = rng.choice(["bf16", "bf16", "fp8"])
    if op == "prompt":
        case["tokens"] = _log(rng, 9, {"qwen": 3001, "minimax": 1500, "zemozen": 1900}[model])
    elif op == "verify":
        case.update(context=_log(rng, 16, 3000), rows=rng.randint(2, 8))
    elif op == "decode":
        case.update(context=_log(rng, 16, 6000 if model == "qwen" else 1400), steps=rng.randint(8, 16))
    else:
        case.update(requests=rng.randint(1, 8), tokens=_log(rng, 5, 60), steps=rng.randint(6, 12))
    return case


def _tokens(seed: int, n: int, vocab: int) -> list[int]:
    return torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(seed)).tolist()


def _normal(name: str, *shape: int) -> torch.Tensor:
    """Standard normal values on the GPU, decided by the name alone."""
    seed = int.from_bytes(name.encode(), "little") % (2 ** 61 - 1)
    return torch.randn(*shape, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))


def _follower(vocab: int) -> torch.Tensor:
    """before[t]: the token that t follows."""
    return torch.randperm(vocab, generator=torch.Generator().manual_seed(5)).cuda()


def _embedding(name: str, vocab: int, width: int, experts: int, top: int) -> tuple[torch.Tensor, torch.Tensor]:
    """(embedding [vocab, width] of unit size, unit directions [experts, width]): a token's vector leans towards `top` directions."""
    u = _normal(name + ".directions", experts, width)
    u /= u.norm(dim=1, keepdim=True)
    e = _normal(name + ".embed", vocab, width)
    pick = torch.rand(vocab, experts, device="cuda", generator=torch.Generator("cuda").manual_seed(9)).topk(top, dim=1).indices
    e += ROUTER_SIGNAL * torch.zeros(vocab, experts, device="cuda").scatter_(1, pick, 1.0) @ u
    return e, u


def _router(u: torch.Tensor, layer: int) -> torch.Tensor:
    return ROUTER_GAIN * u.roll(37 * layer, 0)


# -- the hybrid decoder ------------------------------------------------------------------------------------------------------

def _qwen_config():
    from pocketllm_b200.models.qwen_hybrid import QwenHybridConfig
    return QwenHybridConfig(vocab_size=QWEN_VOCAB, num_hidden_layers=QWEN_LAYERS)


def _quantise(w: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """E4M3 codes and one bf16 scale per 128 x 128 block."""
    n, k = w.shape
    b = w.view(n // 128, 128, k // 128, 128)
    s = (b.abs().amax((1, 3)) / 448).to(torch.bfloat16)
    q = (b / s.float()[:, None, :, None]).clamp(-448, 448).view(n, k)
    return q.to(torch.float8_e4m3fn), s


def _qwen_plan(c) -> dict[str, tuple]:
    """Tensor name -> (shape, mean, standard deviation); linears in FP8 end in a name without `.weight`."""
    H, D, I = c.hidden_size, c.head_dim, c.intermediate_size
    kd, vd, nv = c.linear_num_key_heads * 128, c.linear_num_value_heads * 128, c.linear_num_value_heads
    p = "model.language_model."
    out = {p + "embed_tokens.weight": ((c.vocab_size, H), 0, 1), p + "norm.weight": ((H,), 0, 0.05)}
    for i, kind in enumerate(c.layer_types):
        q = f"{p}layers.{i}."
        out.update({q + "input_layernorm.weight": ((H,), 0, 0.05), q + "post_attention_layernorm.weight": ((H,), 0, 0.05)})
        if kind == "linear_attention":
            a = q + "linear_attn."
            out.update({a + "in_proj_qkv": ((2 * kd + vd, H), 0, 0.02), a + "in_proj_z": ((vd, H), 0, 0.02), a + "out_proj": ((H, vd), 0, 0.006),
                        a + "in_proj_a.weight": ((nv, H), 0, 0.02), a + "in_proj_b.weight": ((nv, H), 0, 0.02),
                        a + "conv1d.weight": ((2 * kd + vd, 1, 4), 0, 0.3), a + "A_log": ((nv,), 0, 0.5), a + "dt_bias": ((nv,), -2, 0.5),
                        a + "norm.weight": ((128,), 1, 0.05)})
        else:
            a = q + "self_attn."
            out.update({a + "q_proj": ((2 * c.num_attention_heads * D, H), 0, 0.02), a + "k_proj": ((c.num_key_value_heads * D, H), 0, 0.02),
                        a + "v_proj": ((c.num_key_value_heads * D, H), 0, 0.02), a + "o_proj": ((H, c.num_attention_heads * D), 0, 0.01),
                        a + "q_norm.weight": ((D,), 0, 0.05), a + "k_norm.weight": ((D,), 0, 0.05)})
        out.update({q + "mlp.gate_proj": ((I, H), 0, 0.02), q + "mlp.up_proj": ((I, H), 0, 0.02), q + "mlp.down_proj": ((H, I), 0, 0.002)})
    return out


def _is_fp8(name: str) -> bool:
    return name.endswith(("_proj", "_qkv", "_z"))


def _qwen_tensors(c):
    """(name, tensor) of the checkpoint, one by one."""
    for name, (shape, mean, std) in _qwen_plan(c).items():
        t = mean + std * _normal(name, *shape)
        if _is_fp8(name):
            q, s = _quantise(t)
            yield name + ".weight", q
            yield name + ".weight_scale_inv", s
        else:
            yield name, t.to(torch.bfloat16)
        if name.endswith("embed_tokens.weight"):
            yield "lm_head.weight", (0.02 * t[_follower(c.vocab_size)]).to(torch.bfloat16)


@lru_cache(maxsize=1)
def _qwen_checkpoint() -> str:
    """A folder with the checkpoint, written once per machine."""
    c = _qwen_config()
    path = os.path.join(tempfile.gettempdir(), f"pocketllm_cases_qwen_{c.num_hidden_layers}x{c.hidden_size}_{os.getuid()}")
    if os.path.exists(path):
        return path
    part = f"{path}.{os.getpid()}"
    os.makedirs(part)
    with open(os.path.join(part, "config.json"), "w") as f:
        f.write(c.to_json())
    names = {torch.float8_e4m3fn: "F8_E4M3", torch.bfloat16: "BF16"}
    header, data, at = {}, [], 0
    for name, t in _qwen_tensors(c):
        raw = t.contiguous().view(torch.uint8).reshape(-1).cpu().numpy()
        header[name] = {"dtype": names[t.dtype], "shape": list(t.shape), "data_offsets": [at, at + raw.size]}
        data.append(raw)
        at += raw.size
    head = json.dumps(header).encode()
    head += b" " * (-len(head) % 8)
    with open(os.path.join(part, "model.safetensors"), "wb") as f:
        f.write(len(head).to_bytes(8, "little") + head)
        for raw in data:
            raw.tofile(f)
    try:
        os.rename(part, path)
    except OSError:          # another process was first
        import shutil
        shutil.rmtree(part)
    return path


def _qwen_prompt(case: dict, seed: int) -> list[int]:
    n = case["tokens"] if case["op"] == "prompt" else case["context"] + case.get("rows", 0)
    return _tokens(seed, n, QWEN_VOCAB)


def _qwen_prepare(case: dict, seed: int) -> dict:
    from pocketllm_b200.models.qwen_hybrid import QwenEngine
    prompt = _qwen_prompt(case, seed)
    eng = QwenEngine(_qwen_config(), max_context=len(prompt) + case.get("steps", 0) + 16, kv_cache_dtype=case["kv"]).load(_qwen_checkpoint())
    state = {"case": case, "engine": eng, "prompt": prompt}
    if case["op"] != "prompt":
        eng.prefill(prompt[:case["context"]])
        state["snapshot"] = eng.snapshot()          # what a speculative loop or a prefix cache keeps; the KV rows stay in place
    return state


def _qwen_run(state: dict):
    case, eng = state["case"], state["engine"]
    if case["op"] == "prompt":
        eng.reset()
        return {"token": eng.prefill(state["prompt"]), "logits": eng.logits()}
    state["snapshot"].restore()
    if case["op"] == "decode":
        return {"tokens": torch.tensor(eng.decode(case["steps"])), "logits": eng.logits()}
    picks = eng.forward_rows(state["prompt"][case["context"]:])
    return {"tokens": torch.tensor(picks), "logits": [eng.logits(r) for r in range(case["rows"])]}


def _qwen_work(case: dict) -> dict:
    c = _qwen_config()
    H, D, Hq, Hk = c.hidden_size, c.head_dim, c.num_attention_heads, c.num_key_value_heads
    fp8 = sum(math.prod(s) for n, (s, _, _) in _qwen_plan(c).items() if _is_fp8(n))
    small = sum(math.prod(s) for n, (s, _, _) in _qwen_plan(c).items() if not _is_fp8(n) and "embed" not in n)
    head = c.vocab_size * H
    weights = fp8 + fp8 // 128 ** 2 * 2 + 2 * small + 2 * head
    kv_row = 2 * Hk * D * 2 if case["kv"] == "bf16" else 2 * Hk * (D + 8)
    n_full = sum(k == "full_attention" for k in c.layer_types)
    n_lin = len(c.layer_types) - n_full
    nv = c.linear_num_value_heads
    states = n_lin * 2 * 4 * nv * 128 * 128                     # each state in and out once per pass

    def tokens(n: int, before: int) -> float:
        """Operations of n tokens behind `before` others, without the output matrix."""
        seen = n * before + n * (n + 1) / 2
        return 2.0 * n * (fp8 + small) + n_full * 4.0 * Hq * D * seen + n_lin * n * nv * 6.0 * 128 * 128

    if case["op"] == "prompt":
        n = case["tokens"]
        return {"bytes": weights + n * (4 + 2 * H) + n_full * n * kv_row + states / 2 + 4 * c.vocab_size, "flops": tokens(n, 0) + 2.0 * head}
    if case["op"] == "verify":
        n, b = case["rows"], case["context"]
        return {"bytes": weights + n * 2 * H + n_full * (n + b) * kv_row + states + n * 4 * c.vocab_size, "flops": tokens(n, b) + 2.0 * n * head}
    n, b = case["steps"], case["context"]                       # a token has to be there before the next one can begin
    return {"bytes": n * (weights + 2 * H + n_full * (b + n / 2) * kv_row + states) + 4 * c.vocab_size, "flops": tokens(n, b) + 2.0 * n * head}


class _Qwen64:
    """The hybrid decoder in 64 bits, a portion of the sequence at a time."""

    def __init__(self):
        self.c = c = _qwen_config()
        self.w = {}
        scale = {}
        for name, t in _qwen_tensors(c):
            if name.endswith("_scale_inv"):
                scale[name[:-len("_scale_inv")]] = t
            else:
                self.w[name] = t
        self.scale, self.state, self.pos = scale, [{} for _ in c.layer_types], 0

    def linear(self, x, name):
        w = self.w[name + ".weight"]
        if name + ".weight" not in self.scale:
            return x @ w.to(F64).T
        n, k = w.shape
        w = w.to(torch.float32).to(F64).view(n // 128, 128, k // 128, 128) * self.scale[name + ".weight"].to(F64)[:, None, :, None]
        return x @ w.view(n, k).T

    def norm(self, x, name):
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + self.c.rms_norm_eps) * (1 + self.w[name].to(F64))

    def turn(self, x, pos):
        half = self.c.rotary_dim // 2
        a = pos[:, None, None] * self.c.rope_theta ** (-torch.arange(half, device="cuda", dtype=F64) / half)
        u, v = x[..., :half], x[..., half:2 * half]
        return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), x[..., 2 * half:]], -1)

    def attention(self, x, p, st, pos):
        c, T = self.c, x.shape[0]
        Hq, Hk, D = c.num_attention_heads, c.num_key_value_heads, c.head_dim
        q, gate = self.linear(x, p + "q_proj").view(T, Hq, 2 * D).chunk(2, -1)
        k, v = (self.linear(x, p + n).view(T, Hk, D) for n in ("k_proj", "v_proj"))
        q, k = self.turn(self.norm(q, p + "q_norm.weight"), pos), self.turn(self.norm(k, p + "k_norm.weight"), pos)
        st["k"] = k = torch.cat([st["k"], k]) if "k" in st else k
        st["v"] = v = torch.cat([st["v"], v]) if "v" in st else v
        hidden = torch.arange(len(k), device="cuda")[None] > pos[:, None]
        out = []
        for h in range(Hq):
            s = (q[:, h] @ k[:, h * Hk // Hq].T * D ** -0.5).masked_fill_(hidden, -math.inf)
            out.append(torch.softmax(s, -1) @ v[:, h * Hk // Hq])
        return self.linear((torch.stack(out, 1) * torch.sigmoid(gate)).view(T, -1), p + "o_proj")

    def delta(self, x, p, st):
        c, T, w = self.c, x.shape[0], self.w
        nk, nv = c.linear_num_key_heads, c.linear_num_value_heads
        y, z = self.linear(x, p + "in_proj_qkv"), self.linear(x, p + "in_proj_z").view(T, nv, 128)
        a, b = self.linear(x, p + "in_proj_a"), self.linear(x, p + "in_proj_b")
        y = torch.cat([st.get("tail", torch.zeros(3, y.shape[1], device="cuda", dtype=F64)), y])
        st["tail"] = y[-3:]
        taps = w[p + "conv1d.weight"].to(F64)[:, 0]
        y = torch.nn.functional.silu(sum(y[j:j + T] * taps[:, j] for j in range(4)))
        q, k, v = y[:, :nk * 128].view(T, nk, 128), y[:, nk * 128:2 * nk * 128].view(T, nk, 128), y[:, 2 * nk * 128:].view(T, nv, 128)
        q, k = (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = (t.repeat_interleave(nv // nk, 1) for t in (q * 128 ** -0.5, k))
        decay = torch.exp(-torch.exp(w[p + "A_log"].to(F64)) * torch.nn.functional.softplus(a + w[p + "dt_bias"].to(F64)))
        beta = torch.sigmoid(b)
        S, out = st.get("S", torch.zeros(nv, 128, 128, device="cuda", dtype=F64)), torch.empty_like(v)
        for t in range(T):
            S = S * decay[t, :, None, None]
            d = (v[t] - (k[t, :, None] @ S)[:, 0]) * beta[t, :, None]
            S = torch.baddbmm(S, k[t, :, :, None], d[:, None])
            out[t] = (q[t, :, None] @ S)[:, 0]
        st["S"] = S
        out = out * torch.rsqrt((out * out).mean(-1, keepdim=True) + c.rms_norm_eps) * w[p + "norm.weight"].to(F64)
        return self.linear((out * torch.nn.functional.silu(z)).view(T, -1), p + "out_proj")

    def __call__(self, tokens, want) -> torch.Tensor:
        """Logits of the wanted places of the next tokens."""
        p = "model.language_model."
        pos = torch.arange(self.pos, self.pos + len(tokens), device="cuda")
        self.pos += len(tokens)
        x = self.w[p + "embed_tokens.weight"][torch.tensor(tokens, device="cuda")].to(F64)
        for i, (kind, st) in enumerate(zip(self.c.layer_types, self.state)):
            q = f"{p}layers.{i}."
            h = self.norm(x, q + "input_layernorm.weight")
            x = x + (self.delta(h, q + "linear_attn.", st) if kind == "linear_attention" else self.attention(h, q + "self_attn.", st, pos))
            h = self.norm(x, q + "post_attention_layernorm.weight")
            x = x + self.linear(torch.nn.functional.silu(self.linear(h, q + "mlp.gate_proj")) * self.linear(h, q + "mlp.up_proj"), q + "mlp.down_proj")
        return self.linear(self.norm(x[want], p + "norm.weight"), "lm_head")


def _qwen_exact(case: dict, seed: int):
    model, prompt = _Qwen64(), _qwen_prompt(case, seed)
    if case["op"] == "prompt":
        z = model(prompt, [-1])[0]
        return {"token": int(z.argmax()), "logits": z}
    z = model(prompt[:case["context"]], [-1])
    if case["op"] == "verify":
        z = model(prompt[case["context"]:], list(range(case["rows"])))
        return {"tokens": z.argmax(-1), "logits": list(z)}
    picks = []
    for _ in range(case["steps"]):
        z = model([int(z[0].argmax())], [0])
        picks.append(int(z[0].argmax()))
    return {"tokens": torch.tensor(picks), "logits": z[0]}


# -- routed experts on GGUF blocks -------------------------------------------------------------------------------------------

def _minimax_config():
    from pocketllm_b200.models.minimax_m2 import MiniMaxM2Config
    return MiniMaxM2Config(vocab_size=MINIMAX_VOCAB, n_layers=MINIMAX_LAYERS)


def _half(x: float) -> torch.Tensor:
    return torch.from_numpy(np.frombuffer(np.float16(x).tobytes(), np.uint8).copy()).cuda()


def _centre(raw: torch.Tensor, kind: str, d: float) -> None:
    """Random Q4_K / Q5_K blocks with minima that put the middle of the codes on zero: w = d * scale * (code - middle)."""
    v = raw.view(-1, {"q4_k": 144, "q5_k": 176}[kind])
    v[:, 0:2], v[:, 2:4] = _half(d), _half(d * {"q4_k": 7.5, "q5_k": 15.5}[kind])
    v[:, 8:12] = v[:, 4:8]
    v[:, 12:16] = (v[:, 12:16] & 15) * 17


def _q4_k(x: torch.Tensor, d: float, scale: int) -> torch.Tensor:
    """x [N, K] as Q4_K blocks with one scale for all."""
    b = torch.zeros(x.numel() // 256, 144, dtype=torch.uint8, device="cuda")
    b[:, 0:2], b[:, 2:4] = _half(d), _half(7.5 * d)
    b[:, 4:12] = scale & 63 | (scale >> 4) << 6
    b[:, 12:16] = (scale & 15) * 17
    q = (x / (d * scale) + 7.5).round().clamp(0, 15).to(torch.uint8).view(-1, 4, 2, 32)
    b[:, 16:] = (q[:, :, 0] | q[:, :, 1] << 4).view(-1, 128)
    return b.view(x.shape[0], -1)


def _minimax_model(max_context: int):
    from pocketllm_b200.models.minimax_m2 import MiniMaxM2Model
    c = _minimax_config()
    model = MiniMaxM2Model.synthetic(c, max_context=max_context, seed=3)
    e, u = _embedding("minimax", c.vocab_size, c.dim, c.n_experts, c.n_experts_used)
    rows = _q4_k(e, 2.0 ** -7, 60)
    model.embed.copy_(rows.view(-1))
    model.head.copy_(rows[_follower(c.vocab_size)].reshape(-1))
    for i, L in enumerate(model.layers):
        _centre(L["qkv"], "q5_k", 2.0 ** -14)
        _centre(L["o"], "q5_k", 2.0 ** -16)
        L["w2"].view(-1, 66)[:, :2] = _half(2.0 ** -12)
        L["router"].copy_(_router(u, i))
    return model


def _minimax_prompt(case: dict, seed: int) -> list[int]:
    return _tokens(seed, case["tokens"] if case["op"] == "prompt" else case["context"] + case["steps"] + 1, MINIMAX_VOCAB)


def _minimax_prepare(case: dict, seed: int) -> dict:
    prompt = _minimax_prompt(case, seed)
    state = {"case": case, "model": _minimax_model(len(prompt) + 8), "prompt": prompt}
    if case["op"] == "decode":
        state["model"].forward_logits(prompt[:case["context"]])
    return state


def _minimax_run(state: dict):
    case, model, prompt = state["case"], state["model"], state["prompt"]
    if case["op"] == "prompt":
        model.reset()
        return model.forward_logits(prompt)
    model.pos = case["context"]                  # the cache is indexed by position: go on behind the context
    picks = [model.decode_one(t) for t in prompt[case["context"]:-1]]
    return {"tokens": torch.tensor(picks), "logits": model.forward_logits(prompt[-1:])}


def _minimax_work(case: dict) -> dict:
    c = _minimax_config()
    qkv, o = (c.n_heads + 2 * c.n_kv_heads) * c.head_dim * c.dim, c.dim * c.n_heads * c.head_dim
    expert, per_256 = 3 * c.dim * c.expert_inter, {"q4_k": 144, "q5_k": 176, "iq2_xxs": 66}
    head = c.vocab_size * c.dim

    def layers(n: int, before: int) -> tuple[float, float]:
        """(bytes, operations) of n tokens in one pass behind `before` others."""
        used = c.n_experts * (1 - (1 - c.n_experts_used / c.n_experts) ** n)
        b = ((qkv + o) * 176 + used * expert * 66) / 256 + c.n_experts * c.dim * 4 + 4 * c.n_kv_heads * c.head_dim * (before + n)
        f = 2.0 * n * (qkv + o + c.n_experts * c.dim + c.n_experts_used * expert) + 4.0 * c.n_heads * c.head_dim * (n * before + n * (n + 1) / 2)
        return c.n_layers * b, c.n_layers * f

    passes = [(case["tokens"], 0)] if case["op"] == "prompt" else [(1, case["context"] + i) for i in range(case["steps"] + 1)]
    each = [layers(*p) for p in passes]
    embedded = sum(p[0] for p in passes) * c.dim * 144 / 256
    return {"bytes": embedded + sum(b for b, _ in each) + len(passes) * (head * 144 / 256 + 4 * c.vocab_size),
            "flops": sum(f for _, f in each) + 2.0 * head * len(passes)}


def _fp16(b: torch.Tensor) -> torch.Tensor:
    return b.contiguous().view(torch.float16).to(F64)


def _k_weights(raw: torch.Tensor, kind: str) -> torch.Tensor:
    """Q4_K / Q5_K blocks -> their 256 weights each."""
    b = raw.view(-1, {"q4_k": 144, "q5_k": 176}[kind])
    s = b[:, 4:16].to(torch.int32)
    sc = torch.cat([s[:, :4] & 63, s[:, 8:] & 15 | s[:, :4] >> 6 << 4], 1).to(F64)
    mn = torch.cat([s[:, 4:8] & 63, s[:, 8:] >> 4 | s[:, 4:8] >> 6 << 4], 1).to(F64)
    qs = b[:, -128:].view(-1, 4, 1, 32)
    q = torch.cat([qs & 15, qs >> 4], 2).view(-1, 8, 32).to(F64)
    if kind == "q5_k":
        q += 16 * (b[:, None, 16:48] >> torch.arange(8, device="cuda", dtype=torch.uint8)[:, None] & 1)
    return (_fp16(b[:, 0:2])[:, :, None] * sc[:, :, None] * q - _fp16(b[:, 2:4])[:, :, None] * mn[:, :, None]).view(-1, 256)


def _iq2_xxs_weights(raw: torch.Tensor) -> torch.Tensor:
    """IQ2_XXS blocks -> their 256 weights each; the table of magnitudes is the file format's."""
    from pocketllm_b200.formats.gguf_quants import codebook
    grid = torch.from_numpy(codebook("iq2_xxs").astype(np.float64)).cuda()
    b = raw.view(-1, 66)
    q = b[:, 2:].view(-1, 8, 8)
    aux = (q[..., 4:].to(torch.int64) << torch.tensor([0, 8, 16, 24], device="cuda")).sum(-1)
    bits = aux[..., None] >> torch.tensor([0, 7, 14, 21], device="cuda") & 127
    signs = bits[..., None] >> torch.arange(7, device="cuda") & 1
    signs = torch.cat([signs, signs.sum(-1, keepdim=True) & 1], -1)               # the eighth makes the number even
    w = grid[q[..., :4].long()] * (1 - 2 * signs) * (0.125 * _fp16(b[:, :2]) * (2 * (aux >> 28) + 1))[..., None, None]
    return w.view(-1, 256)


def _minimax_exact(case: dict, seed: int):
    prompt, c = _minimax_prompt(case, seed), _minimax_config()
    model = _minimax_model(8)          # its weights as they lie in memory
    T, D = len(prompt), c.head_dim
    rows = lambda raw, kind, k: (_iq2_xxs_weights(raw) if kind == "iq2_xxs" else _k_weights(raw, kind)).view(-1, k)
    norm = lambda x, g: x * torch.rsqrt((x * x).mean(-1, keepdim=True) + c.norm_eps) * g.to(F64)
    half = c.rope_dim // 2
    pos = torch.arange(T, device="cuda")
    angle = pos[:, None, None] * c.rope_theta ** (-torch.arange(half, device="cuda", dtype=F64) / half)

    def turn(x):
        u, v = x[..., :half], x[..., half:2 * half]
        return torch.cat([u * angle.cos() - v * angle.sin(), v * angle.cos() + u * angle.sin(), x[..., 2 * half:]], -1)

    x = rows(model.embed.view(c.vocab_size, -1)[torch.tensor(prompt, device="cuda")], "q4_k", c.dim)
    for L in model.layers:
        nq, nk = c.n_heads * D, c.n_kv_heads * D
        q, k, v = (norm(x, L["attn_norm"]) @ rows(L["qkv"], "q5_k", c.dim).T).split([nq, nk, nk], -1)
        q, k = turn(norm(q, L["q_norm"]).view(T, -1, D)), turn(norm(k, L["k_norm"]).view(T, -1, D))
        v, out = v.view(T, -1, D), []
        for h in range(c.n_heads):
            g = h * c.n_kv_heads // c.n_heads
            s = (q[:, h] @ k[:, g].T * D ** -0.5).masked_fill_(pos[None] > pos[:, None], -math.inf)
            out.append(torch.softmax(s, -1) @ v[:, g])
        x = x + torch.cat(out, 1) @ rows(L["o"], "q5_k", nq).T
        h = norm(x, L["ffn_norm"])
        p = torch.sigmoid(h @ L["router"].to(F64).T)
        ids = (p + L["bias"].to(F64)).topk(c.n_experts_used, -1).indices
        weight = p.gather(1, ids)
        weight = weight / weight.sum(-1, keepdim=True)
        y = torch.zeros_like(x)
        for e in ids.unique().tolist():
            t, j = (ids == e).nonzero(as_tuple=True)
            gate, up = (h[t] @ rows(L["w13"][e], "iq2_xxs", c.dim).T).chunk(2, -1)
            down = rows(L["w2"].view(c.n_experts, -1)[e], "iq2_xxs", c.expert_inter)
            y.index_add_(0, t, weight[t, j, None] * ((torch.nn.functional.silu(gate) * up) @ down.T))
        x = x + y
    last = [T - 1] if case["op"] == "prompt" else list(range(case["context"], T))
    z = norm(x[last], model.final_norm) @ rows(model.head, "q4_k", c.dim).T
    return z[0] if case["op"] == "prompt" else {"tokens": z[:-1].argmax(-1), "logits": z[-1]}


# -- a mixer decoder -----------------------------------------------------------------------------------------------------------

ZEMOZEN_WIDTH, ZEMOZEN_EXPERTS, ZEMOZEN_IDENTITIES, ZEMOZEN_TOP, ZEMOZEN_FF = 4096, 32, 4, 2, 2048
ZEMOZEN_PATTERN = ("parallel", "attention", "parallel", "attention")


def _zemozen_config():
    from pocketllm_b200.models.zemozen import ZemozenConfig
    att = {"heads": 32, "kv_heads": 8, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024}, "rot": {"base": 5e5, "dims": 128}}
    mix = {"attention": att | {"v_mix": True, "rot": att["rot"] | {"scaling": {"factor": 8.0}}},
           "parallel": {"left": att | {"softcap": 30.0}, "left_scale": 0.8, "right_scale": 0.9,
                        "right": {"heads": 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}}}
    mlp = {"kind": "moe", "expert": {"ff": ZEMOZEN_FF}, "router": {"experts": ZEMOZEN_EXPERTS, "identity": ZEMOZEN_IDENTITIES, "top": ZEMOZEN_TOP}}
    return ZemozenConfig.from_dict({"architecture": "Zemozen", "vocab": ZEMOZEN_VOCAB, "width": ZEMOZEN_WIDTH, "norm": {"eps": 1e-5}, "embedding": {"scale": 8.0},
                                    "residual_mult": 0.3, "layers": [{"type": t, "mixer": mix[t], "mlp": mlp} for t in ZEMOZEN_PATTERN]})


def _zemozen_tensors(c) -> dict[str, torch.Tensor]:
    from pocketllm_b200.models.zemozen import random_tensors
    t = random_tensors(c, 3, device="cuda")
    e, u = _embedding("zemozen", c.vocab, c.width, ZEMOZEN_EXPERTS + ZEMOZEN_IDENTITIES, ZEMOZEN_TOP)
    t["embed"] = (e / c.embed_scale).to(torch.bfloat16)
    t["head"] = (e[_follower(c.vocab)] * c.width ** -0.5).to(torch.bfloat16)
    for i in range(len(c.layers)):
        t[f"l{i}.mlp.router"] = _router(u, i).to(torch.bfloat16)
        t[f"l{i}.mlp.correction"] = t[f"l{i}.mlp.correction"] * 0.1
    return t


def _zemozen_prompts(case: dict, seed: int) -> list[list[int]]:
    """The tokens of every request: what it is admitted with, then one for every step."""
    if case["op"] == "prompt":
        return [_tokens(seed, case["tokens"], ZEMOZEN_VOCAB)]
    lengths = [max(1, case["tokens"] * (4 + i % 5) // 6) for i in range(case["requests"])]
    return [_tokens(seed * 100 + i, n + case["steps"], ZEMOZEN_VOCAB) for i, n in enumerate(lengths)]


def _zemozen_prepare(case: dict, seed: int) -> dict:
    from pocketllm_b200.models.zemozen import build_model
    from pocketllm_b200.runtime.mixer_runtime import MixerRuntime, StepEntry
    c, prompts = _zemozen_config(), _zemozen_prompts(case, seed)
    n, pages = len(prompts), sum(-(-len(p) // 64) for p in prompts) + 1
    rt = MixerRuntime(build_model(c, _zemozen_tensors(c), slots=n, pages=pages), max_requests=n, pages=pages)
    steps = case.get("steps", 0)
    first = [StepEntry(i, p[:len(p) - steps], (len(p) - steps - 1,)) for i, p in enumerate(prompts)]
    later = [[StepEntry(i, p[len(p) - steps + s:][:1], (0,)) for i, p in enumerate(prompts)] for s in range(steps)]
    return {"runtime": rt, "steps": [first] + later, "requests": n}


def _zemozen_run(state: dict):
    rt = state["runtime"]
    out = [rt.step(entries).clone() for entries in state["steps"]]       # a step's logits live until the next one
    for i in range(state["requests"]):
        rt.release(i)
    return out


def _zemozen_work(case: dict) -> dict:
    W, A, S = ZEMOZEN_WIDTH, 40 * 128, 4096                               # width, rows of q and k, inner size of the state space
    attention, space = (A + 1024 + 4096) * W, (2 * S + 2048 + 64 + S) * W
    n_par = ZEMOZEN_PATTERN.count("parallel")
    n_layers = len(ZEMOZEN_PATTERN)
    dense = n_layers * attention + n_par * space + n_layers * 36 * W + (n_layers - n_par) * 32 * W
    expert, head = 3 * ZEMOZEN_FF * W, ZEMOZEN_VOCAB * W
    places = ZEMOZEN_EXPERTS + ZEMOZEN_IDENTITIES

    def one(ns: list[int], before: list[int]) -> tuple[float, float]:
        """(bytes, operations) of a step with ns tokens of each request behind `before` others."""
        n, r = sum(ns), len(ns)
        used = ZEMOZEN_EXPERTS * (1 - (1 - ZEMOZEN_TOP / places) ** n)
        cached = n_layers * 4096 * sum(min(a, 1023) + b for a, b in zip(before, ns))
        states = n_par * 2 * 4 * 64 * 64 * 128 * r
        b = 2.0 * (dense + used * expert * n_layers + head) + cached + states + 2 * n * W + 4 * r * ZEMOZEN_VOCAB
        seen = sum(min(a + i, 1023) + 1 for a, b_ in zip(before, ns) for i in range(b_))
        f = 2.0 * n * (dense + n_layers * ZEMOZEN_TOP * ZEMOZEN_EXPERTS / places * expert) + 2.0 * r * head
        return b, f + n_layers * 4.0 * 4096 * seen + n_par * n * 4.0 * S * 128

    lengths = [len(p) - case.get("steps", 0) for p in _zemozen_prompts(case, 0)]
    each = [one(lengths, [0] * len(lengths))] + [one([1] * len(lengths), [a + s for a in lengths]) for s in range(case.get("steps", 0))]
    return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}


def _zemozen_exact(case: dict, seed: int):
    c = _zemozen_config()
    t = _zemozen_tensors(c)
    steps, eps = case.get("steps", 0), c.eps
    w = lambda name: t[name].to(F64)
    rms = lambda x: x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    silu = torch.nn.functional.silu

    def turn(x, pos, rot, pairs):
        n = rot["dims"]
        a = pos[:, None, None] * rot["base"] ** (-2 * torch.arange(n // 2, device="cuda", dtype=F64) / n) / (rot.get("scaling") or {"factor": 1.0})["factor"]
        u, v = (x[..., 0:n:2], x[..., 1:n:2]) if pairs else (x[..., :n // 2], x[..., n // 2:n])
        u, v = u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()
        return torch.cat([torch.stack([u, v], -1).flatten(-2) if pairs else torch.cat([u, v], -1), x[..., n:]], -1)

    def heads(h, p, m, pos, v, pairs):
        """Attention outputs [T, heads, vdim]; capped scores and a sink of score 0 with `softcap`."""
        T, H, G, D = len(h), m["heads"], m["kv_heads"], m["dim"]
        q = turn(rms((h @ w(p + "q").T).view(T, H, D)) * w(p + "q.norm"), pos, m["rot"], pairs)
        k = turn(rms((h @ w(p + "k").T).view(T, G, D)) * w(p + "k.norm"), pos, m["rot"], pairs)
        far = pos[:, None] - pos[None]
        hidden, out = (far < 0) | (far >= m["mask"]["size"]), []
        for i in range(H):
            s = q[:, i] @ k[:, i * G // H].T * m["scale"]
            if "softcap" in m:
                s = torch.cat([m["softcap"] * torch.tanh(s / m["softcap"]), torch.zeros(T, 1, device="cuda", dtype=F64)], 1)
                s[:, :T].masked_fill_(hidden, -math.inf)
                out.append(torch.softmax(s, -1)[:, :T] @ v[:, i * G // H])
            else:
                out.append(torch.softmax(s.masked_fill_(hidden, -math.inf), -1) @ v[:, i * G // H])
        return torch.stack(out, 1)

    def space(h, p, m):
        T, H, V, N, G = len(h), m["heads"], m["vdim"], m["state"], m["groups"]
        z, x, dt = (h @ w(p + "in").T).split([H * V, H * V + 2 * G * N, H], -1)
        x = torch.cat([torch.zeros(3, x.shape[1], device="cuda", dtype=F64), x])
        x = silu(sum(x[j:j + T] * w(p + "conv")[:, j] for j in range(4)) + w(p + "conv.b"))
        x, B, C = x.split([H * V, G * N, G * N], -1)
        x, B, C = x.view(T, H, V), B.view(T, G, N).repeat_interleave(H // G, 1), C.view(T, G, N).repeat_interleave(H // G, 1)
        dt = torch.nn.functional.softplus(dt + w(p + "dt_bias"))
        decay, S, y = torch.exp(-torch.exp(w(p + "A_log")) * dt), torch.zeros(H, N, V, device="cuda", dtype=F64), torch.empty_like(x)
        step = dt[..., None] * B
        for i in range(T):
            S = torch.baddbmm(S * decay[i, :, None, None], step[i, :, :, None], x[i, :, None])
            y[i] = (C[i, :, None] @ S)[:, 0]
        y = (y + w(p + "D")[:, None] * x).view(T, -1) * silu(z)
        return (rms(y.view(T, m["norm_groups"], -1)).view(T, -1) * w(p + "norm")) @ w(p + "o").T

    def one(tokens):
        T = len(tokens)
        pos, first_v = torch.arange(T, device="cuda"), None
        x = w("embed")[torch.tensor(tokens, device="cuda")] * c.embed_scale
        for i, L in enumerate(c.layers):
            p, m = f"l{i}.mix.", L.mixer
            h = rms(x) * w(f"l{i}.norm1")
            if L.type == "attention":
                v = (h @ w(p + "v").T).view(T, m["kv_heads"], m["vdim"])
                first_v = v if first_v is None else first_v
                v = v if first_v is v else (1 - w(p + "vmix")) * v + w(p + "vmix") * first_v
                y = (heads(h, p, m, pos, v, False) * torch.sigmoid(h @ w(p + "g").T)[..., None]).flatten(1) @ w(p + "o").T
            else:
                a, q = m["left"], p + "left."
                v = (h @ w(q + "v").T).view(T, a["kv_heads"], a["vdim"])
                y = m["left_scale"] * (heads(h, q, a, pos, v, True).flatten(1) @ w(q + "o").T) + m["right_scale"] * space(h, p + "right.", m["right"])
            x = x + c.residual_mult * y
            h, q = rms(x) * w(f"l{i}.norm2"), f"l{i}.mlp."
            s = torch.softmax(h @ w(q + "router").T, -1)
            ids = (s + w(q + "correction")).topk(L.top, -1).indices
            weight = s.gather(1, ids)
            weight = weight / weight.sum(-1, keepdim=True)
            y = torch.zeros_like(x)
            for e in ids.unique().tolist():
                r, j = (ids == e).nonzero(as_tuple=True)
                g = h[r] if e >= L.experts else (silu(h[r] @ w(f"{q}e{e}.gate").T) * (h[r] @ w(f"{q}e{e}.up").T)) @ w(f"{q}e{e}.down").T
                y.index_add_(0, r, weight[r, j, None] * g)
            x = x + c.residual_mult * y
        return (rms(x[T - 1 - steps:]) * w("final.norm")) @ w("head").T

    each = [one(p) for p in _zemozen_prompts(case, seed)]
    return [torch.stack([z[s] for z in each]) for s in range(steps + 1)]


# -- the interface --------------------------------------------------------------------------------------------------------------

_MODELS = {"qwen": (_qwen_prepare, _qwen_run, _qwen_work, _qwen_exact), "minimax": (_minimax_prepare, _minimax_run, _minimax_work, _minimax_exact),
           "zemozen": (_zemozen_prepare, _zemozen_run, _zemozen_work, _zemozen_exact)}


def prepare(case: dict, seed: int) -> dict:
    return {"model": case["model"], "state": _MODELS[case["model"]][0](case, seed)}


def run(state: dict):
    return _MODELS[state["model"]][1](state["state"])


def work(case: dict) -> dict:
    return _MODELS[case["model"]][2](case)


def tolerance(case: dict) -> dict:
    """Four times what the path was measured to be off `exact` (rel 6.6e-3, 5.0e-3, 3.0e-3; max 3.3e-2, 2.2e-2, 1.6e-2): activations are
    rounded to bf16 between the kernels."""
    rel, most = {"qwen": (0.026, 0.13), "minimax": (0.02, 0.09), "zemozen": (0.012, 0.065)}[case["model"]]
    return {"rel": rel, "max": most, "differ": 0.0}


@torch.no_grad()
def exact(case: dict, seed: int):
    return _MODELS[case["model"]][3](case, seed)
