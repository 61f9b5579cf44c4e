"""What the speed of this framework is measured on: decode steps and prompt passes of its two hybrid decoders.

A case is one pass of a whole decoder -- embedding, every layer, head -- at the widths of the repository's own
configurations (``qwen35-27b``, dense; ``qwen35-35b-a3b``, mixture of experts) over a slice of their layers: 8 of 64
dense layers, 8 of 40 expert layers.  The layers repeat with a period of four, so the slice holds every kind of layer
in the proportion of the whole; embedding and head are whole.  Weights are the GGUF blocks that the repository's
benchmark uses (the Q4_K_M mix; Q8_0 for some), KV pages are bf16.

* ``phase="decode"``: one token for each of ``rows`` resident sequences of about ``context`` tokens, as the replay of
  the captured step graph that serving uses: logits out, recurrent state and KV pages updated.
* ``phase="prefill"``: ``rows`` prompt tokens of one sequence that already holds ``context`` tokens (0: a new one),
  through ``prefill``: logits of the last row out, state and pages updated.

Sizes run from one row to 64 and from 256 to 32768 tokens of context (131072 over all rows) for decoding, and from 16
to 4096 prompt tokens after up to 12288 others: the defaults of the benchmark (4096 tokens, one row) are in the middle.
"""
from __future__ import annotations

import math
from dataclasses import replace
from typing import Dict, List

import torch

from hipengine_b200.loading.synth import build_random_model
from hipengine_b200.models import make_executor
from hipengine_b200.models.config import NAMED_CONFIGS
from hipengine_b200.models.decode_graph import DecodeGraphRunner

PAGE = 16
LAYERS = {"qwen35-27b": 8, "qwen35-35b-a3b": 8}
# A trained decoder's residual stream is several times what one layer adds to it.  Random layers over a random embedding of
# their own size would instead replace it in every layer, and carry each rounding on at full size.
EMBED_SCALE = {"qwen35-27b": 500.0, "qwen35-35b-a3b": 300.0}
KV_TOKENS = 131072           # most tokens that the sequences of one decode step hold together


def _case(name, model, phase, rows, context, recipe="q4_k_m") -> Dict[str, object]:
    return {"name": name, "model": model, "recipe": recipe, "phase": phase, "rows": rows, "context": context}


def listed() -> List[Dict[str, object]]:
    d, m = "qwen35-27b", "qwen35-35b-a3b"
    return [
        # one user's stream in the middle of the benchmark's context: the headline, bound by latency and launches
        _case("dense_decode_1x4096", d, "decode", 1, 4096),
        # one user deep in a long document
        _case("dense_decode_1x32768", d, "decode", 1, 32768),
        # a handful of users on one GPU
        _case("dense_decode_4x2500", d, "decode", 4, 2500),
        # a small serving batch
        _case("dense_decode_16x4096", d, "decode", 16, 4096),
        # a full serving batch of short chats
        _case("dense_decode_64x1000", d, "decode", 64, 1000),
        # a chat turn: a few words after an empty context
        _case("dense_prefill_37", d, "prefill", 37, 0),
        # a page of text, not a multiple of anything, with eight-bit weights
        _case("dense_prefill_777_q8", d, "prefill", 777, 0, "q8_0"),
        # the benchmark's prompt
        _case("dense_prefill_4096", d, "prefill", 4096, 0),
        # the last chunk of a long document
        _case("dense_prefill_4096_after_12288", d, "prefill", 4096, 12288),
        # the same three situations of serving with routed experts
        _case("moe_decode_1x4096", m, "decode", 1, 4096),
        _case("moe_decode_32x2048", m, "decode", 32, 2048),
        _case("moe_prefill_2048", m, "prefill", 2048, 0),
    ]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> Dict[str, object]:
    model = "qwen35-27b" if rng.random() < 0.7 else "qwen35-35b-a3b"
    recipe = "q8_0" if rng.random() < 0.25 else "q4_k_m"
    if rng.random() < 0.6:
        rows = _log_uniform(rng, 1, 64)
        c = {"phase": "decode", "rows": rows, "context": _log_uniform(rng, 256, min(32768, KV_TOKENS // rows))}
    else:
        c = {"phase": "prefill", "rows": _log_uniform(rng, 16, 4096),
             "context": 0 if rng.random() < 0.6 else _log_uniform(rng, 64, 12288)}
    return {"model": model, "recipe": recipe, **c}


# ----------------------------------------------------------------------------- inputs
def _config(case):
    model = case["model"]
    return replace(NAMED_CONFIGS[model], n_layers=LAYERS[model], embed_scale=EMBED_SCALE[model])


def _weights(case, seed: int):
    return build_random_model(_config(case), seed=seed, device="cuda", recipe=case["recipe"])


def _contexts(case, seed: int) -> List[int]:
    """Tokens that each sequence holds before the pass: the stated number for one, half of it to all of it for more."""
    rows, c = case["rows"], case["context"]
    if case["phase"] == "prefill" or rows == 1:
        return [c]
    g = torch.Generator().manual_seed(seed + 17)
    return (c // 2 + (torch.rand(rows, generator=g) * (c - c // 2)).long()).tolist()


def _token_ids(case, seed: int, n: int) -> List[int]:
    g = torch.Generator().manual_seed(seed + 29)
    return torch.randint(0, _config(case).vocab, (n,), generator=g).tolist()


def _geometry(case) -> Dict[str, int]:
    """Sequences, tokens that each may hold, KV pages of the pool (page 0 belongs to no sequence)."""
    seqs = case["rows"] if case["phase"] == "decode" else 1
    new = 1 if case["phase"] == "decode" else case["rows"]
    span = -(-(case["context"] + new) // PAGE)
    return {"seqs": seqs, "max_context": span * PAGE, "span": span, "pages": seqs * span + 1}


def _filled(case, seed: int) -> Dict[str, Dict[int, torch.Tensor]]:
    """What the sequences hold: keys of unit size (they are normalised per head), values and convolution windows of a
    projection's size, recurrent states of the size they settle at."""
    cfg, geo = _config(case), _geometry(case)
    g = torch.Generator(device="cuda").manual_seed(seed + 41)
    rand = lambda *s, dtype=torch.float32: torch.randn(*s, generator=g, device="cuda", dtype=dtype)
    out: Dict[str, Dict[int, torch.Tensor]] = {"kv": {}, "conv": {}, "gdn": {}}
    new = case["context"] == 0
    for i in range(cfg.n_layers):
        if cfg.is_full_attention_layer(i):
            if new:
                kv = torch.zeros(geo["pages"], 2, cfg.n_kv_heads, PAGE, cfg.head_dim, device="cuda", dtype=torch.bfloat16)
            else:
                kv = rand(geo["pages"], 2, cfg.n_kv_heads, PAGE, cfg.head_dim, dtype=torch.bfloat16)
                kv[:, 1] *= 1.4
            out["kv"][i] = kv
        else:
            shape_c = (geo["seqs"], cfg.linear_qkv_width, cfg.conv_kernel - 1)
            shape_s = (geo["seqs"], cfg.ssm_v_heads, cfg.ssm_state, cfg.ssm_state)
            out["conv"][i] = torch.zeros(shape_c, device="cuda") if new else 1.4 * rand(*shape_c)
            out["gdn"][i] = torch.zeros(shape_s, device="cuda") if new else 0.05 * rand(*shape_s)
    return out


def prepare(case, seed):
    cfg, geo = _config(case), _geometry(case)
    ex = make_executor(_weights(case, seed), device="cuda", max_slots=geo["seqs"], max_context=geo["max_context"])
    for have, want in zip((ex.kv, ex.conv_state, ex.gdn_state), _filled(case, seed).values()):
        for i, t in want.items():
            have[i].copy_(t)
    state = {"phase": case["phase"], "ex": ex, "new": case["context"] == 0, "start": case["context"],
             "held": [ex.kv[i] for i in sorted(ex.kv)] + [ex.conv_state[i] for i in sorted(ex.conv_state)] +
                     [ex.gdn_state[i] for i in sorted(ex.gdn_state)]}
    if case["phase"] == "prefill":
        state["tokens"] = _token_ids(case, seed, case["rows"])
        return state
    rows = case["rows"]
    contexts = _contexts(case, seed)
    runner = DecodeGraphRunner(ex, max_rows=rows)
    runner.set_rows(range(rows), _token_ids(case, seed, rows), contexts)
    # serving captures the step of a batch size once; what the capture's warm-up step wrote is put back
    runner.step(rows, max(contexts) + 1, greedy=False)
    for have, want in zip((ex.kv, ex.conv_state, ex.gdn_state), _filled(case, seed).values()):
        for i, t in want.items():
            have[i].copy_(t)
    state.update(runner=runner, rows=rows, max_ctx=max(contexts) + 1)
    return state


def run(state):
    ex = state["ex"]
    if state["phase"] == "decode":
        state["runner"].step(state["rows"], state["max_ctx"], greedy=False)
        return [state["runner"].logits[:state["rows"]], state["held"]]
    if state["new"]:
        ex.reset_slot(0)
    return [ex.prefill(0, state["tokens"], start_pos=state["start"]), state["held"]]


# ----------------------------------------------------------------------------- what a pass cannot do without
def _layer_elements(cfg):
    """Weights of one layer of each kind and its feed-forward part: ({"full", "linear", "ffn", "expert"}: elements)."""
    h = cfg.hidden
    full = h * (cfg.q_proj_width + 2 * cfg.kv_width) + cfg.q_width * h
    linear = h * (cfg.linear_qkv_width + 2 * cfg.ssm_inner + 2 * cfg.ssm_v_heads)
    expert = 3 * h * cfg.expert_ffn
    ffn = h * cfg.n_experts + 3 * h * cfg.shared_ffn if cfg.is_moe else 3 * h * cfg.ffn
    return {"full": full, "linear": linear, "ffn": ffn, "expert": expert}


def work(case):
    cfg = _config(case)
    e = _layer_elements(cfg)
    bits = 8.5 if case["recipe"] == "q8_0" else 4.5
    decode = case["phase"] == "decode"
    seqs, tokens = (case["rows"], case["rows"]) if decode else (1, case["rows"])
    held = case["rows"] * case["context"] * (0.75 if case["rows"] > 1 else 1.0) if decode else case["context"]
    n_full, n_lin = cfg.n_full_layers, cfg.n_linear_layers
    used = cfg.n_experts * (1 - (1 - cfg.n_experts_used / cfg.n_experts) ** tokens) if cfg.is_moe else 0
    streamed = n_full * e["full"] + n_lin * e["linear"] + cfg.n_layers * (e["ffn"] + used * e["expert"])
    active = n_full * e["full"] + n_lin * e["linear"] + cfg.n_layers * (e["ffn"] + cfg.n_experts_used * e["expert"])
    head = cfg.vocab * cfg.hidden
    heads_out = seqs
    kv_token = 2 * cfg.kv_width * 2
    state = seqs * 4 * (cfg.ssm_v_heads * cfg.ssm_state ** 2 + cfg.linear_qkv_width * (cfg.conv_kernel - 1))
    bytes_ = (streamed * bits / 8 + head * (8.5 if case["recipe"] == "q8_0" else 6.5625) / 8 +
              tokens * cfg.hidden * bits / 8 + n_full * kv_token * (held + tokens) +
              n_lin * state * (1 if case["context"] == 0 else 2) + heads_out * cfg.vocab * 4)
    keys = held + seqs if decode else tokens * (case["context"] + (tokens + 1) / 2)      # (row, key) pairs
    flops = (2 * tokens * active + 2 * heads_out * head + n_full * 4 * keys * cfg.q_width +
             n_lin * tokens * 8 * cfg.ssm_v_heads * cfg.ssm_state ** 2)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # Up to five rows (and the head, up to eight) multiply eight-bit activations, more rows bf16 ones, every product rounding
    # its input once.  Measured against 64 bits: at most 0.013 for the former (the head's logits), 0.009 for the latter.
    return {"rel": 0.03}


# ----------------------------------------------------------------------------- the same pass in 64 bits
F64 = torch.float64


def _dequant(raw: torch.Tensor, kind: int) -> torch.Tensor:
    """GGUF rows [n, bytes] -> [n, columns] in 64 bits."""
    n = raw.shape[0]
    half = lambda b: b.contiguous().view(torch.float16).to(F64)
    if kind == 0:
        return raw.contiguous().view(torch.float32).to(F64)
    if kind == 8:                                    # Q8_0: fp16 scale, 32 int8
        b = raw.reshape(n, -1, 34)
        return (half(b[..., :2]) * b[..., 2:].contiguous().view(torch.int8).to(F64)).reshape(n, -1)
    if kind == 12:                                   # Q4_K: fp16 d, fp16 dmin, 8 x (6-bit scale, 6-bit min), 256 nibbles
        b = raw.reshape(n, -1, 144)
        s, q = b[..., 4:16], b[..., 16:].reshape(n, -1, 4, 1, 32)
        sc = torch.cat([s[..., :4] & 63, (s[..., 8:] & 15) | (s[..., :4] >> 6 << 4)], -1).to(F64) * half(b[..., :2])
        mn = torch.cat([s[..., 4:8] & 63, (s[..., 8:] >> 4) | (s[..., 4:8] >> 6 << 4)], -1).to(F64) * half(b[..., 2:4])
        q = torch.cat([q & 15, q >> 4], 3).reshape(n, -1, 8, 32).to(F64)
        return (q * sc[..., None] - mn[..., None]).reshape(n, -1)
    assert kind == 14                                # Q6_K: 128 low nibbles, 64 x four high bit pairs, 16 int8 scales, d
    b = raw.reshape(n, -1, 210)
    lo, hi = b[..., :128].reshape(n, -1, 2, 2, 32), b[..., 128:192].reshape(n, -1, 2, 32)
    q = torch.stack([(lo[..., j % 2, :] >> (4 * (j // 2)) & 15) | ((hi >> 2 * j & 3) << 4) for j in range(4)], 3)
    sc = b[..., 192:208].contiguous().view(torch.int8).to(F64) * half(b[..., 208:])
    q = (q.to(F64) - 32).reshape(n, -1, 16, 16)
    return (q * sc[..., None]).reshape(n, -1)


class _Model64:
    """The decoder of a case in 64 bits over the same blocks."""

    def __init__(self, case, seed: int):
        self.cfg = _config(case)
        self.w = _weights(case, seed).tensors

    def mat(self, name: str, r0: int = 0, r1: int = None) -> torch.Tensor:
        t = self.w[name]
        return _dequant(t.raw[r0:r1], int(t.ggml_type))

    def vec(self, name: str) -> torch.Tensor:
        t = self.w[name]
        return t.raw.contiguous().view(torch.float32).to(F64).reshape(t.shape)

    def lin(self, x: torch.Tensor, name: str, step: int = 16384) -> torch.Tensor:
        n = self.w[name].raw.shape[0]
        return torch.cat([x @ self.mat(name, r, min(n, r + step)).t() for r in range(0, n, step)], -1)

    def norm(self, x: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + self.cfg.rms_eps) * w

    def rope(self, x: torch.Tensor, pos: torch.Tensor) -> torch.Tensor:
        half = self.cfg.rope_dim // 2
        inv = self.cfg.rope_theta ** (-torch.arange(half, dtype=F64, device=x.device) / half)
        ang = pos.to(F64)[:, None, None] * inv
        a, b = x[..., :half], x[..., half:2 * half]
        return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin(), x[..., 2 * half:]], -1)

    def full(self, p: str, x, kv, seq, pos):
        cfg, T = self.cfg, x.shape[0]
        H, G, D = cfg.n_heads, cfg.n_kv_heads, cfg.head_dim
        qg = self.lin(x, p + "attn_q.weight").reshape(T, H, 2, D)
        q = self.rope(self.norm(qg[:, :, 0], self.vec(p + "attn_q_norm.weight")), pos)
        k = self.norm(self.lin(x, p + "attn_k.weight").reshape(T, G, D), self.vec(p + "attn_k_norm.weight"))
        page = 1 + seq * self.span + pos // PAGE
        kv[page, 0, :, pos % PAGE] = self.rope(k, pos)
        kv[page, 1, :, pos % PAGE] = self.lin(x, p + "attn_v.weight").reshape(T, G, D)
        out = torch.empty(T, G, H // G, D, dtype=F64, device=x.device)
        for s in seq.unique().tolist():
            rows = (seq == s).nonzero()[:, 0]
            n = int(pos[rows].max()) + 1
            own = kv[1 + s * self.span:1 + (s + 1) * self.span].permute(1, 2, 0, 3, 4).reshape(2, G, -1, D)[:, :, :n]
            for part in rows.split(max(1, (1 << 26) // n)):
                for g in range(G):
                    sc = q[part].reshape(-1, G, H // G, D)[:, g] @ own[0, g].t() * cfg.scale()
                    dark = torch.arange(n, device=x.device)[None, None] > pos[part][:, None, None]
                    out[part, g] = torch.softmax(sc.masked_fill(dark, -math.inf), -1) @ own[1, g]
        o = out.reshape(T, H, D) * torch.sigmoid(qg[:, :, 1])
        return self.lin(o.reshape(T, H * D), p + "attn_output.weight")

    def linear(self, p: str, x, conv, gdn, decode: bool):
        cfg, T = self.cfg, x.shape[0]
        G, Hv, S, K = cfg.ssm_groups, cfg.ssm_v_heads, cfg.ssm_state, cfg.conv_kernel
        new = self.lin(x, p + "attn_qkv.weight")
        z = self.lin(x, p + "attn_gate.weight").reshape(T, Hv, S)
        beta = torch.sigmoid(self.lin(x, p + "ssm_beta.weight"))
        a = torch.nn.functional.softplus(self.lin(x, p + "ssm_alpha.weight") + self.vec(p + "ssm_dt.bias").reshape(-1))
        decay = torch.exp(self.vec(p + "ssm_a").reshape(-1) * a)
        # windows [sequence, channel, time], oldest first
        line = torch.cat([conv, new[:, :, None] if decode else new.t()[None]], 2)
        conv.copy_(line[:, :, 1 - K:])
        wc = self.vec(p + "ssm_conv1d.weight")
        n = line.shape[2] - K + 1
        y = torch.nn.functional.silu(sum(line[:, :, j:j + n] * wc[:, j, None] for j in range(K)))
        y = y.permute(0, 2, 1).reshape(T, -1)
        unit = lambda v: v / v.norm(dim=-1, keepdim=True).clamp(min=1e-6)
        heads = torch.arange(Hv, device=x.device) % G
        q = (unit(y[:, :G * S].reshape(T, G, S)) * S ** -0.5)[:, heads]
        k = unit(y[:, G * S:2 * G * S].reshape(T, G, S))[:, heads]
        v = y[:, 2 * G * S:].reshape(T, Hv, S)
        o = torch.empty_like(v)
        for t in range(1 if decode else T):
            at = slice(None) if decode else slice(t, t + 1)
            gdn *= decay[at][:, :, None, None]
            d = (v[at] - (k[at][:, :, None] @ gdn)[:, :, 0]) * beta[at][:, :, None]
            gdn += k[at][..., None] * d[:, :, None]
            o[at] = (q[at][:, :, None] @ gdn)[:, :, 0]
        o = self.norm(o, self.vec(p + "ssm_norm.weight").reshape(-1)) * torch.nn.functional.silu(z)
        return self.lin(o.reshape(T, -1), p + "ssm_out.weight")

    def glu(self, x, gate, up, down):
        return (torch.nn.functional.silu(x @ gate.t()) * (x @ up.t())) @ down.t()

    def ffn(self, p: str, x):
        cfg = self.cfg
        if not cfg.is_moe:
            act = torch.nn.functional.silu(self.lin(x, p + "ffn_gate.weight")) * self.lin(x, p + "ffn_up.weight")
            return self.lin(act, p + "ffn_down.weight")
        prob, ids = torch.softmax(self.lin(x, p + "ffn_gate_inp.weight"), -1).topk(cfg.n_experts_used, -1)
        prob = prob / prob.sum(-1, keepdim=True).clamp(min=6.1e-5)
        shared = self.glu(x, *(self.mat(p + f"ffn_{s}_shexp.weight") for s in ("gate", "up", "down")))
        out = torch.sigmoid(x @ self.mat(p + "ffn_gate_inp_shexp.weight").t()) * shared
        H, F = cfg.hidden, cfg.expert_ffn
        for e in ids.unique().tolist():
            t, j = (ids == e).nonzero(as_tuple=True)
            gate, up = (self.mat(p + f"ffn_{s}_exps.weight", e * F, (e + 1) * F) for s in ("gate", "up"))
            y = self.glu(x[t], gate, up, self.mat(p + "ffn_down_exps.weight", e * H, (e + 1) * H))
            out.index_add_(0, t, y * prob[t, j][:, None])
        return out

    def forward(self, tokens, seq, pos, span: int, held, decode: bool):
        self.span = span
        table = self.w["token_embd.weight"]
        h = _dequant(table.raw[tokens], int(table.ggml_type)) * self.cfg.embed_scale
        for i in range(self.cfg.n_layers):
            p = f"blk.{i}."
            x = self.norm(h, self.vec(p + "attn_norm.weight"))
            if self.cfg.is_full_attention_layer(i):
                h = h + self.full(p, x, held["kv"][i], seq, pos)
            else:
                h = h + self.linear(p, x, held["conv"][i], held["gdn"][i], decode)
            h = h + self.ffn(p, self.norm(h, self.vec(p + "post_attention_norm.weight")))
        h = h if decode else h[-1:]
        return self.lin(self.norm(h, self.vec("output_norm.weight")), "output.weight")


@torch.no_grad()
def exact(case, seed):
    geo, decode = _geometry(case), case["phase"] == "decode"
    held = {kind: {i: t.to(F64) for i, t in d.items()} for kind, d in _filled(case, seed).items()}
    dev = torch.device("cuda")
    tokens = torch.tensor(_token_ids(case, seed, case["rows"]), device=dev)
    if decode:
        seq = torch.arange(case["rows"], device=dev)
        pos = torch.tensor(_contexts(case, seed), device=dev)
    else:
        seq = torch.zeros(case["rows"], dtype=torch.long, device=dev)
        pos = case["context"] + torch.arange(case["rows"], device=dev)
    logits = _Model64(case, seed).forward(tokens, seq, pos, geo["span"], held, decode)
    return [logits, [held[kind][i] for kind in ("kv", "conv", "gdn") for i in sorted(held[kind])]]
