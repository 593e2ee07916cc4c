"""The calls whose speed counts: prompts and decoding of whole models through the engine.

A case is one model (a Qwen2.5 decoder, or a Sipilorn decoder for the layers that Qwen2.5 does not have: the gated
delta rule, windowed and gated attention, experts) with seeded random weights, a batch of sequences and one of two kinds of pass:

* "prompt": one step of the engine over all sequences' new tokens, with the logits of every sequence's last token.
  Sequences may hold tokens already (`held_*`): the pass is then a further turn of conversations whose earlier
  turns are in the cache.  Afterwards the sequences are cut back to what they held, as a session does.
* "decode": `steps` steps of the captured decode loop in its serving form, given token ids in from host memory and new
  ids back after each, as a replay of a recorded conversation or a program that constrains its tokens feeds it.  The
  logits of the last step come back beside the ids of all of them.  Consecutive passes go on where the last one ended.

Sequence lengths are spread between `shortest` and `longest` and belong to the case; weights and token ids come from
the seed.  `exact` computes the same logits in 64-bit torch, whole sequences without a cache.
"""
from __future__ import annotations

import math
import random
import zlib

import torch

from sonicboom_b200 import DecoderModel, Engine
from sonicboom_b200.config import spec_from_config_dict
from sonicboom_b200.sampling import Sampling

DEVICE = "cuda:0"
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}

# Layer sizes of the two Qwen2.5 models and the Sipilorn model that the benchmark runs.
MODELS = {
    "qwen2.5-7b": dict(
        architectures=["Qwen2ForCausalLM"], model_type="qwen2", hidden_size=3584, num_hidden_layers=28,
        num_attention_heads=28, num_key_value_heads=4, intermediate_size=18944, vocab_size=152064, rope_theta=1000000.0,
        rms_norm_eps=1e-6, tie_word_embeddings=False, use_sliding_window=False, max_position_embeddings=32768),
    "qwen2.5-1.5b": dict(
        architectures=["Qwen2ForCausalLM"], model_type="qwen2", hidden_size=1536, num_hidden_layers=28,
        num_attention_heads=12, num_key_value_heads=2, intermediate_size=8960, vocab_size=151936, rope_theta=1000000.0,
        rms_norm_eps=1e-6, tie_word_embeddings=True, use_sliding_window=False, max_position_embeddings=32768),
}


def _sipilorn(width, n_layers, vocab, heads, kv_heads, dim, window, d_heads, d_kv, d_dim, d_vdim, p_heads, p_kv, taps, ff,
              experts, top, expert_ff):
    """Three layers of the gated delta rule and one that runs it beside windowed attention, in turn; dense
    feed-forwards and experts in turn."""
    delta = {"heads": d_heads, "kv_heads": d_kv, "dim": d_dim, "vdim": d_vdim, "conv": taps}
    left = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "mask": {"size": window},
            "rot": {"base": 200000.0, "dims": dim // 2}}
    right = dict(delta, heads=p_heads, kv_heads=p_kv)
    layers = []
    for i in range(n_layers):
        mixer = {"type": "delta", "mixer": delta} if i % 4 < 3 else \
            {"type": "parallel", "mixer": {"left": left, "right": right, "left_scale": 0.9, "right_scale": 0.7}}
        mlp = {"kind": "moe", "router": {"experts": experts, "top": top}, "expert": {"ff": expert_ff}} if i % 2 else \
            {"kind": "dense", "ff": ff}
        layers.append(dict(mixer, mlp=mlp))
    return {"architecture": "Sipilorn", "vocab": vocab, "width": width, "norm": {"eps": 1e-5}, "logit_softcap": 30.0, "layers": layers}


MODELS["sipilorn-w2048"] = _sipilorn(
    width=2048, n_layers=8, vocab=32768, heads=16, kv_heads=4, dim=128, window=1024, d_heads=32, d_kv=16, d_dim=128, d_vdim=128,
    p_heads=16, p_kv=8, taps=4, ff=8192, experts=32, top=4, expert_ff=1024)


def _prompt(model, seqs, shortest, longest, held_shortest=0, held_longest=0, dtype="bfloat16", name=None):
    c = dict(model=model, dtype=dtype, kind="prompt", seqs=seqs, shortest=shortest, longest=longest,
             held_shortest=held_shortest, held_longest=held_longest)
    return dict(c, name=name) if name else c


def _decode(model, seqs, shortest, longest, steps, room, temperature=0.0, dtype="bfloat16", name=None):
    c = dict(model=model, dtype=dtype, kind="decode", seqs=seqs, shortest=shortest, longest=longest, steps=steps, room=room,
             temperature=temperature)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user, a small model, a short conversation: the least work a token can be, all latency
        _decode("qwen2.5-1.5b", 1, 333, 333, 8, 4096, name="token_1p5b"),
        # one user of the larger model at the benchmark's context
        _decode("qwen2.5-7b", 1, 2048, 2048, 4, 2048, name="token_7b"),
        # a small server: eight conversations of unequal length (the benchmark's batch), sampled
        _decode("qwen2.5-7b", 8, 1024, 3072, 4, 2048, temperature=0.7, name="decode_7b_b8"),
        # a busy server: the widest batch the benchmark runs
        _decode("qwen2.5-7b", 64, 512, 2560, 4, 1024, temperature=0.7, name="decode_7b_b64"),
        # a short question: a prompt of ordinary chat length, odd
        _prompt("qwen2.5-7b", 1, 97, 97, name="prompt_7b_97"),
        # the benchmark's prompt
        _prompt("qwen2.5-7b", 1, 2048, 2048, name="prompt_7b_2048"),
        # further turns of three long conversations, documents pasted in: unequal new and held parts
        _prompt("qwen2.5-7b", 3, 500, 3500, 900, 4100, name="turns_7b"),
        # the benchmark's batch of many short and long prompts
        _prompt("qwen2.5-1.5b", 64, 16, 1024, name="prompts_1p5b_b64"),
        # the 32-bit path, which results are checked against: a prompt ...
        _prompt("qwen2.5-1.5b", 1, 201, 201, dtype="float32", name="f32_prompt_1p5b"),
        # ... and its tokens one by one, a few sequences together
        _decode("qwen2.5-1.5b", 3, 100, 400, 2, 2048, dtype="float32", name="f32_decode_1p5b"),
        # the recurrent design with experts: a prompt of the benchmark's length ...
        _prompt("sipilorn-w2048", 1, 2048, 2048, name="prompt_sipilorn"),
        # ... and decoding at the benchmark's batch
        _decode("sipilorn-w2048", 8, 300, 1500, 8, 4096, name="decode_sipilorn_b8"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["decode"] * 4 + ["prompt"] * 4 + ["f32", "sipilorn", "sipilorn"])
    qwen = rng.choice(["qwen2.5-7b", "qwen2.5-1.5b"])
    if what == "decode":
        seqs = _log(rng, 1, 64)
        a, b = _log(rng, 100, 2400), _log(rng, 100, 2400)
        return _decode(qwen, seqs, min(a, b), max(a, b), 4, 1024 if seqs > 16 else 2048, rng.choice([0.0, 0.7]))
    if what == "prompt":
        total = _log(rng, 40, 6000 if qwen == "qwen2.5-7b" else 24000)     # of all sequences, at the most
        seqs = _log(rng, 1, max(1, min(64, total // 32)))
        longest = min(max(1, total // seqs), 4096)
        shortest = _log(rng, max(1, longest // 8), longest)
        held = rng.choice([0, 0, _log(rng, 64, 3000)]) if seqs <= 8 else 0
        return _prompt(qwen, seqs, shortest, longest, held // 3, held)
    if what == "f32":
        if rng.random() < 0.5:
            n = _log(rng, 17, 260)
            return _prompt("qwen2.5-1.5b", 1, n, n, dtype="float32")
        a, b = _log(rng, 60, 500), _log(rng, 60, 500)
        return _decode("qwen2.5-1.5b", rng.randint(1, 8), min(a, b), max(a, b), 2, 2048, dtype="float32")
    if rng.random() < 0.5:
        seqs = _log(rng, 1, 8)
        longest = _log(rng, 100, 4096 // seqs + 100)
        return _prompt("sipilorn-w2048", seqs, max(1, longest // rng.randint(1, 6)), longest)
    a, b = _log(rng, 100, 1500), _log(rng, 100, 1500)
    return _decode("sipilorn-w2048", _log(rng, 1, 24), min(a, b), max(a, b), 8, 4096)


# ---------------------------------------------------------------------------- what a case holds
def _spread(n, lo, hi, what):
    """n lengths between lo and hi, both ends among them, in an order of their own."""
    if n == 1:
        return [hi]
    rng = random.Random(f"{what} {n} {lo} {hi}")
    lengths = [lo, hi] + [rng.randint(lo, hi) for _ in range(n - 2)]
    rng.shuffle(lengths)
    return lengths


def _lengths(case):
    """(tokens held before the pass, tokens the first pass brings) of every sequence."""
    n = case["seqs"]
    if case["kind"] == "decode":
        return _spread(n, case["shortest"], case["longest"], "held"), [case["steps"]] * n
    return _spread(n, case["held_shortest"], case["held_longest"], "held"), _spread(n, case["shortest"], case["longest"], "new")


def _vocab(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


def _tokens(case, seed):
    """Per sequence: the tokens it holds and those that follow (for decoding, all that the loop has room for)."""
    g = torch.Generator().manual_seed(seed * 2 + 1)
    held, new = _lengths(case)
    if case["kind"] == "decode":
        new = [case["room"]] * case["seqs"]
    vocab = _vocab(MODELS[case["model"]])
    seqs = [torch.randint(0, vocab, (h + n,), generator=g).tolist() for h, n in zip(held, new)]
    return [s[:h] for s, h in zip(seqs, held)], [s[h:] for s, h in zip(seqs, held)]


def _weight(request, seed, dtype):
    """One tensor of the model, a function of the seed and its name.  Matrices, embeddings and biases are N(0, 0.02),
    norms vary around one; decays, gates and convolutions of the recurrence are spread as a trained model's are."""
    g = torch.Generator(device=DEVICE).manual_seed((seed << 32) ^ zlib.crc32(request.name.encode()))
    shape, last = tuple(request.shape), request.name.rsplit(".", 1)[-1]
    if request.role == "table":
        return torch.rand((shape[0], request.below), generator=g, device=DEVICE).topk(shape[1], dim=1).indices.to(torch.int32)
    t = torch.randn(shape, generator=g, device=DEVICE, dtype=dtype)
    if request.role == "norm":
        return t.mul_(0.05).add_(1.0)
    if last == "A_log":
        return t.mul_(1.5).sub_(2.5)         # decays from about 0.5 to 0.999 a token
    if last == "conv":
        t.mul_(0.3)
        t[:, -1].add_(0.7)
        return t
    return t.mul_(0.02)


def _requests(cfg):
    return {r.name: r for r in DecoderModel(spec_from_config_dict(cfg)[1], torch.float32, "cpu").tensor_requests()
            if not r.optional}


# ---------------------------------------------------------------------------- the passes
class _Kept:
    """The model as it is, its last logits kept in hand."""

    def __init__(self, decoder):
        self.decoder, self.logits = decoder, None

    def __getattr__(self, name):
        return getattr(self.decoder, name)

    def forward(self, plan, cache):
        self.logits = self.decoder.forward(plan, cache)
        return self.logits


def _fill(engine, slots, tokens):
    """Feeds sequences their held tokens, in steps of a bounded number of tokens."""
    batch, size = [], 0
    for s, t in zip(slots, tokens):
        if batch and size + len(t) > 8192:
            engine.step(batch)
            batch, size = [], 0
        batch.append((s, t, []))
        size += len(t)
    engine.step(batch)


def _start(state):
    """Decoding sequences at the place where they begin: their tokens in the cache and the loop captured."""
    case, engine = state["case"], state["engine"]
    for s in state["slots"]:
        engine.close(s)
    state["slots"] = [engine.open() for _ in state["held"]]
    _fill(engine, state["slots"], state["held"])
    state["loop"] = engine.decode_loop(state["slots"], [case["room"]] * case["seqs"],
                                       [Sampling(temperature=case["temperature"], seed=7).checked()] * case["seqs"])
    state["at"] = 0


def prepare(case, seed):
    cfg, dtype = MODELS[case["model"]], DTYPES[case["dtype"]]
    requests = _requests(cfg)
    decoder = DecoderModel(spec_from_config_dict(cfg)[1], dtype, DEVICE)
    decoder.bind(lambda name: _weight(requests[name], seed, dtype))
    held, new = _tokens(case, seed)
    room = sum((len(h) + len(n) + 63) // 64 * 64 for h, n in zip(held, new))
    model = _Kept(decoder)
    state = {"case": case, "model": model, "engine": Engine(model, max_tokens=room, n_slots=case["seqs"]),
             "held": held, "new": new, "slots": []}
    if case["kind"] == "decode":
        _start(state)
        state["feed"] = list(zip(*new))                      # the tokens of one step
    elif held[0]:
        state["slots"] = [state["engine"].open() for _ in held]
        _fill(state["engine"], state["slots"], held)
    return state


def run(state):
    case, engine, model = state["case"], state["engine"], state["model"]
    if case["kind"] == "decode":
        if state["at"] + case["steps"] > case["room"]:       # the conversations are full: they begin again
            state["loop"].close()
            _start(state)
        ids = []
        for i in range(state["at"], state["at"] + case["steps"]):
            ids.append(state["loop"].step_host(state["feed"][i]))
        state["at"] += case["steps"]
        return {"ids": torch.tensor(ids), "logits": list(model.logits.split(8))}
    slots = state["slots"] or [engine.open() for _ in state["new"]]
    logits = engine.step([(s, t, [len(t) - 1]) for s, t in zip(slots, state["new"])])
    for s, h in zip(slots, state["held"]):
        if h:
            engine.cache.truncate(s, len(h))
        else:
            engine.close(s)
    return {"logits": list(logits.split(8))}


# ---------------------------------------------------------------------------- what a pass needs
def _matrix_values(cfg):
    """(values of the matrices every row of a step goes through, values of the head, values of one expert and how many of
    how many a row goes through in how many layers)."""
    if "architecture" not in cfg:
        d, ff = cfg["hidden_size"], cfg["intermediate_size"]
        hd = d // cfg["num_attention_heads"]
        qkv = (cfg["num_attention_heads"] + 2 * cfg["num_key_value_heads"]) * hd
        return cfg["num_hidden_layers"] * (d * qkv + d * d + 3 * d * ff), d * cfg["vocab_size"], (0, 0, 1, 0)
    d, total, moe = cfg["width"], 0, (0, 0, 1, 0)
    for layer in cfg["layers"]:
        m = layer["mixer"]
        for part in [m] if layer["type"] == "delta" else [m["left"], m["right"]]:
            n = 2 * part["kv_heads"] * part["dim"] + 3 * part["heads"] * part["vdim"] + 2 * part["heads"]     # q k v gate o, b a
            if "rot" in part:
                n = (part["heads"] + part["kv_heads"]) * part["dim"] + (2 * part["heads"] + part["kv_heads"]) * part["vdim"]
            total += d * n
        mlp = layer["mlp"]
        if mlp["kind"] == "dense":
            total += 3 * d * mlp["ff"]
        else:
            moe = (2 * d * mlp["expert"]["ff"], mlp["router"]["top"], mlp["router"]["experts"], moe[3] + 1)
    return total, d * cfg["vocab"], moe


def work(case):
    cfg = MODELS[case["model"]]
    size = 2 if case["dtype"] == "bfloat16" else 4
    held, new = _lengths(case)
    passes, rows = (case["steps"], [1] * case["seqs"]) if case["kind"] == "decode" else (1, new)
    n_rows, n_seqs = sum(rows), case["seqs"]
    matrices, head, (expert, top, experts, moe_layers) = _matrix_values(cfg)
    hit = experts * (1.0 - (1.0 - top / experts) ** n_rows)              # experts that the rows' tables name
    nbytes = size * (matrices + head + moe_layers * expert * hit) + 4.0 * n_seqs * _vocab(cfg)
    flops = 2.0 * n_rows * (matrices + moe_layers * top * expert) + 2.0 * n_seqs * head
    if "architecture" not in cfg:
        layers, heads, kv = cfg["num_hidden_layers"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
        hd, window = cfg["hidden_size"] // heads, 1 << 30
        nbytes += size * n_rows * cfg["hidden_size"]
    else:
        a = next(layer["mixer"]["left"] for layer in cfg["layers"] if layer["type"] == "parallel")
        layers = sum(layer["type"] == "parallel" for layer in cfg["layers"])
        heads, kv, hd, window = a["heads"], a["kv_heads"], a["dim"], a["mask"]["size"]
        nbytes += size * n_rows * cfg["width"]
        for layer in cfg["layers"]:
            m = layer["mixer"] if layer["type"] == "delta" else layer["mixer"]["right"]
            state = m["heads"] * m["dim"] * m["vdim"]
            nbytes += 4.0 * n_seqs * state * (2 if case["kind"] == "decode" else 1)
            flops += 7.0 * n_rows * state
    for h, n in zip(held, rows):
        keys = min(h, window) + n
        pairs = sum(min(i + 1, window) for i in range(h, h + n))
        nbytes += 2.0 * size * layers * kv * hd * (keys + n)
        flops += 4.0 * layers * heads * hd * pairs
    return {"bytes": passes * nbytes, "flops": passes * flops}


def tolerance(case):
    """Relative errors against `exact` are, measured, 3.3e-2 to 4.9e-2 for the 7B layers in bfloat16 (28 layers of random
    weights multiply what the first ones round), 1.7e-2 for the 1.5B ones, 6e-3 for the recurrent model, 7.5e-6 to
    9e-6 in float32; two correct implementations differ by about as much again.  Sampled ids differ at near ties."""
    rel = 4e-5 if case["dtype"] == "float32" else {"qwen2.5-7b": 0.15, "qwen2.5-1.5b": 0.07, "sipilorn-w2048": 0.025}[case["model"]]
    return {"rel": rel, "max": 6 * rel, "differ": 0.3}


# ---------------------------------------------------------------------------- the same in 64 bits
F = torch.float64


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, base, dims):
    """x [T, heads, d]: the first `dims` values of a head turn with the position, value i with value i + dims/2."""
    half = dims // 2
    inv = float(base) ** (-2.0 * torch.arange(half, dtype=F, device=x.device) / dims)
    a = torch.arange(x.shape[0], dtype=F, device=x.device)[:, None] * inv
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], dim=-1)


def _attend(q, k, v, scale, window):
    """q [T, H, d], k and v [T, G, d]: causal softmax attention, at most `window` keys back."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    at = torch.arange(T, device=q.device)
    out = torch.empty(T, H, v.shape[2], dtype=F, device=q.device)
    for lo in range(0, T, 2048):
        hi = min(T, lo + 2048)
        back = at[lo:hi, None] - at[None, :hi]
        hidden = (back < 0) | (back >= window)
        for h in range(H):
            s = (q[lo:hi, h] @ k[:hi, h // (H // G)].T) * scale
            out[lo:hi, h] = torch.softmax(s.masked_fill_(hidden, -torch.inf), -1) @ v[:hi, h // (H // G)]
    return out


def _qwen2(cfg, W, seqs):
    """Logits of every sequence's last token; the sequences' rows side by side."""
    lens = [len(s) for s in seqs]
    d, H, G, eps = cfg["hidden_size"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["rms_norm_eps"]
    hd = d // H
    x = W("model.embed_tokens.weight")[torch.tensor([t for s in seqs for t in s], device=DEVICE)]
    last = torch.tensor(lens, device=DEVICE).cumsum(0) - 1
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * W(p + "input_layernorm.weight")
        q, k, v = (h @ W(p + f"self_attn.{n}_proj.weight").T + W(p + f"self_attn.{n}_proj.bias") for n in "qkv")
        mixed = []
        for qs, ks, vs in zip(q.split(lens), k.split(lens), v.split(lens)):
            qs, ks, vs = qs.view(-1, H, hd), ks.view(-1, G, hd), vs.view(-1, G, hd)
            mixed.append(_attend(_rotate(qs, cfg["rope_theta"], hd), _rotate(ks, cfg["rope_theta"], hd), vs, hd ** -0.5, 1 << 30))
        x = x + torch.cat(mixed).view(-1, d) @ W(p + "self_attn.o_proj.weight").T
        h = _rms(x, eps) * W(p + "post_attention_layernorm.weight")
        gate = h @ W(p + "mlp.gate_proj.weight").T
        gate = torch.nn.functional.silu(gate, inplace=True).mul_(h @ W(p + "mlp.up_proj.weight").T)
        x = x + gate @ W(p + "mlp.down_proj.weight").T
        del gate
    head = "model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"
    return (_rms(x[last], eps) * W("model.norm.weight")) @ W(head).T


def _delta_rule(h, W, p, m, eps, lens):
    """The gated delta rule over sequences side by side, before its output matrix: per head, from S = 0,
    S <- decay S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q."""
    H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    pad = lambda x: torch.nn.utils.rnn.pad_sequence(list(x.split(lens)), batch_first=True)       # noqa: E731

    def conv(name):
        x, w = pad(h @ W(p + name).T), W(p + name + ".conv")
        taps, T = w.shape[1], x.shape[1]
        x = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
        return torch.nn.functional.silu(sum(w[:, j] * x[:, j:j + T] for j in range(taps)))

    q, k, v = conv("q"), conv("k"), conv("v")
    B, T = q.shape[:2]
    q, k = (x.view(B, T, G, d) / torch.sqrt((x.view(B, T, G, d) ** 2).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    q, k = (x.repeat_interleave(H // G, dim=2) for x in (q * d ** -0.5, k))
    v = v.view(B, T, H, dv)
    beta = torch.sigmoid(pad(h @ W(p + "b").T))
    decay = torch.exp(-torch.exp(W(p + "A_log")) * torch.nn.functional.softplus(pad(h @ W(p + "a").T) + W(p + "dt_bias"), threshold=200.0))
    S = torch.zeros(B, H, d, dv, dtype=F, device=h.device)
    o = torch.empty(B, T, H, dv, dtype=F, device=h.device)
    for t in range(T):
        kt = k[:, t, :, None]                                                                      # [B, H, 1, d]
        S = S * decay[:, t, :, None, None]
        u = beta[:, t, :, None, None] * (v[:, t, :, None] - kt @ S)
        S = torch.baddbmm(S.view(B * H, d, dv), kt.reshape(B * H, d, 1), u.view(B * H, 1, dv)).view(B, H, d, dv)
        o[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
    o = torch.cat([o[b, :n] for b, n in enumerate(lens)])
    gate = torch.nn.functional.silu(h @ W(p + "g").T).view(-1, H, dv)
    return (_rms(o, eps) * W(p + "norm") * gate).reshape(-1, H * dv)


def _gated_attention(h, W, p, a, eps, lens):
    H, G, d, dv = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
    q = _rms((h @ W(p + "q").T).view(-1, H, d), eps) * W(p + "q.norm")
    k = _rms((h @ W(p + "k").T).view(-1, G, d), eps) * W(p + "k.norm")
    v = (h @ W(p + "v").T).view(-1, G, dv)
    turn = lambda x: _rotate(x, a["rot"]["base"], a["rot"]["dims"])                               # noqa: E731
    out = torch.cat([_attend(turn(qs), turn(ks), vs, a["scale"], a["mask"]["size"])
                     for qs, ks, vs in zip(q.split(lens), k.split(lens), v.split(lens))])
    return out.reshape(-1, H * dv) * torch.sigmoid(h @ W(p + "g").T)


def _sipilorn_logits(cfg, W, seqs):
    lens, eps = [len(s) for s in seqs], cfg["norm"]["eps"]
    tokens = torch.tensor([t for s in seqs for t in s], device=DEVICE)
    x = _rms(W("embed")[tokens], eps) * W("embed.norm")
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        h = _rms(x, eps) * W(p + "norm1")
        if layer["type"] == "delta":
            y = _delta_rule(h, W, p + "mix.", m, eps, lens) @ W(p + "mix.o").T
        else:
            y = m["left_scale"] * (_gated_attention(h, W, p + "mix.left.", m["left"], eps, lens) @ W(p + "mix.left.o").T)
            y = y + m["right_scale"] * (_delta_rule(h, W, p + "mix.right.", m["right"], eps, lens) @ W(p + "mix.right.o").T)
        h = _rms(x, eps) * W(p + "norm2")
        if mlp["kind"] == "dense":
            y = y + (torch.nn.functional.silu(h @ W(p + "mlp.gate").T) * (h @ W(p + "mlp.up").T)) @ W(p + "mlp.down").T
        else:
            mine, top = W(p + "mlp.table").long()[tokens], mlp["router"]["top"]
            for e in range(mlp["router"]["experts"]):
                rows = (mine == e).any(1).nonzero()[:, 0]
                y[rows] += torch.relu(h[rows] @ W(p + f"mlp.e{e}.up").T) ** 2 @ W(p + f"mlp.e{e}.down").T / top
        x = x + y
    last = torch.tensor(lens, device=DEVICE).cumsum(0) - 1
    logits = (_rms(x[last], eps) * W("final.norm")) @ W("head").T
    return cfg["logit_softcap"] * torch.tanh(logits / cfg["logit_softcap"])


def exact(case, seed):
    """The logits of the first eight sequences (more are a matter of time only), by group of eight as `run` gives them."""
    cfg, dtype = MODELS[case["model"]], DTYPES[case["dtype"]]
    requests = _requests(cfg)
    held, new = _tokens(case, seed)
    seqs = [h + (n[:case["steps"]] if case["kind"] == "decode" else n) for h, n in zip(held, new)]

    def weight(name):
        t = _weight(requests[name], seed, dtype)
        return t if requests[name].role == "table" else t.to(F)

    logits = (_sipilorn_logits if "architecture" in cfg else _qwen2)(cfg, weight, seqs[:8])
    out = {"logits": [logits] + [None] * ((len(seqs) - 1) // 8)}
    return dict(out, ids=None) if case["kind"] == "decode" else out
