"""What this framework is timed on: prompts, single-token steps and whole generations of its decoders, through `Model`.

A case names a configuration of `rai_b200.configs`, a data type, and one of four kinds of work:

  prompt    `Model.forward` of a batch of equal prompts on an empty cache: logits of the last position
  steps     a filled cache, `tokens` greedy steps of the batch kept on the device (`Model.decode_loop`), then one more step
            through `Model.forward`, whose logits show what the steps before it left in the cache
  session   what a chat program does: `Model.generate` (prompt of `length` tokens on the host, `tokens` sampled ones back),
            then one `Model.forward` of the last token
  ragged    the same for prompts of different lengths in one batch: `Model.generate_ragged`, `Model.forward_rows`

Weights are random, drawn on the GPU from the seed, at the scale that keeps a row's size through a matrix.  A trained model is
mostly sure of its next token, a random one never is; so the output matrix holds the embedding of the token before (or the
embedding itself, where the two are tied), and greedy tokens do not hang on the last bit of a sum.  For the same reason the
router of a model with experts reads well separated numbers that the token alone sets.
"""
import ctypes
import math

import numpy as np
import torch

from rai_b200 import _lib, configs, synth
from rai_b200.device import Cuda
from rai_b200.models import Model

_DTYPES = {"bf16": (_lib.BF16, torch.bfloat16), "f32": (_lib.F32, torch.float32)}


def _case(kind, config, batch, length, tokens=0, dtype="bf16"):
    return dict(kind=kind, config=config, dtype=dtype, batch=batch, length=length, tokens=tokens)


def listed():
    return [
        # one user, a small model: a 128-token prompt and an answer, where launches and latency are everything
        dict(_case("session", "qwen2-0.5b", 1, 128, 24), name="chat-0.5b"),
        # the same model in float32, an odd prompt: the precision the reference's examples run in on a CPU
        dict(_case("session", "qwen2-0.5b", 1, 77, 8, "f32"), name="chat-0.5b-f32"),
        # a small batch of short prompts and the start of their answers; heads of 80
        dict(_case("session", "phi2", 8, 512, 8), name="batch-phi2"),
        # reading long prompts (summaries, retrieval); heads of 96
        dict(_case("prompt", "phi3-mini", 4, 2048), name="prompt-phi3"),
        # answering after such a prompt: few sequences, every head has keys of its own
        dict(_case("steps", "phi3-mini", 4, 2048, 6), name="steps-phi3"),
        # prompts whose length is no multiple of anything; heads of 256, one for keys and values
        dict(_case("prompt", "gemma-2b", 3, 1001), name="prompt-gemma"),
        # a server's decode batch on a small model with a large vocabulary
        dict(_case("steps", "gemma-2b", 32, 1024, 6), name="steps-gemma"),
        # a server's decode batch on the 7B model: weights and cache stream once per step
        dict(_case("steps", "qwen2-7b", 64, 2048, 4), name="steps-7b"),
        # the largest: bulk prompt processing
        dict(_case("prompt", "qwen2-7b", 8, 4096), name="prompt-7b"),
        # requests of different lengths admitted together, then answered together
        dict(_case("ragged", "qwen2-7b", 16, 611, 6), name="ragged-7b"),
        # routed experts beside attention over shared keys and values, prompts and answers
        dict(_case("session", "votapel-1k", 8, 1024, 8), name="experts-1k"),
        # a linear recurrence alternating with windowed attention, prompts and answers
        dict(_case("session", "malasun-2k", 6, 1500, 8), name="recurrent-2k"),
    ]


# what may be drawn: configuration, data type, kinds, largest batch, longest prompt or context, most tokens of a prompt in all
# and of a cache in all
_RANGES = [
    ("qwen2-0.5b", "bf16", ("session", "prompt", "steps", "ragged"), 64, 3000, 24000, 60000),
    ("qwen2-0.5b", "f32", ("session",), 3, 200, 300, 0),
    ("phi2", "bf16", ("session", "prompt", "steps", "ragged"), 32, 1900, 8000, 24000),
    ("phi3-mini", "bf16", ("session", "prompt", "steps", "ragged"), 24, 3500, 9000, 24000),
    ("gemma-2b", "bf16", ("session", "prompt", "steps", "ragged"), 64, 4000, 16000, 100000),
    ("qwen2-7b", "bf16", ("session", "prompt", "steps", "ragged"), 64, 4500, 16000, 130000),
    ("votapel-1k", "bf16", ("session", "prompt", "ragged"), 32, 2500, 12000, 0),
    ("malasun-2k", "bf16", ("session", "prompt", "ragged"), 32, 2500, 12000, 0),
]


def draw(rng):
    config, dtype, kinds, most_batch, longest, prompt, cached = rng.choice(_RANGES)
    kind = rng.choice(kinds)
    whole = cached if kind == "steps" else prompt
    spread = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    length = spread(17, longest)
    batch = spread(2 if kind == "ragged" else 1, max(2, min(most_batch, whole // length)))
    return _case(kind, config, batch, length, 0 if kind == "prompt" else rng.randint(3, 10), dtype)


# ---- weights, prompts and cached keys and values, from the seed -------------------------------------------------------------

def _normal(shape, seed, index, dtype):
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 100003 + index)
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype)


def _levels(cfg, vocab, experts, groups, seed):
    """[vocab, experts]: for every token a number per expert, a different order each, no two close: a step per group of
    neighbours and a smaller one within it, whose sums keep apart."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 100003 + 99991)
    n = experts // groups
    order = torch.rand((vocab, groups), generator=g, device="cuda").argsort(-1).float()
    within = torch.rand((vocab, groups, n), generator=g, device="cuda").argsort(-1).float()
    return (0.343 * (order[..., None] - (groups - 1) / 2) + 0.2 * (within - (n - 1) / 2)).reshape(vocab, experts)


_INTO_STREAM = ("o_proj", "dense", "down", "fc2", "mix.o")


class _Weights:
    """Parameters by name, one at a time."""

    def __init__(self, cfg, seed, dtype):
        self.cfg, self.seed, self.dtype = cfg, seed, dtype
        self.shapes = {n: (i, s, k) for i, (n, s, k) in enumerate(synth.param_shapes(cfg))}
        moe = [x["mlp"] for x in cfg.get("layers", ()) if x["mlp"] and x["mlp"]["kind"] == "moe"]
        self.moe = moe[0] if moe else None

    def names(self):
        return list(self.shapes)

    def __getitem__(self, name):
        index, shape, kind = self.shapes[name]
        cfg, arch, last = self.cfg, self.cfg["arch"], name.rsplit(".", 1)[-1]
        n = lambda: _normal(shape, self.seed, index, self.dtype)  # noqa: E731
        if name in ("lm_head.weight", "head"):
            e = self["embed" if name == "head" else "model.embed_tokens.weight"]
            return torch.roll(e, 1, 0) * (1.0 / shape[1] ** 0.5)
        if name == "model.embed_tokens.weight":
            return n() * (1.0 / shape[1] ** 0.5) if arch == "gemma" else n()
        if name == "embed":
            e = n()
            if self.moe:
                e[:, :self.moe["experts"]] = _levels(cfg, shape[0], self.moe["experts"], self.moe["groups"], self.seed).to(self.dtype)
            return e
        if name == "pos":
            e = n() * 0.3
            e[:, :self.moe["experts"]] = 0
            return e
        if kind == "norm_w":
            return n() * 0.05 + (0.0 if arch == "gemma" else 1.0)
        if kind == "delta":
            e = n() * 0.1
            if self.moe:
                e[:self.moe["experts"]] = 0
            return e
        if kind in ("matrix", "fan_in"):
            if last == "router":
                e = n() * (0.002 / shape[1] ** 0.5)
                e[:, :shape[0]] += 3.0 * torch.eye(shape[0], device="cuda", dtype=self.dtype)
                return e
            w = n() * (1.0 / shape[1] ** 0.5)
            if any(part in name for part in _INTO_STREAM):
                w *= 0.5  # a layer adds less than what it was given, as trained ones do
                if self.moe:
                    w[:self.moe["experts"]] = 0  # nothing but the token sets what the router reads
            return w
        if kind == "conv":
            return n() * (1.0 / shape[1] ** 0.5)
        if kind == "gain":
            return 0.3 + 0.06 * n()
        if kind in ("lower", "forget_b", "act"):
            u = torch.erf(n().float()).to(self.dtype)  # within (-1, 1)
            return {"lower": 0.45 + 0.45 * u, "forget_b": 3.0 + 3.0 * u, "act": u}[kind]
        return n() if kind == "sink" else n() * 0.02  # sinks; biases


def _rng(case, seed):
    return np.random.Generator(np.random.PCG64([int(seed), case["batch"], case["length"]]))


def _prompt_ids(case, vocab, seed):
    """[batch, length] token ids; uniform, as nothing here depends on which are frequent."""
    return _rng(case, seed).integers(0, vocab, size=(case["batch"], case["length"]), dtype=np.int32)


def _lengths(case):
    """Prompt lengths of a ragged batch: from a few tokens to the longest, most of them short."""
    share = _rng(case, 0).uniform(math.log(min(0.03, 8 / case["length"])), 0.0, size=case["batch"])
    lens = np.maximum(1, np.round(case["length"] * np.exp(share))).astype(int)
    lens[0] = case["length"]
    return lens


def _config(case):
    cfg = configs.get(case["config"])
    room = case["length"] + case["tokens"] + 8
    if "layers" not in cfg:
        cfg["max_position_embeddings"] = max(cfg["max_position_embeddings"], room)
    return cfg


def _kv_heads(cfg):
    return cfg.get("num_key_value_heads") or cfg["num_attention_heads"]


def _cached_rows(case, cfg, layer, seed):
    """Rows [query | key | value] of a layer's cached tokens, sequence by sequence."""
    width = 3 * _kv_heads(cfg) * configs.head_dim(cfg)
    return _normal((case["batch"] * case["length"], width), seed, 50000 + layer, _DTYPES[case["dtype"]][1])


def prepare(case, seed):
    cfg, (dtype, torch_dtype) = _config(case), _DTYPES[case["dtype"]]
    b, s = case["batch"], case["length"]
    dev = Cuda(0)
    model = Model(cfg, dtype, dev, b, s + case["tokens"] + 8, b if case["kind"] == "steps" else b * s)
    weights = _Weights(cfg, seed, torch_dtype)
    for name in weights.names():
        model.update_param(name, weights[name])
    model.finalize()
    state = dict(case=case, model=model)
    ids = _prompt_ids(case, cfg["vocab_size"], seed)
    if case["kind"] == "ragged":
        state["prompts"] = [row[:n] for row, n in zip(ids, _lengths(case))]
    elif case["kind"] == "steps":
        cache = ctypes.c_void_p(_lib.lib().rb_model_kv_cache(model._m))
        nkv, d = _kv_heads(cfg), configs.head_dim(cfg)
        none = torch.zeros(64, device="cuda")
        q = torch.empty((b * s, nkv * d), dtype=torch_dtype, device="cuda")
        _lib.call("rb_kv_cache_set_len", cache, b, s)
        for layer in range(cfg["num_hidden_layers"]):  # a rotary width of 0: rows are stored as they are
            rows = _cached_rows(case, cfg, layer, seed)
            _lib.call("rb_rope_kv_append", dev.ctx, ctypes.c_void_p(rows.data_ptr()), None, 0, None, ctypes.c_void_p(none.data_ptr()),
                      ctypes.c_void_p(none.data_ptr()), 0, b, s, nkv, cache, layer, ctypes.c_void_p(q.data_ptr()), dtype)
        dev.synchronize()
        state.update(cache=cache, first=torch.from_numpy(ids[:, 0].copy()).cuda())
    else:
        state["ids"] = ids
    return state


def run(state):
    case, model = state["case"], state["model"]
    kind, b, s, n = case["kind"], case["batch"], case["length"], case["tokens"]
    if kind == "prompt":
        model.clear_kv_cache()
        return {"logits": model.forward(state["ids"], 0)}
    if kind == "steps":
        _lib.call("rb_kv_cache_set_len", state["cache"], b, s)
        tokens = model.decode_loop(state["first"], s, n)
        return {"tokens": tokens, "logits": model.forward(tokens[-1].reshape(b, 1), s + n)}
    if kind == "session":
        tokens = model.generate(state["ids"], n)
        return {"tokens": tokens, "logits": model.forward(tokens[:, -1:], s + n - 1)}
    tokens = model.generate_ragged(state["prompts"], n)
    return {"tokens": tokens, "logits": model.forward_rows(tokens[:, -1:], None, range(b))}


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------

def _sizes(cfg):
    """(parameters every token is multiplied by, those of the output matrix, those of one expert, experts, used, moe layers)"""
    head = expert = 0
    dense, layers = 0, cfg.get("layers", ())
    for name, shape, _ in synth.param_shapes(cfg):
        size = math.prod(shape)
        if name in ("lm_head.weight", "head"):
            head = size
        elif name in ("model.embed_tokens.weight", "embed", "pos"):
            if "layers" not in cfg and configs.tied(cfg):
                head = size
        elif ".mlp.e" in name:
            expert += size
        else:
            dense += size
    moe = [x["mlp"] for x in layers if x["mlp"] and x["mlp"]["kind"] == "moe"]
    if not moe:
        return dense, head, 0, 0, 0, 0
    return dense, head, expert // (len(moe) * moe[0]["experts"]), moe[0]["experts"], moe[0]["top"], len(moe)


def _attention(cfg):
    """Per layer: (multiply-adds per query and key over all heads, numbers cached per token, window)."""
    if "layers" not in cfg:
        d = configs.head_dim(cfg)
        return [(2 * cfg["num_attention_heads"] * d, 2 * _kv_heads(cfg) * d, 0)] * cfg["num_hidden_layers"]
    out = []
    for m in (x["mixer"] for x in cfg["layers"]):
        if m["type"] == "attention":
            shared = cfg["arch"] == "votapel"
            out.append((m["heads"] * (m["dim"] + m["vdim"]), m["kv_heads"] * (m["dim"] + (0 if shared else m["vdim"])), m.get("window", 0)))
    return out


def _state_size(cfg):
    """Numbers of recurrent state per sequence."""
    return sum(m["heads"] * m["dim"] * m["vdim"] for m in (x["mixer"] for x in cfg.get("layers", ())) if m["type"] == "hgrn2")


def work(case):
    cfg, lens = _config(case), [case["length"]] * case["batch"]
    if case["kind"] == "ragged":
        lens = [int(x) for x in _lengths(case)]
    b, es, vocab = case["batch"], 2 if case["dtype"] == "bf16" else 4, cfg["vocab_size"]
    dense, head, expert, experts, top, moe = _sizes(cfg)
    attention, state = _attention(cfg), _state_size(cfg)
    touched = lambda rows: moe * expert * experts * (1 - (1 - top / experts) ** rows) if moe else 0  # noqa: E731
    total = {"bytes": 0.0, "flops": 0.0}
    if case["kind"] != "steps":
        rows = sum(lens)
        total["bytes"] += es * (dense + head + touched(rows) + rows * sum(c for _, c, _ in attention) + b * vocab) + 4 * b * state + 4 * rows
        total["flops"] += 2.0 * rows * (dense + moe * top * expert) + 2.0 * b * head + 4.0 * rows * state
        for per, _, window in attention:
            total["flops"] += 2.0 * per * sum(n * (n + 1) / 2 if not window or n <= window else window * (window + 1) / 2 + (n - window) * window
                                              for n in lens)
    singles = {"prompt": 0, "steps": case["tokens"] + 1}.get(case["kind"], case["tokens"])
    for i in range(singles):
        keys = [n + i + 1 for n in lens]
        total["bytes"] += es * (dense + head + touched(b) + b * vocab) + 8 * b * state
        total["flops"] += 2.0 * b * (dense + head + moe * top * expert) + 4.0 * b * state
        for per, cached, window in attention:
            seen = sum(min(n, window) if window else n for n in keys)
            total["bytes"] += es * cached * seen
            total["flops"] += 2.0 * per * seen
    return total


def tolerance(case):
    # float32: 1.5e-6 from 64 bits.  bf16: the stream is rounded twice a layer and each sublayer's rows several times; from 64
    # bits that is 0.3 to 1.9 %, and two orders of summation are up to 1.4 times that from each other
    return {"rel": 1e-5} if case["dtype"] == "f32" else {"rel": 0.03}


# ---- the same in 64 bits, plain torch --------------------------------------------------------------------------------------

def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, adjust=None):
    """q [B, H, S, d] are the last S positions of k, v [B, G, T, ...]; adjust changes the scores [H, S, T] of a sequence."""
    (b, h, s, _), (g, t) = q.shape, k.shape[1:3]
    hidden = torch.arange(t, device=q.device) > torch.arange(t - s, t, device=q.device)[:, None]
    out = q.new_empty(b, h, s, v.shape[-1])
    for i in range(b):
        z = (q[i].reshape(g, -1, q.shape[-1]) @ k[i].double().transpose(1, 2)).reshape(h, s, t) * scale
        z, sink = (z, None) if adjust is None else adjust(z)
        z = z.masked_fill(hidden, -math.inf)
        if sink is not None:
            z = torch.cat([z, sink.reshape(h, 1, 1).expand(h, s, 1)], -1)
        p = torch.softmax(z, -1)[..., :t]
        out[i] = (p.reshape(g, -1, t) @ v[i].double()).reshape(h, s, -1)
    return out


def _heads(x, n):
    return x.reshape(*x.shape[:2], n, -1).transpose(1, 2)


def _merge(x):
    return x.transpose(1, 2).flatten(2)


def _turn(x, dims, base, first):
    pos = torch.arange(first, first + x.shape[2], device=x.device, dtype=torch.float64)
    angle = pos[:, None] * base ** (-torch.arange(0, dims, 2, device=x.device, dtype=torch.float64) / dims)
    a, b, rest = x[..., :dims // 2], x[..., dims // 2:dims], x[..., dims:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin(), rest], -1)


_ACT = {"silu": torch.nn.functional.silu, "gelu_new": lambda x: torch.nn.functional.gelu(x, approximate="tanh")}


def _decoder64(cfg, w, ids, last, prefix=None):
    """Logits [B, last, V] of the last positions of ids [B, S]; prefix(layer) gives keys and values cached before them."""
    arch, eps, act = cfg["arch"], configs.norm_eps(cfg), _ACT[cfg["hidden_act"]]
    nq, nkv, d, rot = cfg["num_attention_heads"], _kv_heads(cfg), configs.head_dim(cfg), configs.rotary_dim(cfg)

    def linear(x, name):
        y = x @ w[name + ".weight"].double().T
        return y + w[name + ".bias"].double() if name + ".bias" in w else y

    def norm(x, name):
        g = w[name + ".weight"].double()
        if arch == "phi2":
            return torch.nn.functional.layer_norm(x, x.shape[-1:], g, w[name + ".bias"].double(), eps)
        return _rms(x, eps) * (1.0 + g if arch == "gemma" else g)

    embed = w["model.embed_tokens.weight"]
    x = embed[ids].double() * (cfg["hidden_size"] ** 0.5 if arch == "gemma" else 1.0)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = norm(x, p + "input_layernorm")
        if arch == "phi3":
            q, k, v = linear(h, p + "self_attn.qkv_proj").split([nq * d, nkv * d, nkv * d], -1)
        else:
            q, k, v = (linear(h, p + f"self_attn.{n}_proj") for n in "qkv")
        before = prefix(i) if prefix else None
        first = before[0].shape[2] if before else 0
        q, k, v = _turn(_heads(q, nq), rot, cfg["rope_theta"], first), _turn(_heads(k, nkv), rot, cfg["rope_theta"], first), _heads(v, nkv)
        if before:
            k, v = torch.cat([before[0].double(), k], 2), torch.cat([before[1].double(), v], 2)
        a = linear(_merge(_attend(q, k, v, d ** -0.5)), p + ("self_attn.dense" if arch == "phi2" else "self_attn.o_proj"))
        if arch == "phi2":
            x = x + a + linear(act(linear(h, p + "mlp.fc1")), p + "mlp.fc2")
            continue
        x = x + a
        h = norm(x, p + "post_attention_layernorm")
        if arch == "phi3":
            gate, up = linear(h, p + "mlp.gate_up_proj").chunk(2, -1)
        else:
            gate, up = linear(h, p + "mlp.gate_proj"), linear(h, p + "mlp.up_proj")
        x = x + linear(act(gate) * up, p + "mlp.down_proj")
    x = norm(x[:, -last:], "model.final_layernorm" if arch == "phi2" else "model.norm")
    return x @ embed.double().T if configs.tied(cfg) else linear(x, "lm_head")


def _votapel64(cfg, w, ids, last):
    silu, eps = torch.nn.functional.silu, cfg["norm_eps"]
    get = lambda name: w[name].double()  # noqa: E731
    glu = lambda h, p: (silu(h @ get(p + ".gate").T) * (h @ get(p + ".up").T)) @ get(p + ".down").T  # noqa: E731
    x = get("embed")[ids] + get("pos")[:ids.shape[1]]
    at = torch.arange(1, ids.shape[1] + 1, device=ids.device)
    for i, layer in enumerate(cfg["layers"]):
        mix, mlp, m = layer["mixer"], layer["mlp"], f"l{i}.mix"
        h = _rms(x, eps) * (1.0 + get(f"l{i}.norm1"))
        q, k = _heads(h @ get(m + ".q").T + get(m + ".q.b"), mix["heads"]), _heads(h @ get(m + ".k").T + get(m + ".k.b"), mix["kv_heads"])
        q = q * (1.0 + mix["temp_coef"] * torch.log(at // mix["temp_every"] + 1.0).double())[:, None]
        cap = lambda z: (mix["softcap"] * torch.tanh(z / mix["softcap"]), get(m + ".sink"))  # noqa: E731
        y = _merge(_attend(q, k, k, mix["scale"], cap)) @ get(m + ".o").T + glu(h, f"l{i}.mlp.shared")
        s = torch.sigmoid(h @ get(f"l{i}.mlp.router").T)
        runs = s.reshape(*s.shape[:2], mlp["groups"], -1)
        kept = runs.topk(2, -1).values.sum(-1).topk(mlp["keep"], -1).indices
        open_ = torch.zeros(runs.shape[:3], dtype=torch.bool, device=s.device).scatter(-1, kept, True)
        best = runs.masked_fill(~open_[..., None], -1.0).flatten(2).topk(mlp["top"], -1)
        for e in range(mlp["experts"]):
            rows = (best.indices == e).any(-1)
            y[rows] += glu(h[rows], f"l{i}.mlp.e{e}") * (s[rows][:, e:e + 1] * mlp["router_scale"])
        x = x + cfg["residual_mult"] * y
    return (_rms(x[:, -last:], eps) * (1.0 + get("final.norm"))) @ get("head").T


def _malasun64(cfg, w, ids, last):
    eps, f = cfg["norm_eps"], torch.nn.functional
    get = lambda name: w[name].double()  # noqa: E731
    x = get("embed")[ids]
    t = torch.arange(ids.shape[1], device=ids.device, dtype=torch.float64)
    away = t[:, None] - t

    def conv(u, taps):
        return f.conv1d(f.pad(u.transpose(1, 2), (taps.shape[1] - 1, 0)), taps[:, None], groups=taps.shape[0]).transpose(1, 2)

    def recurrence(h, m, mix):
        part = lambda z: z.reshape(*z.shape[:2], mix["heads"], -1)  # noqa: E731
        q, lower, v = part(f.silu(h @ get(m + ".q").T)), get(m + ".lower"), part(h @ get(m + ".v").T)
        keep = part(lower + (1.0 - lower) * torch.sigmoid(h @ get(m + ".f").T + get(m + ".f.b")))
        s, out = q.new_zeros(*q[:, 0].shape, v.shape[-1]), []
        for i in range(q.shape[1]):
            s = keep[:, i, ..., None] * s + (1.0 - keep[:, i])[..., None] * v[:, i, :, None]
            out.append((q[:, i, :, None] @ s)[:, :, 0])
        return (_rms(torch.stack(out, 1), eps) * get(m + ".norm")).flatten(2) @ get(m + ".o").T

    for i, layer in enumerate(cfg["layers"]):
        mix, m = layer["mixer"], f"l{i}.mix"
        if mix["type"] == "hgrn2":
            y = recurrence(x, m, mix)
        else:
            q, k, v = (conv(x @ get(f"{m}.{n}").T + get(f"{m}.{n}.b"), get(f"{m}.{n}.conv")) for n in "qkv")
            q, k = _rms(q, eps) * get(m + ".q.norm"), _rms(k, eps) * get(m + ".k.norm")
            slopes = 2.0 ** (-8.0 * torch.arange(1, mix["heads"] + 1, device=x.device, dtype=torch.float64) / mix["heads"])
            near = lambda z: ((z - slopes[:, None, None] * away).masked_fill(away >= mix["window"], -math.inf), None)  # noqa: E731
            y = _merge(_attend(_heads(q, mix["heads"]), _heads(k, mix["kv_heads"]), _heads(v, mix["kv_heads"]), mix["scale"], near))
            y = (y * torch.sigmoid(x @ get(m + ".g").T)) @ get(m + ".o").T
        x = x + _rms(y, eps) * get(f"l{i}.norm1")
        z, (a, b) = x @ get(f"l{i}.mlp.up").T, f.softplus(get(f"l{i}.mlp.act"))
        low = z.clamp(max=0.0)
        z = 0.5 * z + torch.where(z > 0, a * z * z, (0.5 + b) * (torch.expm1(low) - low))
        x = x + _rms(z @ get(f"l{i}.mlp.down").T, eps) * get(f"l{i}.norm2")
    return (_rms(x[:, -last:], eps) * get("final.norm")) @ get("head").T


def _greedy64(model, ids, tokens, cfg):
    """Logits after `tokens` greedy tokens on ids [B, S]: a guess (what the output matrix was made for) is run whole, and mended
    where it is not what its own logits say, until it is."""
    step = 0 if "layers" not in cfg and configs.tied(cfg) else 1
    guess = (ids[:, -1:] + step * torch.arange(1, tokens + 1, device=ids.device)) % cfg["vocab_size"]
    for _ in range(tokens + 1):
        logits = model(torch.cat([ids, guess], 1), tokens + 1)
        said = logits[:, :tokens].argmax(-1)
        if torch.equal(said, guess):
            break
        guess = said
    return logits[:, -1], guess


@torch.no_grad()
def exact(case, seed):
    if work(case)["flops"] > 1.2e14:
        return None  # half a minute and more in 64 bits
    cfg, dtype = _config(case), _DTYPES[case["dtype"]][1]
    source = _Weights(cfg, seed, dtype)
    w = {name: source[name] for name in source.names()}
    kind, s, n, vocab = case["kind"], case["length"], case["tokens"], cfg["vocab_size"]
    ids = torch.from_numpy(_prompt_ids(case, vocab, seed)).cuda().long()
    plain = {"votapel": _votapel64, "malasun": _malasun64}.get(cfg["arch"], _decoder64)
    model = lambda t, last: plain(cfg, w, t, last)  # noqa: E731
    if kind == "prompt":
        out = model(ids, 1)
        return {"logits": out[:, 0] if cfg["arch"] == "phi2" else out}
    if kind == "steps":
        def prefix(layer):
            rows = _cached_rows(case, cfg, layer, seed).reshape(case["batch"], s, 3, _kv_heads(cfg), -1)
            return rows[:, :, 1].transpose(1, 2), rows[:, :, 2].transpose(1, 2)
        logits, _ = _greedy64(lambda t, last: _decoder64(cfg, w, t, last, prefix), ids[:, :1], n, cfg)
    elif kind == "session":
        logits, _ = _greedy64(model, ids, n, cfg)
    else:
        rows = [_greedy64(model, ids[i:i + 1, :m], n, cfg)[0] for i, m in enumerate(_lengths(case))]
        return {"tokens": None, "logits": torch.cat(rows)}
    return {"tokens": None, "logits": logits if cfg["arch"] == "phi2" else logits[:, None]}
