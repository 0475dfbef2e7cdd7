"""The work that is timed: steps of the serving engine, through its step function.

A case is a program that serves a model: ``running`` requests with about ``context`` stored tokens
each are being decoded, and ``prompts`` new ones bring ``prompt_tokens`` tokens together, at most
``portion`` a step (0: all in one step).  One pass (``run``) admits the new requests, calls
``ModelRunner.step`` until their prompts are read, every running request taking one token in each of
these steps, and releases them; without new requests a pass is one decode step.  What comes back are
the logits of every step: those of the running requests and those after the last token of each
prompt.  Running requests grow by a token a step and start over ``ROOM`` tokens later.

The models are the layer sizes of ``bench.py``: Qwen2.5 with 1.5B and 7B parameters and the eight
layers of Puludra and Pikalorn at the width of the first.  Weights and tokens are random, drawn on
the device from the seed; ``exact`` is the same arithmetic in 64 bits, whole sequences at a time.
"""
from __future__ import annotations

import math

import torch

from dispec_b200 import ModelRunner, SeqEntry, load_model_config
from dispec_b200.weights import build_model, load_into

DEVICE = "cuda:0"
ROOM = 4096  # tokens a running request may grow by before it starts over
PREPARE_TOKENS = 8192  # tokens a step that reads the contexts of the running requests, before anything is timed

QWEN2 = {
    "1.5b": dict(num_hidden_layers=28, hidden_size=1536, num_attention_heads=12, num_key_value_heads=2,
                 intermediate_size=8960, vocab_size=151936, rms_norm_eps=1e-6, tie_word_embeddings=True),
    "7b": dict(num_hidden_layers=28, hidden_size=3584, num_attention_heads=28, num_key_value_heads=4,
               intermediate_size=18944, vocab_size=152064, rms_norm_eps=1e-6, tie_word_embeddings=False),
}
WIDTH, HEADS, DIM, FF, VOCAB = 1536, 12, 128, 8960, 151936  # of Puludra and Pikalorn
ROT_DIM, KV_RANK, Q_RANK, KV_HEADS = 64, 512, 768, 2


def model_config(name: str) -> dict:
    """config.json of a model."""
    if name in QWEN2:
        return dict(architectures=["Qwen2ForCausalLM"], model_type="qwen2", head_dim=128, rope_theta=1000000.0,
                    hidden_act="silu", max_position_embeddings=131072, use_sliding_window=False, **QWEN2[name])
    mlp = {"kind": "dense", "ff": FF}
    layer = lambda kind, mixer: {"type": kind, "mlp": mlp, "mixer": mixer}
    latent = {"heads": HEADS, "dim": DIM, "rot_dim": ROT_DIM, "vdim": DIM, "kv_rank": KV_RANK, "q_rank": Q_RANK,
              "scale": (DIM + ROT_DIM) ** -0.5, "rot": {"base": 1e6, "dims": ROT_DIM}}
    if name == "puludra":
        retention = layer("retention", {"heads": HEADS, "dim": DIM, "vdim": DIM, "rot": {"base": 1e6, "dims": DIM},
                                        "decay": [1 - 2.0 ** (-5 - 3 * i / (HEADS - 1)) for i in range(HEADS)]})
        hgrn2 = layer("hgrn2", {"heads": HEADS, "dim": DIM, "vdim": DIM})
        attention = layer("latent_attention", latent)
        return {"architecture": "Puludra", "vocab": VOCAB, "width": WIDTH, "postln_alpha": 2.0, "norm": {"eps": 1e-6},
                "layers": [retention, attention, hgrn2, attention] * 2}
    latent = dict(latent, rot={"base": 1e6, "dims": ROT_DIM,
                               "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}})
    delta = layer("delta", {"heads": HEADS, "kv_heads": HEADS, "dim": DIM, "vdim": DIM, "conv": 4})
    attention = layer("attention", {"heads": HEADS, "kv_heads": KV_HEADS, "dim": DIM, "vdim": DIM, "scale": DIM ** -0.5,
                                    "rot": {"base": 1e6, "dims": DIM}})
    return {"architecture": "Pikalorn", "vocab": VOCAB, "width": WIDTH, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6},
            "layers": [delta, layer("latent_attention", latent), delta, attention,
                       delta, layer("latent_attention", dict(latent, kv_from=1)), delta, attention]}


# ------------------------------------------------------------------------------------- cases
def case(model, running=0, context=0, prompts=0, prompt_tokens=0, portion=0, page=16, dtype="bfloat16"):
    return dict(model=model, dtype=dtype, running=running, context=context, prompts=prompts,
                prompt_tokens=prompt_tokens, portion=portion, page=page)


def listed():
    return [
        # one user waits for the next token: the smallest call, where launches and latency count
        dict(case("1.5b", running=1, context=1000), name="decode_1"),
        # a small service in the middle of its answers (the benchmark's batch)
        dict(case("1.5b", running=8, context=1024), name="decode_8"),
        # a busy service
        dict(case("1.5b", running=64, context=700), name="decode_64"),
        # an answer over a long document
        dict(case("1.5b", running=1, context=30000), name="decode_long"),
        # time to the first token of a chat message
        dict(case("1.5b", prompts=1, prompt_tokens=137), name="prompt_short"),
        # time to the first token of a document
        dict(case("1.5b", prompts=1, prompt_tokens=2048), name="prompt_2048"),
        # several prompts of different lengths read in one step
        dict(case("1.5b", prompts=9, prompt_tokens=4500), name="prompts_ragged"),
        # continuous batching: a prompt read in portions while other requests are decoded
        dict(case("1.5b", running=24, context=900, prompts=1, prompt_tokens=1100, portion=512), name="mixed"),
        # the larger size under the same load, in one step
        dict(case("7b", running=16, context=600, prompts=2, prompt_tokens=1000), name="mixed_7b"),
        # true 32-bit serving, as the trace replay for comparing logits runs it
        dict(case("1.5b", running=4, context=300, prompts=1, prompt_tokens=260, dtype="float32"), name="mixed_float32"),
        # latent attention and recurrences: prompts
        dict(case("puludra", prompts=2, prompt_tokens=2500), name="puludra_prompts"),
        # latent attention, delta rule and attention with sinks: a prompt in portions beside decoded requests
        dict(case("pikalorn", running=8, context=800, prompts=1, prompt_tokens=1500, portion=1024), name="pikalorn_mixed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same ranges: decode steps, prompts, or both."""
    model = rng.choice(["1.5b", "1.5b", "1.5b", "7b", "puludra", "pikalorn"])
    dtype = "float32" if model != "7b" and rng.random() < 0.12 else "bfloat16"
    kind = rng.choice(["decode", "prompts", "mixed"])
    page = rng.choice([16, 16, 16, 32, 64])
    most = 260 if dtype == "float32" else 1000 if model == "7b" else 2500 if model != "1.5b" else 4500
    running = context = prompts = tokens = portion = 0
    if kind != "prompts":
        small = dtype == "float32" or model == "7b"
        running = _log_int(rng, 1, 4 if dtype == "float32" else 16 if model == "7b" else 64 if kind == "decode" else 24)
        stored = 1200 if dtype == "float32" else 9600 if model == "7b" else 40000 if model == "1.5b" else 12000
        context = _log_int(rng, 40, min(stored // running, 2000 if small else 30000))
    if kind != "decode":
        prompts = rng.choice([1, 1, 1, 2, 3, 5])
        tokens = _log_int(rng, 20 * prompts, most if kind == "prompts" else most // 2)
        if kind == "mixed" and tokens > 300:
            portion = rng.choice([0, 256, 512])
    return case(model, running, context, prompts, tokens, portion, page, dtype)


def _shares(total, n):
    """``total`` tokens among ``n`` prompts of different lengths (weights 1, 2, 3, ... in a fixed shuffle)."""
    weights = [1 + (5 * i) % n for i in range(n)]
    out = [max(1, total * w // sum(weights)) for w in weights]
    out[-1] += total - sum(out)
    return out


def _contexts(c):
    """Stored tokens of each running request before a pass: ragged around ``context``."""
    n = c["running"]
    return [max(8, c["context"] * (8 + (3 * i) % 5) // 10 if n > 1 else c["context"]) for i in range(n)]


def _tokens(c, seed):
    """(tokens of the running requests, of the new prompts), as lists of host integers."""
    g = torch.Generator().manual_seed(seed * 7919 + 1)
    vocab = model_config(c["model"]).get("vocab_size", VOCAB)
    more = lambda n: torch.randint(0, vocab, (n,), generator=g).tolist()
    return ([more(n + ROOM + 64) for n in _contexts(c)],
            [more(n) for n in (_shares(c["prompt_tokens"], c["prompts"]) if c["prompts"] else [])])


def _portions(c, lengths):
    """The steps of a pass: for each, (prompt, first token, end) of every portion it carries."""
    budget = c["portion"] or sum(lengths)
    steps, room = [[]], budget
    for i, n in enumerate(lengths):
        at = 0
        while at < n:
            if room == 0:
                steps.append([])
                room = budget
            take = min(room, n - at)
            steps[-1].append((i, at, at + take))
            at, room = at + take, room - take
    return steps


# ------------------------------------------------------------------------------------- weights
def tensor_shapes(name: str) -> dict:
    cfg = model_config(name)
    if name in QWEN2:
        h, ff, V = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"]
        q, kv = cfg["num_attention_heads"] * cfg["head_dim"], cfg["num_key_value_heads"] * cfg["head_dim"]
        out = {"model.embed_tokens.weight": (V, h), "model.norm.weight": (h,)}
        if not cfg["tie_word_embeddings"]:
            out["lm_head.weight"] = (V, h)
        for i in range(cfg["num_hidden_layers"]):
            a, m = f"model.layers.{i}.self_attn.", f"model.layers.{i}.mlp."
            for n, rows in (("q", q), ("k", kv), ("v", kv)):
                out[f"{a}{n}_proj.weight"], out[f"{a}{n}_proj.bias"] = (rows, h), (rows,)
            out[f"{a}o_proj.weight"] = (h, q)
            out.update({f"{m}gate_proj.weight": (ff, h), f"{m}up_proj.weight": (ff, h), f"{m}down_proj.weight": (h, ff)})
            out[f"model.layers.{i}.input_layernorm.weight"] = out[f"model.layers.{i}.post_attention_layernorm.weight"] = (h,)
        return out
    H, d, W = HEADS, DIM, WIDTH
    out = {"embed": (VOCAB, W), "head": (VOCAB, W), "final.norm": (W,)}
    for i, layer in enumerate(cfg["layers"]):
        p, kind, m = f"l{i}.mix.", layer["type"], layer["mixer"]
        out[f"l{i}.norm1"] = (W,)
        out[p + "o"] = (W, H * d)
        if kind == "latent_attention":
            out.update({p + "dq": (Q_RANK, W), p + "dq.norm": (Q_RANK,), p + "uq": (H * (d + ROT_DIM), Q_RANK),
                        p + "uk": (H * d, KV_RANK), p + "uv": (H * d, KV_RANK)})
            if "kv_from" not in m:
                out.update({p + "dkv": (KV_RANK + ROT_DIM, W), p + "dkv.norm": (KV_RANK,)})
        elif kind == "retention":
            out.update({p + n: (H * d, W) for n in "qkvg"})
        elif kind == "hgrn2":
            out.update({p + n: (H * d, W) for n in "qfv"})
            out.update({p + "f.b": (H * d,), p + "lower": (H * d,), p + "norm": (d,)})
        elif kind == "delta":
            out.update({p + n: (H * d, W) for n in "qkvg"})
            out.update({p + n + ".conv": (H * d, m["conv"]) for n in "qkv"})
            out.update({p + "b": (H, W), p + "a": (H, W), p + "A_log": (H,), p + "dt_bias": (H,), p + "norm": (d,)})
        else:
            G = KV_HEADS
            out.update({p + "q": (H * d, W), p + "q.b": (H * d,), p + "k": (G * d, W), p + "k.b": (G * d,),
                        p + "q.norm": (d,), p + "k.norm": (d,), p + "g": (H * d, W), p + "o.b": (W,)})
        if name == "pikalorn" and kind in ("latent_attention", "attention"):
            out[p + "sink"] = (H,)
        p = f"l{i}.mlp."
        out.update({p + "up": (FF, W), p + "down": (W, FF)})
        if name == "puludra":
            out.update({f"l{i}.norm2": (W,), p + "act": (2,)})
        else:
            out[p + "gate"] = (FF, W)
    return out


def make_weights(c, seed) -> dict:
    """Random tensors by checkpoint name, on the device: matrices that keep the size of what passes through
    them, the last product of every sublayer smaller with the depth, gains around one."""
    g = torch.Generator(DEVICE).manual_seed(seed * 104729 + 3)
    store = torch.float32 if c["dtype"] == "float32" else torch.bfloat16
    depth, out = len(model_config(c["model"]).get("layers", [])) or 28, {}
    for name, shape in tensor_shapes(c["model"]).items():
        last = name.split(".")[-2 if name.endswith(".weight") else -1]
        t = torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float32 if len(shape) == 1 else store)
        if "norm" in last:
            t = 1.0 + 0.1 * t
        elif last == "lower":
            t = 0.9 * torch.sigmoid(t)
        elif last == "A_log":
            t = 0.7 * t - 1.0
        elif last == "dt_bias":
            t = t - 1.0
        elif last in ("act", "sink"):
            t = 0.5 * t
        elif last == "b" and name.endswith("f.b"):
            pass
        elif len(shape) == 1:  # biases
            t.mul_(0.1)
        elif last in ("embed", "embed_tokens"):
            t.mul_(0.02 if c["model"] in QWEN2 else 1.0)
        else:
            t.mul_(shape[-1] ** -0.5 * ((2 * depth) ** -0.5 if last in ("o_proj", "down_proj", "o", "down") else 1.0))
        out[name] = t.to(store)
    return out


class _Source:
    """The weights as ``load_into`` reads them."""

    def __init__(self, tensors):
        self.tensors = tensors

    def names(self):
        return list(self.tensors)

    def shape(self, name):
        return tuple(self.tensors[name].shape)

    def dtype(self, name):
        return self.tensors[name].dtype

    def get(self, name):
        return self.tensors[name]


# ------------------------------------------------------------------------------------- a pass
class _Service:
    """A model, its runner and the requests that are being decoded."""

    def __init__(self, c, seed):
        config = load_model_config(model_config(c["model"]))
        model = load_into(build_model(config), _Source(make_weights(c, seed)), c["dtype"], DEVICE)
        self.contexts = _contexts(c)
        self.running, self.prompts = _tokens(c, seed)
        self.steps = _portions(c, [len(p) for p in self.prompts])
        pages = sum((n + ROOM + 64) // c["page"] + 2 for n in self.contexts) + sum(len(p) // c["page"] + 2 for p in self.prompts)
        self.runner = ModelRunner(model, page_size=c["page"], num_pages=pages,
                                  max_num_seqs=max(1, c["running"] + c["prompts"]), cuda_graph=True)
        self.start()

    def start(self):
        """Reads the contexts of the running requests and decodes one token of each."""
        self.grown = 0
        entries, used = [], 0
        for i, n in enumerate(self.contexts):
            self.runner.admit(i)
            at = 0
            while at < n:
                take = min(n - at, PREPARE_TOKENS - used)
                entries.append(SeqEntry(i, self.running[i][at:at + take], at))
                at, used = at + take, used + take
                if used == PREPARE_TOKENS:
                    self.runner.step(entries)
                    entries, used = [], 0
        if entries:
            self.runner.step(entries)
        if self.contexts:
            self.decode([])

    def decode(self, more):
        """One step: a token of every running request, and ``more`` entries."""
        entries = []
        for i, n in enumerate(self.contexts):
            at = n + self.grown
            entries.append(SeqEntry(i, self.running[i][at:at + 1], at, [0]))
        self.grown += 1
        return self.runner.step(entries + more)


def prepare(c, seed):
    return _Service(c, seed)


def run(state):
    runner = state.runner
    if state.grown + len(state.steps) > ROOM:
        for i in range(len(state.contexts)):
            runner.release(i)
        state.start()
    names = [("prompt", i) for i in range(len(state.prompts))]
    for name, p in zip(names, state.prompts):
        runner.admit(name, len(p), len(p), len(p))
    logits = []
    for step in state.steps:
        more = [SeqEntry(names[i], state.prompts[i][a:b], a, [b - a - 1] if b == len(state.prompts[i]) else [])
                for i, a, b in step]
        logits.append(state.decode(more))
    for name in names:
        runner.release(name)
    return logits


# ------------------------------------------------------------------------------------- work
def _sizes(name):
    """(weights of the layers' matrices, output matrix, cached values a token, FLOPs a query and key, FLOPs a token in
    recurrences, bytes of a request's states)."""
    shapes = tensor_shapes(name)
    flat = ("embed", "model.embed_tokens.weight", "head", "lm_head.weight")
    matrices = sum(s[0] * s[1] for n, s in shapes.items() if len(s) == 2 and n not in flat and not n.endswith(".conv"))
    cfg = model_config(name)
    if name in QWEN2:
        L, H, G = cfg["num_hidden_layers"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
        return matrices, cfg["vocab_size"] * cfg["hidden_size"], 2 * L * G * 128, 4 * L * H * 128, 0, 0
    cached = pair = token = state = 0
    for layer in cfg["layers"]:
        kind = layer["type"]
        if kind == "latent_attention":
            cached += 0 if "kv_from" in layer["mixer"] else KV_RANK + ROT_DIM
            pair += 2 * HEADS * (2 * DIM + ROT_DIM)  # on the latents expanded to keys and values
        elif kind == "attention":
            cached += 2 * KV_HEADS * DIM
            pair += 4 * HEADS * DIM
        else:
            state += 4 * HEADS * DIM * DIM
            token += (6 if kind == "delta" else 4) * HEADS * DIM * DIM
    return matrices, VOCAB * WIDTH, cached, pair, token, state


def work(c):
    matrices, head, cached, pair, token, state = _sizes(c["model"])
    element = 4 if c["dtype"] == "float32" else 2
    contexts = _contexts(c)
    lengths = _shares(c["prompt_tokens"], c["prompts"]) if c["prompts"] else []
    total = {"bytes": 0, "flops": 0}
    for s, step in enumerate(_portions(c, lengths)):
        tokens = len(contexts) + sum(b - a for _, a, b in step)
        wanted = len(contexts) + sum(b == lengths[i] for i, _, b in step)
        stored = sum(contexts) + len(contexts) * (s + 1) + sum(a for _, a, _ in step)  # read from the cache
        pairs = sum(n + s + 2 for n in contexts) + sum((b - a) * (a + b + 1) // 2 for _, a, b in step)
        total["bytes"] += (element * (matrices + (head if wanted else 0) + cached * (stored + tokens))
                           + 2 * state * (len(contexts) + len(step)) + 4 * wanted * (head // _width(c["model"])))
        total["flops"] += 2 * tokens * matrices + 2 * wanted * head + pair * pairs + token * tokens
    return total


def _width(name):
    return model_config(name).get("hidden_size", WIDTH)


def tolerance(c):
    """Against 64 bits the logits are 4e-6 off in float32; in bfloat16 1.4e-2 after the 28 layers of Qwen2 and 2e-3
    after the eight layers on a 32-bit stream."""
    if c["dtype"] == "float32":
        return {"rel": 2e-5}
    return {"rel": 0.03} if c["model"] in QWEN2 else {"rel": 0.01}


# ------------------------------------------------------------------------------------- in 64 bits
F = torch.float64


def _rms(x, w, eps):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _frequencies(rot):
    """(f_i, factor on cosine and sine); with ``scaling`` slow pairs are slowed further, those between blended."""
    dims, base, sc = rot["dims"], rot.get("base"), rot.get("scaling")
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=F, device=DEVICE) / dims)
    if not sc:
        return f, 1.0
    pair = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
    lo, hi = max(math.floor(pair(sc["fast"])), 0), min(math.ceil(pair(sc["slow"])), dims - 1)
    r = ((torch.arange(dims // 2, dtype=F, device=DEVICE) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / sc["factor"] * r + f * (1 - r), 0.1 * math.log(sc["factor"]) + 1.0


def _turn(x, rot, interleaved=False):
    """x [T, heads, dims], positions from 0: pairs (2i, 2i + 1) or (i, i + dims / 2)."""
    f, m = _frequencies(rot)
    a = torch.arange(x.shape[0], dtype=F, device=DEVICE)[:, None] * f
    c, s = (torch.cos(a) * m)[:, None], (torch.sin(a) * m)[:, None]
    half = rot["dims"] // 2
    u, v = (x[..., 0::2], x[..., 1::2]) if interleaved else (x[..., :half], x[..., half:])
    p, q = u * c - v * s, v * c + u * s
    return torch.stack([p, q], -1).flatten(-2) if interleaved else torch.cat([p, q], -1)


def _attention(q, k, v, scale, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv] of one sequence from position 0 -> [T, H dv]."""
    T, H = q.shape[:2]
    k, v = (t.repeat_interleave(H // t.shape[1], 1).transpose(0, 1) for t in (k, v))
    out, at = [], torch.arange(T, device=DEVICE)
    rows = max(16, min(T, (1 << 28) // (H * T)))
    for a in range(0, T, rows):
        b = min(T, a + rows)
        s = (q[a:b].transpose(0, 1) * scale) @ k[:, :b].transpose(1, 2)
        s.masked_fill_(at[None, None, :b] > at[None, a:b, None], -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(-1, b - a, 1)], -1)
        w = torch.softmax(s, -1)[..., :b]
        out.append((w @ v[:, :b]).transpose(0, 1).flatten(1))
    return torch.cat(out)


def _recurrence(q, k, v, decay):
    """S <- decay S + k v^T, o = S^T q, token after token; decay [T, H, d or 1]."""
    S, out = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F, device=DEVICE), torch.empty_like(v)
    for t in range(q.shape[0]):
        S.mul_(decay[t][:, :, None]).add_(k[t][:, :, None] * v[t][:, None, :])
        out[t] = (S * q[t][:, :, None]).sum(1)
    return out


def _delta_rule(q, k, v, beta, decay):
    """S <- g S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q."""
    S, out = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F, device=DEVICE), torch.empty_like(v)
    for t in range(q.shape[0]):
        S.mul_(decay[t][:, None, None])
        u = beta[t][:, None] * (v[t] - (S * k[t][:, :, None]).sum(1))
        S.add_(k[t][:, :, None] * u[:, None, :])
        out[t] = (S * q[t][:, :, None]).sum(1)
    return out


def _mixer(layer, w, h, eps, shared):
    """A mixer of Puludra or Pikalorn; ``w(name)``: its tensors in 64 bits; ``shared``: latents by layer."""
    T, kind, m = h.shape[0], layer["type"], layer["mixer"]
    heads = lambda name, n=HEADS: (h @ w(name).T).view(T, n, -1)
    silu = torch.nn.functional.silu
    if kind == "latent_attention":
        q = (_rms(h @ w("dq").T, w("dq.norm"), eps) @ w("uq").T).view(T, HEADS, -1)
        if "kv_from" in m:
            c, k_rot = shared[m["kv_from"]]
        else:
            down = h @ w("dkv").T
            c, k_rot = _rms(down[:, :KV_RANK], w("dkv.norm"), eps), _turn(down[:, None, KV_RANK:], m["rot"], True)
        shared["last"] = (c, k_rot)
        q = torch.cat([q[..., :DIM], _turn(q[..., DIM:], m["rot"], True)], -1)
        k = torch.cat([(c @ w("uk").T).view(T, HEADS, DIM), k_rot.expand(T, HEADS, ROT_DIM)], -1)
        y = _attention(q, k, (c @ w("uv").T).view(T, HEADS, DIM), m["scale"], w("sink"))
    elif kind == "retention":
        decay = torch.tensor(m["decay"], dtype=F, device=DEVICE)[None, :, None].expand(T, HEADS, 1)
        q, k = _turn(heads("q"), m["rot"]), _turn(heads("k"), m["rot"]) * DIM ** -0.5
        y = _rms(_recurrence(q, k, heads("v"), decay), None, eps).flatten(1) * silu(h @ w("g").T)
    elif kind == "hgrn2":
        low = w("lower")
        f = (low + (1 - low) * torch.sigmoid(h @ w("f").T + w("f.b"))).view(T, HEADS, DIM)
        y = _rms(_recurrence(silu(heads("q")), 1 - f, heads("v"), f), w("norm"), eps).flatten(1)
    elif kind == "delta":
        unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
        rows = []
        for n in "qkv":
            taps = w(n + ".conv")
            u = torch.nn.functional.pad((h @ w(n).T).T, (taps.shape[1] - 1, 0))
            y = sum(taps[:, j:j + 1] * u[:, j:j + T] for j in range(taps.shape[1]))
            rows.append(silu(y.T).view(T, HEADS, DIM))
        decay = torch.exp(-torch.exp(w("A_log")) * torch.nn.functional.softplus(h @ w("a").T + w("dt_bias")))
        y = _delta_rule(unit(rows[0]) * DIM ** -0.5, unit(rows[1]), rows[2], torch.sigmoid(h @ w("b").T), decay)
        y = _rms(y, w("norm"), eps).flatten(1) * silu(h @ w("g").T)
    else:
        q = (h @ w("q").T + w("q.b")).view(T, HEADS, DIM)
        k = (h @ w("k").T + w("k.b")).view(T, KV_HEADS, DIM)
        y = _attention(_turn(_rms(q, w("q.norm"), eps), m["rot"]), _turn(_rms(k, w("k.norm"), eps), m["rot"]), k,
                       m["scale"], w("sink"))
        return (y * torch.sigmoid(h @ w("g").T)) @ w("o").T + w("o.b")
    return y @ w("o").T


def _qwen2_layer(cfg, w, h):
    T, H, G, D = h.shape[0], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    heads = lambda n, count: (h @ w(f"{n}_proj.weight").T + w(f"{n}_proj.bias")).view(T, count, D)
    rot = {"dims": D, "base": cfg["rope_theta"]}
    y = _attention(_turn(heads("q", H), rot), _turn(heads("k", G), rot), heads("v", G), D ** -0.5)
    return y @ w("o_proj.weight").T


def _xielu(z, act):
    p, q = torch.nn.functional.softplus(act)
    return torch.where(z > 0, p * z * z, (0.5 + q) * (torch.expm1(z.clamp(max=0)) - z)) + z / 2


def _forward(name, weights, sequences):
    """The logits at the last ``want`` places of every sequence: [(tokens, want)] -> list of [want, vocab].
    Layer by layer over all sequences, each from its position 0."""
    cfg, silu = model_config(name), torch.nn.functional.silu
    spans, a = [], 0
    for ids, _ in sequences:
        spans.append((a, a + len(ids)))
        a += len(ids)
    ids = torch.tensor([t for s, _ in sequences for t in s], device=DEVICE)
    each = lambda f, h: torch.cat([f(h[a:b], i) for i, (a, b) in enumerate(spans)])
    if name in QWEN2:
        eps, embed = cfg["rms_norm_eps"], "model.embed_tokens.weight"
        x = weights[embed][ids].to(F)
        for i in range(cfg["num_hidden_layers"]):
            part = lambda n: (lambda t: weights[f"model.layers.{i}.{n}{t}"].to(F))
            h = _rms(x, part("input_layernorm.")("weight"), eps)
            x = x + each(lambda s, _: _qwen2_layer(cfg, part("self_attn."), s), h)
            h, m = _rms(x, part("post_attention_layernorm.")("weight"), eps), part("mlp.")
            x = x + (silu(h @ m("gate_proj.weight").T) * (h @ m("up_proj.weight").T)) @ m("down_proj.weight").T
        norm, head = "model.norm.weight", embed if cfg["tie_word_embeddings"] else "lm_head.weight"
    else:
        eps, x = cfg["norm"]["eps"], weights["embed"][ids].to(F)
        shared = [{} for _ in spans]
        for i, layer in enumerate(cfg["layers"]):
            w = lambda n: weights[f"l{i}.{n}"].to(F) if f"l{i}.{n}" in weights else None

            def mix(h, s):
                y = _mixer(layer, lambda n: w("mix." + n), h, eps, shared[s])
                if layer["type"] == "latent_attention":
                    shared[s][i] = shared[s]["last"]
                return y
            if name == "puludra":
                x = _rms(cfg["postln_alpha"] * x + each(mix, x), w("norm1"), eps)
                x = _rms(cfg["postln_alpha"] * x + _xielu(x @ w("mlp.up").T, w("mlp.act")) @ w("mlp.down").T, w("norm2"), eps)
            else:
                h = _rms(x, w("norm1"), eps)
                x = x + each(mix, h) + (silu(h @ w("mlp.gate").T) * (h @ w("mlp.up").T)) @ w("mlp.down").T
        norm, head = "final.norm", "head"
    out = []
    for (_, b), (_, want) in zip(spans, sequences):
        out.append(_rms(x[b - want:b], weights[norm].to(F), eps) @ weights[head].to(F).T)
    return out


def exact(c, seed):
    """The first pass's logits in 64 bits.  (Before it every running request has decoded one token.)"""
    if work(c)["flops"] > 1e15 or sum(_contexts(c)) > 70000:
        return None
    weights = make_weights(c, seed)
    running, prompts = _tokens(c, seed)
    steps = _portions(c, [len(p) for p in prompts])
    contexts = _contexts(c)
    sequences = [(running[i][:n + 1 + len(steps)], len(steps)) for i, n in enumerate(contexts)] + [(p, 1) for p in prompts]
    rows = []
    budget, group = 1 << 14, []  # tokens a group of sequences may have
    for s in sequences + [None]:
        if group and (s is None or sum(len(t) for t, _ in group) + len(s[0]) > budget):
            rows += _forward(c["model"], weights, group)
            group = []
        group.append(s)
    out = []
    for n, step in enumerate(steps):
        done = [i for i, _, b in step if b == len(prompts[i])]
        parts = [r[n:n + 1] for r in rows[:len(contexts)]] + [rows[len(contexts) + i] for i in done]
        out.append(torch.cat(parts) if parts else torch.zeros(0, weights[next(iter(weights))].shape[0], dtype=F))
    return out
