"""The work that is timed when this library's speed is measured: a batch of requests goes through `Engine.step`, all prompts
in one step, then one token per sequence and step, with the logits of every request's last place after each of them.

A case names a model (its sizes are those of the benchmark and the tests), a data type, the number of requests, the
lengths of their prompts and how many single tokens follow.  The single tokens are given, as in a replay, so that the
logits of two builds belong to the same tokens.  Weights are the library's own random ones.

The feed-forwards of the designs are dense here: which experts a random router picks turns on roundings, and a row that
took another expert has other logits, so that outputs of routed layers cannot be held against each other.  Kudonex, whose
feed-forwards are always routed, is left out for that reason, as are Zeluzen and Vokelix at width 4096, whose random
weights enlarge a bfloat16 rounding to several percent of the logits (measured against float64: 3 to 6 %; the others 0.3
to 2.5 %), and every model has six layers, as those of the benchmark's designs and of the LLaMA models beside them.
"""
import math
import re

import numpy as np
import torch

from inferllm_b200 import Engine, EngineOptions, StepItem, config_from_dict
from inferllm_b200.weights import tensor_decls

VOCAB = 32000
LAYERS = 6
LLAMA = {  # width, layers, heads, kv heads, head size, feed-forward, words, base, eps, positions, tied
    "tiny-a": (64, 2, 4, 4, 16, 176, 256, 1e4, 1e-5, 128, False),
    "tiny-b": (144, 3, 6, 2, 24, 384, 512, 5e5, 1e-6, 256, True),
    "llama-7b": (4096, LAYERS, 32, 32, 128, 11008, VOCAB, 1e4, 1e-5, 4096, False),      # the layers of these three sizes
    "llama-8b": (4096, LAYERS, 32, 8, 128, 14336, 128256, 5e5, 1e-5, 8192, False),
    "llama-13b": (5120, LAYERS, 40, 40, 128, 13824, VOCAB, 1e4, 1e-5, 4096, False),
}
SIZES = {"1k": (1024, 2816, 8, 2), "2k": (2048, 5632, 16, 4), "4k": (4096, 11008, 32, 8)}  # width, feed-forward, heads, kv heads
DESIGNS = ("vokelix-1k", "vokelix-2k") + tuple(d + "-" + z for d in ("vizosun", "tukulorn", "fifotar") for z in SIZES)
HEAD = 128       # channels of a head, and of the rows and columns of a recurrent layer's state


def listed():
    def case(name, model, dtype, prompts, shortest, longest, new):
        return dict(name=name, model=model, dtype=dtype, prompts=prompts, shortest=shortest, longest=longest, new=new)

    return [
        # the smallest model that the tests run, three short prompts: latency and launches
        case("tiny", "tiny-a", "bfloat16", 3, 5, 16, 8),
        # one user's chat turn at 7B size: a middling prompt, then an answer token by token
        case("chat-1", "llama-7b", "bfloat16", 1, 200, 200, 48),
        # one long prompt, whose first token is waited for (reading, retrieval, scoring)
        case("prompt-2048", "llama-7b", "bfloat16", 1, 2048, 2048, 0),
        # eight long conversations up to the end of the context
        case("long-8", "llama-7b", "bfloat16", 8, 1024, 4000, 60),
        # a full server: sixty-four unequal short requests
        case("serve-64", "llama-7b", "bfloat16", 64, 64, 384, 48),
        # sixteen unequal requests at the 8B size: keys and values shared by groups of heads, a large vocabulary
        case("serve-16", "llama-8b", "bfloat16", 16, 64, 2048, 48),
        # the checking mode in true float32, at the layer sizes of a 7B model
        case("float32", "llama-7b", "float32", 1, 512, 512, 32),
        # four designs with dense feed-forwards: prompts and answers at the widths of their benchmark, alone and in
        # batches, lengths that fill pages and lengths that do not
        case("vokelix", "vokelix-2k", "bfloat16", 1, 2048, 2048, 32),
        case("vizosun", "vizosun-2k", "bfloat16", 8, 250, 1500, 32),
        case("tukulorn", "tukulorn-4k", "bfloat16", 1, 1777, 1777, 32),
        case("fifotar", "fifotar-4k", "bfloat16", 1, 200, 200, 48),
        case("vokelix-32", "vokelix-1k", "bfloat16", 32, 100, 900, 48),
    ]


def draw(rng):
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("tiny", "llama", "llama", "llama", "float32", "design", "design", "design", "design", "design"))
    dtype = "bfloat16"
    if kind == "tiny":
        model, dtype = rng.choice(("tiny-a", "tiny-b")), rng.choice(("bfloat16", "float32"))
        budget, most, top = 600, 8, LLAMA[model][9] - 20
    elif kind == "llama":
        model = rng.choice(("llama-7b", "llama-7b", "llama-8b", "llama-13b"))
        budget, most, top = 16384 if model != "llama-13b" else 8192, 64, 4000
    elif kind == "float32":
        model, dtype = "llama-7b", "float32"
        budget, most, top = 2048, 8, 2048
    else:
        model = rng.choice(DESIGNS)
        budget, most, top = 16384, 64, 3000
    prompts = between(1, most)
    longest = min(between(8, top), max(8, budget // prompts))
    shortest = between(max(1, longest // 8), longest) if prompts > 1 else longest
    return dict(model=model, dtype=dtype, prompts=prompts, shortest=shortest, longest=longest, new=min(rng.choice((0, 8, 16, 32, 48)), 16 if kind == "tiny" else 48))


# ---------------------------------------------------------------- models


def config(model):
    """The configuration, as config.json holds it."""
    if model in LLAMA:
        width, layers, heads, kv, d, ff, vocab, base, eps, positions, tied = LLAMA[model]
        return dict(architectures=["LlamaForCausalLM"], hidden_size=width, num_hidden_layers=layers, num_attention_heads=heads, num_key_value_heads=kv,
                    head_dim=d, intermediate_size=ff, vocab_size=vocab, rope_theta=base, rms_norm_eps=eps, max_position_embeddings=positions,
                    tie_word_embeddings=tied)
    design, size = model.split("-")
    width, ff, H, G = SIZES[size]
    d, window, half = HEAD, dict(size=1024), max(1, H // 2)
    out = dict(architecture=design.capitalize(), width=width, vocab=VOCAB, norm=dict(eps=1e-5), max_positions=4096)
    mlp, att = dict(kind="dense", ff=ff), dict(heads=H, kv_heads=G, dim=d, vdim=d, scale=d ** -0.5)
    yarn = dict(factor=4.0, original=4096, fast=32.0, slow=1.0)
    if design == "vokelix":
        att["rot"] = dict(base=5e5, dims=d // 2, scaling=dict(factor=4.0, original=4096, fast=16.0, slow=2.0))
        linear = dict(heads=H, dim=d, vdim=d, decay=[1.0 - 2.0 ** -(5 + 5 * h / max(H - 1, 1)) for h in range(H)])
        kinds = dict(lightning=linear, attention=att, retention=dict(linear, rot=dict(base=1e4, dims=d)), reader=dict(att, kv_from=1))
        order = ("lightning", "attention", "retention", "reader", "lightning", "retention")
        out["postln_alpha"] = 1.5
    elif design == "vizosun":
        kinds = dict(channel_delta=dict(heads=H, kv_heads=half, dim=d, vdim=d, conv=4, a_rank=64, g_rank=64),
                     latent_attention=dict(heads=H, dim=d, vdim=d, q_rank=width // 4, kv_rank=128, scale=d ** -0.5, mask=window))
        order = ("channel_delta", "latent_attention") * 3
        out.update(embedding=dict(bigram=dict(buckets=65521, mul_prev=1000003, mul_cur=31)), loop=dict(start=1, stop=3, times=2))
    elif design == "tukulorn":
        kinds = dict(attention=dict(heads=H, kv_heads=G, dim=d // 2, vdim=d, diff=0.4, scale=(d // 2) ** -0.5, q_temp=dict(coef=0.25, every=256)),
                     latent_attention=dict(heads=H, dim=d, rot_dim=64, vdim=d, kv_rank=64, scale=(d + 64) ** -0.5, mask=window, rot=dict(base=5e5, dims=64)))
        order = ("attention", "latent_attention") * 3
        out.update(norm=dict(eps=1e-6), loop=dict(start=1, stop=3, times=2))
    else:
        kinds = dict(delta=dict(heads=H, kv_heads=half, dim=d, vdim=d, conv=4), attention=dict(att, softcap=50.0, v_mix=True, mask=window),
                     latent_attention=dict(heads=H, dim=d, rot_dim=64, vdim=d, q_rank=width // 4, kv_rank=64, scale=(d + 64) ** -0.5,
                                           rot=dict(base=5e5, dims=64, scaling=yarn)))
        order = ("delta", "attention", "delta", "latent_attention", "delta", "attention")
        mlp["limit"] = 7.0
        out.update(embedding=dict(scale=8.0), residual_mult=0.5, logit_softcap=30.0)
    out["layers"] = [dict(type="attention" if t == "reader" else t, mixer=kinds[t], mlp=mlp) for t in order]
    return out


def runs(cfg):
    """The layers in the order they run (a run of layers may be looped), each with whether a pass of the loop begins there."""
    n, loop = len(cfg["layers"]) if "layers" in cfg else cfg["num_hidden_layers"], cfg.get("loop")
    if not loop:
        return [(i, -1) for i in range(n)]
    inner = [(i, p if i == loop["start"] else -1) for p in range(loop["times"]) for i in range(loop["start"], loop["stop"])]
    return [(i, -1) for i in range(loop["start"])] + inner + [(i, -1) for i in range(loop["stop"], n)]


def lengths(case):
    """The prompts' lengths, spread from the shortest to the longest in no order."""
    lo, hi = case["shortest"], case["longest"]
    return [hi - int((hi - lo) * ((i * 0.6180339887498949) % 1.0) + 0.5) for i in range(case["prompts"])]


def words(case, seed):
    """Per request the ids of its prompt and the ids that follow."""
    cfg = config(case["model"])
    rng = np.random.default_rng(seed)
    return [rng.integers(0, cfg.get("vocab_size", cfg.get("vocab")), n + case["new"]).tolist() for n in lengths(case)]


# ---------------------------------------------------------------- what is timed


def prepare(case, seed):
    cfg, lens, new = config(case["model"]), lengths(case), case["new"]
    room = sum(-(-(n + new) // 64) * 64 for n in lens) + 64
    engine = Engine.from_config(config_from_dict(cfg), EngineOptions(dtype=case["dtype"], max_tokens=room, max_batch=len(lens)), seed=seed)
    ids = words(case, seed)
    return dict(engine=engine, prompts=[t[:n] for t, n in zip(ids, lens)], after=[[t[n + j] for t, n in zip(ids, lens)] for j in range(new)])


def run(state):
    engine, prompts = state["engine"], state["prompts"]
    slots = [engine.new_sequence() for _ in prompts]
    logits = [engine.step([StepItem(s, p, [len(p) - 1]) for s, p in zip(slots, prompts)])]
    for ids in state["after"]:
        logits.append(engine.step([StepItem(s, [t], [0]) for s, t in zip(slots, ids)]))
    for s in slots:
        engine.end_sequence(s)
    return logits


def work(case):
    """Matrices are read once per step and their products done once per token; a token's keys and values are read by the
    single tokens behind it; a recurrent layer's state is read and written by every single token."""
    cfg, lens, new = config(case["model"]), lengths(case), case["new"]
    size = 4 if case["dtype"] == "float32" else 2
    count = {}
    for name, (shape, _) in tensor_decls(config_from_dict(cfg)).items():
        layer = re.match(r"(?:model\.layers\.|l)(\d+)\.", name)
        if layer:
            count[int(layer[1])] = count.get(int(layer[1]), 0) + math.prod(shape)
    width, vocab = cfg.get("hidden_size", cfg.get("width")), cfg.get("vocab_size", cfg.get("vocab"))
    order = [i for i, _ in runs(cfg)]
    elements = sum(count[i] for i in order) + sum(2 * width * width for _, p in runs(cfg) if p >= 0 and case["model"].startswith("vizosun"))
    tokens, steps = sum(lens) + new * len(lens), 1 + new
    flops = 2 * elements * tokens + 2 * width * vocab * steps * len(lens)
    nbytes = size * ((elements + width * vocab) * steps + width * tokens) + 4 * vocab * steps * len(lens)
    for i in order:
        m = cfg["layers"][i]["mixer"] if "layers" in cfg else dict(heads=cfg["num_attention_heads"], kv_heads=cfg["num_key_value_heads"],
                                                                   dim=cfg["head_dim"], vdim=cfg["head_dim"], scale=1)
        if "scale" not in m:                       # a recurrent layer: a state of HEAD x HEAD per head
            flops += 6 * m["heads"] * HEAD * HEAD * tokens
            nbytes += 8 * m["heads"] * HEAD * HEAD * new * len(lens)
            continue
        span = (m.get("mask") or dict(size=1 << 30))["size"]
        per_pair = 2 * m["heads"] * ((m["dim"] + m.get("rot_dim", 0)) * (2 if "diff" in m else 1) + m["vdim"] * (2 if "diff" in m else 1))
        row = m["kv_heads"] * (m["dim"] * (2 if "diff" in m else 1) + m["vdim"]) if "kv_heads" in m else m["kv_rank"] + m.get("rot_dim", 0)
        for n in lens:
            seen = sum(min(p + 1, span) for p in range(n, n + new))
            pairs = n * (n + 1) // 2 if n <= span else span * (span + 1) // 2 + (n - span) * span
            flops += per_pair * (pairs + seen)
            nbytes += size * row * (seen + n + new)
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """Two correct builds: float32 sums in another order (1e-5 at 7B size, 5e-7 at the tiny ones), bfloat16 activations rounded
    in other places (0.8 to 2 % of the logits' norm, 0.3 % at the tiny sizes); what was seen, times two to four."""
    tiny = case["model"].startswith("tiny")
    if case["dtype"] == "float32":
        return dict(rel=4e-6, max=1e-4) if tiny else dict(rel=4e-5, max=1e-3)
    return dict(rel=1.2e-2, max=0.1) if tiny else dict(rel=3e-2, max=0.4)


# ---------------------------------------------------------------- the same in 64 bits


def exact(case, seed):
    """The logits in float64, whole sequences at once, without this library.  None where that takes long."""
    return Exact(case, seed).logits() if work(case)["flops"] < 4e14 else None


def rms(x, eps, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def silu(x):
    return x * torch.sigmoid(x)


def unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


class Exact:
    def __init__(self, case, seed, device=None):
        self.case, self.seed, self.cfg, self.lens = case, seed, config(case["model"]), lengths(case)
        self.dev = device or ("cuda" if torch.cuda.is_available() else "cpu")
        self.ids = words(case, seed)
        self.full = [len(t) for t in self.ids]
        self.longest = max(self.full)
        self.eps = self.cfg["rms_norm_eps"] if "rms_norm_eps" in self.cfg else self.cfg["norm"]["eps"]
        self.valid = (torch.arange(self.longest, device=self.dev)[None, :] < torch.tensor(self.full, device=self.dev)[:, None])
        self.first_values, self.kept = None, {}

    # the library's random numbers: csrc/random_init.h
    def w(self, name, *shape, mean=0.0):
        signed = lambda v: (v & (2 ** 64 - 1)) - 2 ** 64 * ((v >> 63) & 1)  # noqa: E731
        gamma, m1, m2, key = 0x9E3779B97F4A7C15, 0xBF58476D1CE4E5B9, 0x94D049BB133111EB, 0xCBF29CE484222325
        for c in name.encode():
            key = ((key ^ c) * 0x100000001B3) % 2 ** 64

        def fin(z, shift, mul=lambda a, b: a * signed(b)):
            z = mul(z ^ shift(z, 30), m1)
            z = mul(z ^ shift(z, 27), m2)
            return z ^ shift(z, 31)

        base = fin(((key ^ (self.seed * gamma % 2 ** 64)) + gamma) % 2 ** 64, lambda z, n: z >> n, lambda a, b: a * b % 2 ** 64)
        n, out = math.prod(shape), []
        for lo in range(0, n, 1 << 26):
            i = torch.arange(lo, min(n, lo + (1 << 26)), device=self.dev)
            total = torch.zeros_like(i)
            for j in (1, 2, 3):
                r = fin((3 * i + j) * signed(gamma) + signed(base), lambda z, n: (z >> n) & ((1 << (64 - n)) - 1))
                total += (r & 0xFFFF) + ((r >> 16) & 0xFFFF) + ((r >> 32) & 0xFFFF) + ((r >> 48) & 0xFFFF)
            v = (total - 393210).float() * (float(np.float32(0.02)) / 65536.0) + mean
            out.append((v if self.case["dtype"] == "float32" else v.bfloat16()).double())
        return torch.cat(out).view(shape)

    def lin(self, x, name, rows):
        return x @ self.w(name, rows, x.shape[-1]).t()

    # rows [tokens of all sequences, ...] <-> [sequence, position, ...]
    def pad(self, x):
        out = x.new_zeros(self.valid.shape + x.shape[1:])
        out[self.valid] = x
        return out

    def rotate(self, x, freqs, mag=1.0, halves=True):
        """Rotates the first 2 * len(freqs) channels of x [sequence, position, heads, channels]."""
        n = len(freqs)
        ang = torch.arange(x.shape[1], device=self.dev).double()[:, None] * torch.tensor(freqs, device=self.dev, dtype=torch.float64)
        c, s, out = (ang.cos() * mag)[:, None], (ang.sin() * mag)[:, None], x.clone()
        a, b = (slice(0, n), slice(n, 2 * n)) if halves else (slice(0, 2 * n, 2), slice(1, 2 * n, 2))
        out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
        return out

    def freqs(self, rot):
        dims, base, sc = rot["dims"], rot["base"], rot.get("scaling")
        f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
        if not sc:
            return f, 1.0
        at = lambda t: dims * math.log(sc["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        return [x / sc["factor"] * r + x * (1.0 - r) for x, r in zip(f, ramp)], 0.1 * math.log(sc["factor"]) + 1.0

    def attend(self, q, k, v, scale, window=0, chunk=0, cap=0.0, sink=None):
        """q [sequence, position, H, d], k and v with G heads; causal; sink: one more score per head that has no value."""
        H, G = q.shape[2], k.shape[2]
        out = q.new_zeros(q.shape[:3] + (v.shape[3],))
        for b, n in enumerate(self.full):
            p = torch.arange(n, device=self.dev)
            seen = p[None, :] <= p[:, None]
            if window:
                seen &= p[:, None] - p[None, :] < window
            if chunk:
                seen &= torch.div(p[None, :], chunk, rounding_mode="floor") == torch.div(p[:, None], chunk, rounding_mode="floor")
            step = max(1, min(H, (1 << 28) // (n * n)))
            for lo in range(0, H, step):
                h = torch.arange(lo, min(H, lo + step), device=self.dev)
                g = h * G // H
                s = q[b, :n, h].transpose(0, 1) @ k[b, :n, g].permute(1, 2, 0) * scale
                s = cap * torch.tanh(s / cap) if cap else s
                s = s.masked_fill(~seen, -math.inf)
                top = s.amax(-1, keepdim=True)
                top = top if sink is None else torch.maximum(top, sink[h][:, None, None])
                e = torch.exp(s - top)
                den = e.sum(-1, keepdim=True) + (0.0 if sink is None else torch.exp(sink[h][:, None, None] - top))
                out[b, :n, h] = ((e / den) @ v[b, :n, g].transpose(0, 1)).transpose(0, 1)
        return out

    def conv(self, x, name, taps):
        """Causal convolution per channel of x [sequence, position, channels]."""
        t, y = self.w(name, x.shape[-1], taps), torch.zeros_like(x)
        for j in range(taps):
            y[:, j:] += t[:, taps - 1 - j] * x[:, :x.shape[1] - j]
        return y

    def rows(self, x, *tail):
        return self.pad(x).view(self.valid.shape + tail)

    # -------- mixers: x [tokens, width] -> [tokens, width of the output map's input]

    def softmax_mixer(self, x, i, m, pre):
        """Grouped attention of LLaMA, Vokelix and Fifotar."""
        H, G, d, eps, kind = m["heads"], m["kv_heads"], m["dim"], self.eps, self.case["model"].split("-")[0]
        llama = kind in ("llama", "tiny")
        n = [pre + s for s in (("q_proj.weight", "k_proj.weight", "v_proj.weight") if llama else "qkv")]
        own = m.get("kv_from") is None
        q = self.lin(x, n[0], H * d)
        k, v = (self.lin(x, n[1], G * d), self.lin(x, n[2], G * d)) if own else (None, None)
        if kind == "vokelix":
            q = rms(q + self.w(pre + "q.b", H * d), eps, self.w(pre + "q.norm", H * d, mean=1.0))
            if own:
                k = rms(k + self.w(pre + "k.b", G * d), eps, self.w(pre + "k.norm", G * d, mean=1.0))
                v = v + self.w(pre + "v.b", G * d)
        if kind == "fifotar":
            if self.first_values is None:
                self.first_values = v
            else:
                lam = self.w(pre + "vmix", 1)
                v = (1.0 - lam) * v + lam * self.first_values
        q = self.rows(q, H, d)
        if own:
            k, v = self.rows(k, G, d), self.rows(v, G, d)
        if "rot" in m:
            f, mag = self.freqs(m["rot"])
            q = self.rotate(q, f, mag, llama)
            k = self.rotate(k, f, mag, llama) if own else None
        if not own:
            k, v = self.kept[m["kv_from"]]
        elif kind == "vokelix":                      # a later layer reads them
            self.kept[i] = k, v
        sink = self.w(pre + "sink", H) if kind == "vokelix" else None if llama else x.new_zeros(H)
        o = self.attend(q, k, v, m["scale"], chunk=(m.get("mask") or dict(size=0))["size"], cap=m.get("softcap", 0.0), sink=sink)[self.valid]
        if kind == "vokelix":
            o = o * torch.sigmoid(self.lin(x, pre + "g", H))[..., None]
        o = o.reshape(len(x), H * d)
        return o * torch.sigmoid(self.lin(x, pre + "g", H * d)) if kind == "fifotar" else o

    def latent_mixer(self, x, m, pre):
        """Attention through latents: Vizosun's (no rotation, a query latent), Tukulorn's and Fifotar's."""
        H, d, dv, r, rank, eps = m["heads"], m["dim"], m["vdim"], m.get("rot_dim", 0), m["kv_rank"], self.eps
        if "q_rank" in m:
            q = self.lin(rms(self.lin(x, pre + "dq", m["q_rank"]), eps, self.w(pre + "dq.norm", m["q_rank"], mean=1.0)), pre + "uq", H * (d + r))
        else:
            q = self.lin(x, pre + "q", H * (d + r))
        q, down = self.rows(q, H, d + r), self.lin(x, pre + "dkv", rank + r)
        c = rms(down[:, :rank], eps, self.w(pre + "dkv.norm", rank, mean=1.0))
        k, v = self.rows(self.lin(c, pre + "uk", H * d), H, d), self.rows(self.lin(c, pre + "uv", H * dv), H, dv)
        if r:
            f, mag = self.freqs(m["rot"])
            halves = self.case["model"].startswith("fifotar")
            shared = self.rotate(self.rows(down[:, rank:], 1, r), f, mag, halves).expand(-1, -1, H, -1)
            q, k = torch.cat([q[..., :d], self.rotate(q[..., d:], f, mag, halves)], -1), torch.cat([k, shared], -1)
        o = self.attend(q, k, v, m["scale"], window=(m.get("mask") or dict(size=0))["size"])[self.valid]
        if r:
            o = o * torch.sigmoid(self.lin(x, pre + "g", H))[..., None]
        return o.reshape(len(x), H * dv)

    def differential_mixer(self, x, m, pre):
        """Two score maps over the same values, the second subtracted."""
        H, G, d, dv, t = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["q_temp"]
        q = self.rows(self.lin(x, pre + "q", 2 * H * d) + self.w(pre + "q.b", 2 * H * d), H, 2, d)
        k = self.rows(self.lin(x, pre + "k", 2 * G * d) + self.w(pre + "k.b", 2 * G * d), G, 2, d)
        v = self.rows(self.lin(x, pre + "v", G * dv) + self.w(pre + "v.b", G * dv), G, dv)
        p = torch.arange(self.longest, device=self.dev)
        grow = 1.0 + t["coef"] * torch.log(torch.div(p + 1, t["every"], rounding_mode="floor").double() + 1.0)
        q = q * grow[:, None, None, None]
        lam = [torch.exp(self.w(pre + "lq" + c, d) @ self.w(pre + "lk" + c, d)) for c in "12"]
        a, b = (self.attend(q[..., c, :], k[..., c, :], v, m["scale"]) for c in (0, 1))
        return (rms(a - (lam[0] - lam[1] + m["diff"]) * b, self.eps) * (1.0 - m["diff"]))[self.valid].reshape(len(x), H * dv)

    def decay_mixer(self, x, m, pre, kind):
        """Linear attention with one fixed decay per head: Vokelix."""
        H, d = m["heads"], m["dim"]
        q, k, v, g = (self.lin(x, pre + s, H * d) for s in "qkvg")
        if kind == "lightning":
            q, k, v = silu(q), silu(k), silu(v)
        q, k, v = (self.rows(t, H, d) for t in (q, k, v))
        if kind == "retention":
            f, mag = self.freqs(m["rot"])
            q, k = self.rotate(q, f, mag), self.rotate(k, f, mag) * d ** -0.5
        decay = torch.tensor(m["decay"], device=self.dev, dtype=torch.float64)[None, :, None, None]
        S, o = x.new_zeros(len(self.full), H, d, d), torch.zeros_like(v)
        for t in range(self.longest):
            S = decay * S + k[:, t, :, :, None] * v[:, t, :, None, :]
            o[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0]
        o = o[self.valid]
        if kind == "retention":
            return rms(o, self.eps).reshape(len(x), H * d) * silu(g)
        return rms(o.reshape(len(x), H * d), self.eps, self.w(pre + "norm", H * d, mean=1.0)) * torch.sigmoid(g)

    def delta_mixer(self, x, m, pre, kind):
        """The gated delta rule: a decay per head (Fifotar) or per head and key channel (Vizosun)."""
        H, G, d = m["heads"], m["kv_heads"], m["dim"]
        q, k, v = (self.rows(silu(self.conv(self.pad(self.lin(x, pre + s, n * d)), pre + s + ".conv", m["conv"]))[self.valid], n, d)
                   for s, n in (("q", G), ("k", G), ("v", H)))
        q, k = (t.repeat_interleave(H // G, dim=2) for t in (unit(q) * d ** -0.5, unit(k)))
        beta, rate = self.pad(torch.sigmoid(self.lin(x, pre + "b", H))), torch.exp(self.w(pre + "A_log", H))
        if kind == "delta":
            a, gate = self.lin(x, pre + "a", H) + self.w(pre + "dt_bias", H), silu(self.lin(x, pre + "g", H * d))
            decay = torch.exp(-rate * self.pad(torch.nn.functional.softplus(a)))[..., None]
        else:
            a = self.lin(self.lin(x, pre + "a1", m["a_rank"]), pre + "a2", H * d) + self.w(pre + "dt_bias", H * d)
            gate = torch.sigmoid(self.lin(self.lin(x, pre + "g1", m["g_rank"]), pre + "g2", H * d))
            decay = torch.exp(-rate[:, None] * self.rows(torch.nn.functional.softplus(a), H, d))
        S, o = x.new_zeros(len(self.full), H, d, d), torch.zeros_like(v)
        for t in range(self.longest):
            S = decay[:, t, :, :, None] * S
            u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None, :] @ S)[:, :, 0])
            S = S + k[:, t, :, :, None] * u[:, :, None, :]
            o[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0]
        return rms(o[self.valid], self.eps, self.w(pre + "norm", d, mean=1.0)).reshape(len(x), H * d) * gate

    def feed_forward(self, x, names, ff, kind):
        g, u = self.lin(x, names[0], ff), self.lin(x, names[1], ff)
        if kind == "fifotar":
            g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
            h = g * torch.sigmoid(1.702 * g) * (u + 1.0)
        else:
            h = (torch.relu(g) if kind == "vizosun" else silu(g)) * u
        return self.lin(h, names[2], x.shape[-1])

    # -------- the models

    def logits(self):
        cfg, eps, kind = self.cfg, self.eps, self.case["model"].split("-")[0]
        llama = kind in ("llama", "tiny")
        width, vocab = cfg.get("hidden_size", cfg.get("width")), cfg.get("vocab_size", cfg.get("vocab"))
        ids = torch.tensor([t for s in self.ids for t in s], device=self.dev)
        table = self.w("model.embed_tokens.weight" if llama else "embed", vocab, width)
        x = table[ids] * (cfg["embedding"]["scale"] if kind == "fifotar" else 1.0)
        if kind == "vizosun":
            bg = cfg["embedding"]["bigram"]
            last = [None if j == 0 else s[j - 1] for s in self.ids for j in range(len(s))]
            at = [bg["buckets"] if p is None else (p * bg["mul_prev"] + c * bg["mul_cur"]) % bg["buckets"] for p, c in zip(last, ids.tolist())]
            x = x + self.w("bigram", bg["buckets"] + 1, width)[torch.tensor(at, device=self.dev)]
        start, offset = x, kind in ("vokelix", "tukulorn")       # there a norm's stored weight is the offset from one

        def norm(t, name):
            return rms(t, eps, 1.0 + self.w(name, width) if offset else self.w(name, width, mean=1.0))

        for i, loop in runs(cfg):
            if llama:
                p = "model.layers.%d." % i
                m = dict(heads=cfg["num_attention_heads"], kv_heads=cfg["num_key_value_heads"], dim=cfg["head_dim"], scale=cfg["head_dim"] ** -0.5,
                         rot=dict(dims=cfg["head_dim"], base=cfg["rope_theta"]))
                o = self.softmax_mixer(norm(x, p + "input_layernorm.weight"), i, m, p + "self_attn.")
                x = x + self.lin(o, p + "self_attn.o_proj.weight", width)
                names = [p + "mlp." + s + "_proj.weight" for s in ("gate", "up", "down")]
                x = x + self.feed_forward(norm(x, p + "post_attention_layernorm.weight"), names, cfg["intermediate_size"], kind)
                continue
            L, p = cfg["layers"][i], "l%d." % i
            m, t, names = L["mixer"], L["type"], [p + "mlp." + s for s in ("gate", "up", "down")]
            if loop >= 0 and kind == "vizosun":
                x = self.lin(torch.cat([x, start], -1), "loop.in", width)
            if loop > 0 and kind == "tukulorn":
                x = x + start
            h = x if kind == "vokelix" else norm(x, p + "norm1")
            if t == "latent_attention":
                y = self.latent_mixer(h, m, p + "mix.")
            elif t == "attention":
                y = self.differential_mixer(h, m, p + "mix.") if kind == "tukulorn" else self.softmax_mixer(h, i, m, p + "mix.")
            elif t in ("lightning", "retention"):
                y = self.decay_mixer(h, m, p + "mix.", t)
            else:
                y = self.delta_mixer(h, m, p + "mix.", t)
            y = self.lin(y, p + "mix.o", width)
            ff = L["mlp"]["ff"]
            if kind == "vokelix":                     # a norm after each sum
                x = norm(cfg["postln_alpha"] * x + y, p + "norm1")
                x = norm(cfg["postln_alpha"] * x + self.feed_forward(x, names, ff, kind), p + "norm2")
            elif kind == "vizosun":                   # mixer and feed-forward side by side
                x = x + y + self.feed_forward(h, names, ff, kind)
            elif kind == "tukulorn":                  # a factor per channel on what a sublayer gives
                y = y + self.w(p + "mix.o.b", width) if t == "attention" else y
                x = x + y * self.w(p + "ls1", width, mean=1.0)
                x = x + self.feed_forward(norm(x, p + "norm2"), names, ff, kind) * self.w(p + "ls2", width, mean=1.0)
            else:                                     # norms on both sides of a sublayer
                x = x + cfg["residual_mult"] * norm(y, p + "norm1b")
                x = x + cfg["residual_mult"] * norm(self.feed_forward(norm(x, p + "norm2"), names, ff, kind), p + "norm2b")
        tied = kind in ("vizosun", "fifotar") or cfg.get("tie_word_embeddings")
        head = table if tied else self.w("lm_head.weight" if llama else "head", vocab, width)
        starts = np.cumsum([0] + self.full[:-1])
        out = []
        for j in range(self.case["new"] + 1):
            z = norm(x[torch.tensor([s + n - 1 + j for s, n in zip(starts, self.lens)], device=self.dev)], "model.norm.weight" if llama else "final.norm")
            z = z @ head.t()
            out.append(30.0 * torch.tanh(z / 30.0) if kind == "fifotar" else z)
        return out
