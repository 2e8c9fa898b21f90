"""What a user of this engine has it do, as cases that can be prepared, run, timed and compared.

A case is one or more steps of the engine's step function on a model with random weights: the contexts of its requests are
in the cache already (earlier steps stored them), the step's tokens are lists on the host, and the result is the float32
logits at the last token of every request, as a scheduler or `bin/trace_run` would take them.  The cases span

    decode      one token per request, from a lone short request to full batches and long contexts
    prefill     whole prompts, one or several of uneven lengths in a step
    chunk       a portion of a long prompt beside decoding requests (chunked prefill)
    request     a prompt and the decode steps that follow, from the admission to the release of the request

at the layer sizes of the Llama 3.1 8B and 3.2 3B and 1B presets in bfloat16, at the 1B sizes in float32 (the engine's other
type: the one to check a checkpoint, a quantisation or a trace against), and of the families beside Llama that between them
reach every kind of mixer: retention and chunked attention with mixed heads (Lifusun), latent and windowed attention and wkv
(Rodapel), matrix memory and attention beside a delta rule (Kobolix).  As in the benchmark of the families the larger models
are cut to their first layers, here so that two correct bfloat16 implementations still agree on the logits (behind 32 layers
of random weights they are 5 % off the exact ones).  Kobolix and routed feed-forwards are run in float32 only: in bfloat16
the choice of experts, and the sign of a memory that one token dominates, flip on roundings.

Fields of a case: `shape` (a preset; in bfloat16 with every feed-forward dense), `layers` of it, `dtype`, `batch` requests
with `context` tokens in the cache and `prompt` new ones, `riders` more with `rider_context` and one new token, `steps`
further decode steps, `spread` (how far lengths lie from their mean, as a share of it).
"""
import math
import random

import torch

from iitj_llm_coopt_b200 import LLM, StepEntry
from iitj_llm_coopt_b200.config.registry import architecture_for
from iitj_llm_coopt_b200.models.decoder import cache_needs, model_parameter_specs
from iitj_llm_coopt_b200.presets import shape_config
from iitj_llm_coopt_b200.weights.random_init import random_checkpoint

PAGE = 16
CONTEXT_STEP = 8192        # contexts are stored in portions of at most this many tokens
EXACT_FLOPS = 2.5e14       # what a GPU does in 64 bits within a few seconds

LAYERS = {"8b": 8, "3b": 12, "1b": 16, "lifusun-8b": 8, "lifusun-3b": 8, "lifusun-1b": 8, "rodapel-3b": 4, "rodapel-1b": 4,
          "kobolix-1b": 4}

_BASE = {"dtype": "bfloat16", "batch": 1, "context": 0, "prompt": 1, "riders": 0, "rider_context": 0,
         "steps": 0, "spread": 0.0}


def _case(name, shape, **fields):
    return {"name": name, "shape": shape, "layers": LAYERS[shape], **_BASE, **fields}


def listed():
    return [
        # one user at a prompt: the least work a step can have; launches and latency count
        _case("decode-1b-b1", "1b", context=500),
        # the headline configuration: eight long conversations at the 8B sizes
        _case("decode-8b-b8", "8b", batch=8, context=8192),
        # a server's decode batch, uneven contexts, a batch size between the padded ones
        _case("decode-3b-b37", "3b", batch=37, context=600, spread=0.7),
        # the headline prompt
        _case("prefill-8b-2048", "8b", prompt=2048),
        # a long document
        _case("prefill-8b-8111", "8b", prompt=8111),
        # several prompts of uneven, odd lengths in one step
        _case("prefill-1b-ragged", "1b", batch=7, prompt=571, spread=0.8),
        # a portion of a long prompt beside a decode batch
        _case("chunk-3b-15k", "3b", context=15000, prompt=512, riders=32, rider_context=700, spread=0.3),
        # float32: a prompt, and a few requests decoding
        _case("prefill-1b-f32", "1b", dtype="float32", prompt=777),
        _case("decode-1b-f32-b5", "1b", dtype="float32", batch=5, context=600, spread=0.5),
        # the other families: a prompt and the first decode steps behind it
        _case("request-lifusun-8b", "lifusun-8b", prompt=1500, steps=8),
        _case("request-rodapel-3b", "rodapel-3b", prompt=1111, steps=8),
        # matrix memories, a delta rule and routed experts, in float32
        _case("request-kobolix-1b-f32", "kobolix-1b", dtype="float32", prompt=333, steps=4),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "chunk", "f32-prefill", "f32-decode", "lifusun", "rodapel", "family-f32"])
    f = dict(_BASE, spread=round(rng.uniform(0.0, 0.8), 2))
    if kind == "decode":
        f.update(shape=rng.choice(["1b", "3b", "8b"]), batch=_log(rng, 1, 64))
        f["context"] = _log(rng, 100, min(8192, 40000 // f["batch"]))
    elif kind == "prefill":
        f.update(shape=rng.choice(["1b", "3b", "8b"]), batch=_log(rng, 1, 8))
        f["prompt"] = max(2, _log(rng, 64, 8000) // f["batch"])
    elif kind == "chunk":
        f.update(shape=rng.choice(["1b", "3b"]), context=_log(rng, 512, 15000), prompt=_log(rng, 64, 1024),
                 riders=rng.randint(0, 32), rider_context=_log(rng, 100, 1000))
    elif kind == "f32-prefill":
        f.update(shape="1b", dtype="float32", batch=rng.randint(1, 3))
        f["prompt"] = max(2, _log(rng, 16, 777) // f["batch"])
    elif kind == "f32-decode":
        f.update(shape="1b", dtype="float32", batch=_log(rng, 1, 16), context=_log(rng, 50, 700))
    elif kind == "family-f32":
        f.update(shape=rng.choice(["rodapel-1b", "kobolix-1b"]), dtype="float32", prompt=_log(rng, 16, 333), steps=rng.randint(1, 4))
    else:
        f.update(shape=f"{kind}-{rng.choice(['1b', '3b'])}", prompt=_log(rng, 64, 1500), steps=rng.randint(1, 8))
    return dict(f, layers=LAYERS[f["shape"]])


# ---- what a case consists of -----------------------------------------------------------------------------------------
def _config(case):
    cfg = shape_config(case["shape"])
    if "layers" not in cfg:
        return dict(cfg, num_hidden_layers=case["layers"])
    cfg["layers"] = cfg["layers"][:case["layers"]]
    if case["dtype"] == "bfloat16":
        dense = next(lay["mlp"] for lay in cfg["layers"] if lay["mlp"]["kind"] == "dense")
        for lay in cfg["layers"]:
            lay["mlp"] = dict(dense)
    return cfg


def _lengths(case):
    """[(tokens in the cache, new tokens)] of the case's requests."""
    rng = random.Random(case["batch"] * 100003 + case["context"] + case["prompt"] + case["riders"])

    def around(mean):
        return max(min(mean, 1), round(mean * (1.0 + case["spread"] * rng.uniform(-1.0, 1.0))))
    one = case["prompt"] == 1
    out = [(around(case["context"]) if one else case["context"], 1 if one else around(case["prompt"])) for _ in range(case["batch"])]
    return out + [(around(case["rider_context"]), 1) for _ in range(case["riders"])]


def _tokens(case, vocab, seed):
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(0, vocab, (c + n + case["steps"],), generator=g).tolist() for c, n in _lengths(case)]


def _spec(case):
    cfg = _config(case)
    arch = architecture_for(cfg)
    typed = arch.config_class.from_dict(cfg)
    return cfg, arch, typed, arch.model_spec(typed)


class _State:
    pass


def prepare(case, seed):
    cfg, arch, typed, spec = _spec(case)
    lengths, tokens = _lengths(case), _tokens(case, spec.vocab, seed)
    s = _State()
    s.case = case
    s.llm = LLM(config=typed, random_seed=seed, dtype=case["dtype"], page_size=PAGE, max_num_seqs=max(8, len(lengths)),
                num_pages=sum(-(-len(t) // PAGE) + 1 for t in tokens), max_num_batched_tokens=max(2048, sum(n for _, n in lengths)),
                max_model_len=max(len(t) for t in tokens) + PAGE, seed=0)
    s.runner, s.cache = s.llm.engine.runner, s.llm.engine.cache
    s.ids = [f"r{i}" for i in range(len(tokens))]
    s.contexts = [c for c, _ in lengths]
    s.steps = [[StepEntry(r, t[c:c + n], [n - 1]) for r, t, (c, n) in zip(s.ids, tokens, lengths)]]
    for j in range(case["steps"]):
        s.steps.append([StepEntry(r, [t[c + n + j]], [0]) for r, t, (c, n) in zip(s.ids, tokens, lengths)])
    for r, t, c in zip(s.ids, tokens, s.contexts):
        if c:
            s.cache.admit(r)
            for at in range(0, c, CONTEXT_STEP):
                s.runner.step([StepEntry(r, t[at:min(c, at + CONTEXT_STEP)], [])])
    return s


def run(s):
    cache, runner = s.cache, s.runner
    for r, c in zip(s.ids, s.contexts):
        if not c:
            cache.admit(r)
    if len(s.steps) == 1:
        out = [runner.step(s.steps[0])]
    else:
        out = [runner.step(entries).clone() for entries in s.steps]        # the next step writes into the same rows
    for r, c in zip(s.ids, s.contexts):
        if c:
            cache.truncate(r, c)          # back to the context, as after a rejected draft
        else:
            cache.release(r)
    return out


# ---- what it cannot do without ---------------------------------------------------------------------------------------
def _attention_layers(cfg):
    """(query heads, numbers of a key, numbers of a value, window or 0, chunk or 0) of every softmax attention."""
    if "layers" not in cfg:
        D = cfg["head_dim"]
        return [(cfg["num_attention_heads"], D, D, 0, 0)] * cfg["num_hidden_layers"]
    out = []
    for lay in cfg["layers"]:
        m = lay["mixer"].get("left", lay["mixer"])
        size = (m.get("mask") or {}).get("size", 0)
        if lay["type"] in ("attention", "parallel"):
            chunked = cfg["architecture"] == "Lifusun"
            out.append((m["heads"], m["dim"], m["vdim"], 0 if chunked else size, size if chunked else 0))
        elif lay["type"] == "latent_attention":
            out.append((m["heads"], m["dim"] + m["rot_dim"], m["vdim"], 0, 0))
    return out


def _recurrent_layers(cfg):
    """Multiply-adds a token costs in every matrix state."""
    out = []
    for lay in cfg.get("layers", []):
        m = lay["mixer"].get("right", lay["mixer"])
        if lay["type"] in ("retention", "mlstm", "wkv"):
            out.append(2 * m["heads"] * m["dim"] * m.get("vdim", m["dim"]))
        elif lay["type"] == "parallel":
            out.append(3 * m["heads"] * m["dim"] * m["vdim"])
    return out


def _pairs(start, n, window, chunk):
    """(query, key) pairs of the tokens start .. start + n - 1."""
    if chunk:
        return sum(p % chunk + 1 for p in range(start, start + n))
    total = n * start + n * (n + 1) // 2
    if window:                                    # position p does not see its first max(0, p + 1 - window) predecessors
        last, before = max(0, start + n - window), max(0, start - window)
        total -= (last * (last + 1) - before * (before + 1)) // 2
    return total


def _step_lengths(case):
    """[(start, new tokens)] of the requests, for every step."""
    lengths = _lengths(case)
    return [lengths] + [[(c + n + j, 1) for c, n in lengths] for j in range(case["steps"])]


def work(case):
    cfg, arch, typed, spec = _spec(case)
    size = 4 if case["dtype"] == "float32" else 2
    per_token, always, expert, share = 0.0, 0, 0, 1.0
    for path, p in model_parameter_specs(spec).items():
        n = math.prod(p.shape)
        if path.startswith("embedding.") and not (spec.tie_embeddings and p.kind == "table"):
            continue                                  # a row per token is read, counted below; a tied table is the head's matrix
        if ".expert_" in path:
            expert += n
        else:
            always += n
            per_token += 0 if path.startswith(("lm_head.", "embedding.")) else n
    if expert:
        r = next(lay["mlp"]["router"] for lay in cfg["layers"] if lay["mlp"]["kind"] == "moe")
        share = min(1.0, r["top"] / (r["experts"] + r.get("identity", 0)))
        per_token += expert * share
    kv = [(n.page_elements(PAGE) / PAGE, n.window) for n in cache_needs(spec) if n.kind == "paged_kv"]
    state = sum(math.prod(n.state_shape) for n in cache_needs(spec) if n.kind == "state")
    nbytes = flops = 0.0
    for step in _step_lengths(case):
        tokens = sum(n for _, n in step)
        nbytes += size * (always + expert * (1.0 - (1.0 - share) ** tokens) + tokens * spec.width)
        nbytes += 4.0 * len(step) * (spec.vocab + 2 * state)
        nbytes += size * sum(e * (n + min(c, w or c)) for c, n in step for e, w in kv)
        flops += 2.0 * tokens * per_token + 2.0 * len(step) * spec.vocab * spec.width
        for heads, k, v, window, chunk in _attention_layers(cfg):
            flops += 2.0 * heads * (k + v) * sum(_pairs(c, n, window, chunk) for c, n in step)
        flops += 2.0 * tokens * sum(_recurrent_layers(cfg))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 5e-5}
    return {"rel": 0.03, "max": 0.25}


# ---- the same in 64 bits, whole sequences at once, plain torch --------------------------------------------------------
def _silu(z):
    return z * torch.sigmoid(z)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, inv_freq, neighbours):
    """x [T, heads, D]; the leading 2 * len(inv_freq) numbers rotate, as neighbours or as halves.  The angles are float32 by
    definition (position * inverse frequency)."""
    half = inv_freq.numel()
    a = (torch.arange(x.shape[0], dtype=torch.float32, device=x.device).view(-1, 1, 1) * inv_freq.to(x.device).float()).double()
    c, s = a.cos(), a.sin()
    out = x.clone()
    u, v = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if neighbours else (slice(0, half), slice(half, 2 * half))
    out[..., u], out[..., v] = x[..., u] * c - x[..., v] * s, x[..., v] * c + x[..., u] * s
    return out


def _frequencies(dims, base):
    return 1.0 / (float(base) ** (torch.arange(0, dims, 2).double() / dims))


def _llama_frequencies(cfg):
    D, rs = cfg["head_dim"], cfg["rope_scaling"]
    f = 1.0 / (cfg["rope_theta"] ** (torch.arange(0, D, 2).float() / D))
    if not rs:
        return f
    old, lo, hi = rs["original_max_position_embeddings"], rs["low_freq_factor"], rs["high_freq_factor"]
    wavelen = 2 * math.pi / f
    scaled = torch.where(wavelen > old / lo, f / rs["factor"], f)
    smooth = (old / wavelen - lo) / (hi - lo)
    between = (wavelen >= old / hi) & (wavelen <= old / lo)
    return torch.where(between, (1 - smooth) * scaled / rs["factor"] + smooth * scaled, scaled)


def _attend(q, k, v, scale, visible, rows=1024):
    """q [T, H, D], k [T, G, D], v [T, G, V] -> [T, H, V]; `visible(i, j)`: which keys a query sees."""
    T, H, _ = q.shape
    rep = H // k.shape[1]
    out = q.new_empty(T, H, v.shape[2])
    j = torch.arange(T, device=q.device).view(1, T)
    for h0 in range(0, H, 8):
        kk = k[:, [h // rep for h in range(h0, min(H, h0 + 8))]].permute(1, 2, 0)
        vv = v[:, [h // rep for h in range(h0, min(H, h0 + 8))]].transpose(0, 1)
        for i0 in range(0, T, rows):
            i = torch.arange(i0, min(T, i0 + rows), device=q.device).view(-1, 1)
            sc = torch.matmul(q[i0:i0 + rows, h0:h0 + 8].transpose(0, 1), kk) * scale
            sc.masked_fill_(~visible(i, j), float("-inf"))
            out[i0:i0 + rows, h0:h0 + 8] = torch.matmul(torch.softmax(sc, -1), vv).transpose(0, 1)
    return out


def _window(size):
    return lambda i, j: (j <= i) & (i - j < size) if size else j <= i


class _Plain:
    """One model in 64 bits: `hidden(tokens)` is the stream behind the final norm, [T, width]."""

    def __init__(self, case, seed):
        self.cfg, arch, _typed, spec = _spec(case)
        self.w = random_checkpoint(arch, spec, seed, dtype=torch.bfloat16, device="cuda")
        self.eps = self.cfg["norm"]["eps"] if "norm" in self.cfg else self.cfg["rms_norm_eps"]

    def __getitem__(self, name):
        return self.w[name].double()

    def mul(self, x, name):
        return x @ self[name].T

    def glu(self, h, p, names=("gate", "up", "down")):
        return self.mul(_silu(self.mul(h, p + names[0])) * self.mul(h, p + names[1]), p + names[2])

    # Llama
    def llama(self, x):
        c = self.cfg
        H, G, D, T = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], x.shape[0]
        f = _llama_frequencies(c)
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h = _rms(x, self.eps) * self[p + "input_layernorm.weight"]
            q, k, v = (self.mul(h, f"{p}self_attn.{n}_proj.weight").view(T, -1, D) for n in "qkv")
            o = _attend(_rotate(q, f, False), _rotate(k, f, False), v, D ** -0.5, _window(0))
            x = x + self.mul(o.reshape(T, H * D), p + "self_attn.o_proj.weight")
            h = _rms(x, self.eps) * self[p + "post_attention_layernorm.weight"]
            x = x + self.glu(h, p + "mlp.", names=("gate_proj.weight", "up_proj.weight", "down_proj.weight"))
        return _rms(x, self.eps) * self["model.norm.weight"]

    # Lifusun
    def conv(self, u, name):
        taps = self[name]
        n = taps.shape[1]
        u = torch.cat([u.new_zeros(n - 1, u.shape[1]), u])
        return sum(u[j:u.shape[0] - n + 1 + j] * taps[:, j] for j in range(n))

    def talking(self, h, p, m, shared):
        T, H, G, D, V = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]

        def project(n):
            return self.conv(self.mul(h, p + n) + self[p + n + ".b"], p + n + ".conv")
        q = (_rms(project("q"), self.eps) * self[p + "q.norm"]).view(T, H, D)
        if m.get("kv_from") is not None:
            k, v = shared[m["kv_from"]]
        else:
            k = (_rms(project("k"), self.eps) * self[p + "k.norm"]).view(T, G, D)
            v = _rms(project("v").view(T, G, V), self.eps)
            shared[int(p[1:p.index(".")])] = (k, v)
        k, v = k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1)
        slopes = torch.tensor([2.0 ** (-8.0 * (n + 1) / H) for n in range(H)], dtype=torch.float64, device=h.device).view(H, 1, 1)
        size, out = m["mask"]["size"], h.new_empty(T, H, V)
        for a in range(0, T, size):
            b = min(T, a + size)
            i = torch.arange(b - a, device=h.device, dtype=torch.float64)
            s = torch.einsum("ihd,jhd->hij", q[a:b], k[a:b]) * m["scale"] - slopes * (i.view(-1, 1) - i)
            s = torch.einsum("hg,gij->hij", self[p + "talk"], s).masked_fill(i > i.view(-1, 1), float("-inf"))
            out[a:b] = torch.einsum("hij,jhv->ihv", torch.softmax(s, -1), v[a:b])
        return self.mul(out.reshape(T, H * V), p + "o")

    def retention(self, h, p, m):
        T, H, D, V = h.shape[0], m["heads"], m["dim"], m["vdim"]
        f = _frequencies(m["rot"]["dims"], m["rot"]["base"])
        q, k = (_rotate(self.mul(h, p + n).view(T, H, D), f, False) for n in "qk")
        k, v = k * D ** -0.5, self.mul(h, p + "v").view(T, H, V)
        decay = torch.tensor(m["decay"], dtype=torch.float64, device=h.device).view(H, 1, 1)
        S, o = h.new_zeros(H, D, V), h.new_empty(T, H, V)
        for t in range(T):
            S = decay * S + k[t].unsqueeze(-1) * v[t].unsqueeze(-2)
            o[t] = torch.matmul(q[t].unsqueeze(1), S)[:, 0]
        return self.mul(_rms(o, self.eps).reshape(T, H * V) * _silu(self.mul(h, p + "g")), p + "o")

    def lifusun(self, x):
        shared = {}
        for i, lay in enumerate(self.cfg["layers"]):
            p, h = f"l{i}.", _rms(x, self.eps) * self[f"l{i}.norm1"]
            attention = lay["type"] == "attention"
            x = x + (self.talking(h, p + "mix.", lay["mixer"], shared) if attention else self.retention(h, p + "mix.", lay["mixer"]))
            x = x + self.glu(_rms(x, self.eps) * self[p + "norm2"], p + "mlp.")
        return _rms(x, self.eps) * self["final.norm"]

    # Rodapel
    def latent(self, h, p, m):
        T, H, D, R, V, C = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        f = _frequencies(m["rot"]["dims"], m["rot"]["base"])
        q, down = self.mul(h, p + "q").view(T, H, D + R), self.mul(h, p + "dkv")
        lat = _rms(down[:, :C], self.eps) * self[p + "dkv.norm"]
        rot = _rotate(down[:, C:].view(T, 1, R), f, True).expand(T, H, R)
        q = torch.cat([q[..., :D], _rotate(q[..., D:], f, True)], -1)
        k = torch.cat([self.mul(lat, p + "uk").view(T, H, D), rot], -1)
        return self.mul(_attend(q, k, self.mul(lat, p + "uv").view(T, H, V), m["scale"], _window(0)).reshape(T, H * V), p + "o")

    def windowed(self, h, p, m):
        T, H, G, D = h.shape[0], m["heads"], m["kv_heads"], m["dim"]
        q = _rms(self.mul(h, p + "q").view(T, H, D), self.eps) * self[p + "q.norm"]
        k = _rms(self.mul(h, p + "k").view(T, G, D), self.eps) * self[p + "k.norm"]
        o = _attend(q, k, self.mul(h, p + "v").view(T, G, -1), m["scale"], _window(m["mask"]["size"]))
        return self.mul((o * torch.sigmoid(self.mul(h, p + "g")).unsqueeze(-1)).reshape(T, -1), p + "o")

    def wkv(self, h, p, m):
        T, H, D = h.shape[0], m["heads"], m["dim"]
        before = torch.cat([h.new_zeros(1, h.shape[1]), h[:-1]])
        mix = {n: h + (before - h) * self[f"{p}mu.{n}"] for n in "rkvgw"}
        r, k, v = (self.mul(mix[n], p + n).view(T, H, D) for n in "rkv")
        decay = torch.exp(-torch.exp(self.mul(torch.tanh(self.mul(mix["w"], p + "w1")), p + "w2") + self[p + "w0"])).view(T, H, D)
        u, S, o = self[p + "u"].unsqueeze(2), h.new_zeros(H, D, D), h.new_empty(T, H, D)
        for t in range(T):
            kv = k[t].unsqueeze(2) * v[t].unsqueeze(1)
            o[t] = torch.matmul(r[t].unsqueeze(1), S + u * kv)[:, 0]
            S = decay[t].unsqueeze(2) * S + kv
        return self.mul(_rms(o, self.eps).reshape(T, H * D) * self[p + "norm"] * _silu(self.mul(mix["g"], p + "g")), p + "o")

    def clamped(self, h, p, limit):
        g, u = self.mul(h, p + "gate").clamp(max=limit), self.mul(h, p + "up").clamp(-limit, limit)
        return self.mul(g * torch.sigmoid(1.702 * g) * (u + 1.0), p + "down")

    def routed(self, h, p, weight, expert):
        """The sum of the experts' outputs; `weight` [T, experts] is zero where an expert was not chosen."""
        out = torch.zeros_like(h)
        for e in range(weight.shape[1]):
            rows = weight[:, e].nonzero()[:, 0]
            if rows.numel():
                out[rows] += weight[rows, e].unsqueeze(1) * expert(h[rows], f"{p}e{e}.")
        return out

    def best_of_all(self, h, p, mlp):
        r = mlp["router"]
        s = torch.softmax(self.mul(h, p + "router"), -1)
        chosen = torch.topk(s + self[p + "correction"], r["top"], -1).indices
        weight = torch.zeros_like(s).scatter_(1, chosen, torch.gather(s, 1, chosen))
        y = self.routed(h, p, weight[:, :r["experts"]], lambda z, q: self.clamped(z, q, mlp["expert"]["limit"]))
        return y + h * weight[:, r["experts"]:].sum(-1, keepdim=True)          # the other outputs hand the input back

    def best_of_groups(self, h, p, mlp):
        r, g = mlp["router"], mlp["router"]["groups"]
        s = torch.sigmoid(self.mul(h, p + "router"))
        T, E = s.shape
        worth = torch.topk(s.view(T, g["count"], -1), 2, -1).values.sum(-1)
        kept = torch.zeros_like(worth, dtype=torch.bool).scatter_(1, torch.topk(worth, g["keep"], -1).indices, True)
        chosen = torch.topk(s.masked_fill(~kept.repeat_interleave(E // g["count"], 1), -1.0), r["top"], -1).indices
        weight = torch.zeros_like(s).scatter_(1, chosen, torch.gather(s, 1, chosen) * r["scale"])
        return self.routed(h, p, weight, self.glu) + self.glu(h, p + "shared.")

    def rodapel(self, x):
        x = _rms(x, self.eps) * self["embed.norm"]
        kinds = {"latent_attention": self.latent, "attention": self.windowed, "wkv": self.wkv}
        for i, lay in enumerate(self.cfg["layers"]):
            p, mlp = f"l{i}.", lay["mlp"]
            x = x + _rms(kinds[lay["type"]](x, p + "mix.", lay["mixer"]), self.eps) * self[p + "norm1"]
            y = self.clamped(x, p + "mlp.", mlp["limit"]) if mlp["kind"] == "dense" else self.best_of_all(x, p + "mlp.", mlp)
            x = x + _rms(y, self.eps) * self[p + "norm2"]
        return _rms(x, self.eps) * self["final.norm"]

    # Kobolix
    def memory(self, h, p, m):
        T, H, D, V, cap = h.shape[0], m["heads"], m["dim"], m["vdim"], float(m["gate_cap"])
        q, k = (self.mul(h, p + n).view(T, H, D) for n in "qk")
        q, v = q * D ** -0.5, self.mul(h, p + "v").view(T, H, V)
        gate = [cap * torch.tanh((self.mul(h, p + n) + self[f"{p}{n}.b"]) / cap) for n in "if"]
        i, f = gate[0], torch.nn.functional.logsigmoid(gate[1])
        S, n, top, o = h.new_zeros(H, D, V), h.new_zeros(H, D), h.new_zeros(H), h.new_empty(T, H, V)
        for t in range(T):
            new = torch.maximum(f[t] + top, i[t])
            keep, add, top = torch.exp(f[t] + top - new), torch.exp(i[t] - new), new
            S = keep.view(H, 1, 1) * S + add.view(H, 1, 1) * (k[t].unsqueeze(2) * v[t].unsqueeze(1))
            n = keep.unsqueeze(1) * n + add.unsqueeze(1) * k[t]
            o[t] = torch.matmul(q[t].unsqueeze(1), S)[:, 0] / (torch.maximum((n * q[t]).sum(1).abs(), torch.exp(-top)) + 1e-6).unsqueeze(1)
        return self.mul(_rms(o, self.eps).reshape(T, H * V) * self[p + "norm"] * torch.sigmoid(self.mul(h, p + "g")), p + "o")

    def delta(self, h, p, m):
        T, H, G, D, V = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(self.conv(self.mul(h, p + n), f"{p}{n}.conv")) for n in "qkv")
        q, k = (z.view(T, G, D) / torch.sqrt((z.view(T, G, D) ** 2).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
        q, k, v = q.repeat_interleave(H // G, 1) * D ** -0.5, k.repeat_interleave(H // G, 1), v.view(T, H, V)
        beta = torch.sigmoid(self.mul(h, p + "b"))
        g = torch.exp(-torch.exp(self[p + "A_log"]) * torch.nn.functional.softplus(self.mul(h, p + "a") + self[p + "dt_bias"]))
        S, o = h.new_zeros(H, D, V), h.new_empty(T, H, V)
        for t in range(T):
            S = g[t].view(H, 1, 1) * S
            S = S + k[t].unsqueeze(2) * (beta[t].unsqueeze(1) * (v[t] - torch.matmul(k[t].unsqueeze(1), S)[:, 0])).unsqueeze(1)
            o[t] = torch.matmul(q[t].unsqueeze(1), S)[:, 0]
        o = _rms(o, self.eps) * self[p + "norm"] * _silu(self.mul(h, p + "g")).view(T, H, V)
        return self.mul(o.reshape(T, H * V), p + "o")

    def side_by_side(self, h, p, m):
        left, T = m["left"], h.shape[0]
        f = _frequencies(left["rot"]["dims"], left["rot"]["base"])
        q, k, v = (self.mul(h, f"{p}left.{n}").view(T, -1, left["dim"]) for n in "qkv")
        a = _attend(_rotate(q, f, True), _rotate(k, f, True), v, left["scale"], _window(0)).reshape(T, -1)
        a = _rms(self.mul(a, p + "left.o"), self.eps) * self[p + "left.out"]
        return 0.5 * (a + _rms(self.delta(h, p + "right.", m["right"]), self.eps) * self[p + "right.out"])

    def kobolix(self, x):
        c = self.cfg
        x = x * c["embedding"]["scale"]
        for i, lay in enumerate(c["layers"]):
            p, h = f"l{i}.", _rms(x, self.eps) * (1.0 + self[f"l{i}.norm1"])
            y = self.memory(h, p + "mix.", lay["mixer"]) if lay["type"] == "mlstm" else self.side_by_side(h, p + "mix.", lay["mixer"])
            x = x + c["residual_mult"] * y
            h, mlp = _rms(x, self.eps) * (1.0 + self[p + "norm2"]), lay["mlp"]
            x = x + c["residual_mult"] * (self.glu(h, p + "mlp.") if mlp["kind"] == "dense" else self.best_of_groups(h, p + "mlp.", mlp))
        return _rms(x, self.eps) * (1.0 + self["final.norm"])

    def rows(self, tokens, places):
        """Logits at `places` of one sequence."""
        name = self.cfg.get("architecture", "Llama").lower()
        table = self.w["model.embed_tokens.weight" if name == "llama" else "embed"]
        x = table[torch.tensor(tokens, device=table.device)].double()
        x = getattr(self, name)(x)[places]
        head = self.w.get("lm_head.weight", self.w.get("head", table))
        return torch.cat([x @ head[a:a + 16384].double().T for a in range(0, head.shape[0], 16384)], -1)


def exact(case, seed):
    lengths = _lengths(case)
    cost = work(case)["flops"] / sum(n for _, n in _lengths(case)) * sum(c + n for c, n in lengths)
    if cost > EXACT_FLOPS:
        return None
    model = _Plain(case, seed)
    vocab = _spec(case)[3].vocab
    out = [torch.empty(len(lengths), vocab, dtype=torch.float64, device="cuda") for _ in range(case["steps"] + 1)]
    for r, (tokens, (c, n)) in enumerate(zip(_tokens(case, vocab, seed), lengths)):
        last = c + n - 1
        for j, row in enumerate(model.rows(tokens, list(range(last, last + case["steps"] + 1)))):
            out[j][r] = row
    return out
