"""What this framework is measured on: requests served by its models, and the draw of their tokens.

A case is one of two things.

* ``requests``: sequences are opened, their prompts run in one step, then ``new`` tokens are fed to each of them one
  step at a time, and the sequences are closed again: ``Model.open_sequence``, ``Model.step``, ``Model.close_sequence``,
  which the generation loop, scoring and trace replay are made of.  The tokens are given (as in replay and scoring), so
  that the logits of every step can be compared.  ``new`` 0 is a prompt step alone.
* ``sample``: a step's logits become tokens (``Sampler``), a row per live sequence.

Models: the Llama presets, and the Sotavik, Ronelorn and Vufadra designs at the two widths at which ``bench.py`` measures
them: full and windowed softmax attention, latent attention, linear and gated recurrences, dense feed-forwards and experts.
"""
from __future__ import annotations

import math
import random

import torch

from supersonic_b200.api import Engine
from supersonic_b200.config import config_from_dict, preset_config
from supersonic_b200.csrc.kernel_sets import kernel_set_for
from supersonic_b200.engine import Model, StepEntry
from supersonic_b200.sampling import Sampler, SamplingParams, request_seed
from supersonic_b200.weights import WeightStore

DEVICE = "cuda:0"
PAGE = 64


# ---- models -------------------------------------------------------------------------------------------------------
def _sotavik(width):
    def latent(heads, dim, rot, vdim, rank):
        return {"type": "latent_attention", "mixer": {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "kv_rank": rank,
                "rot": {"base": 10000.0, "dims": rot}, "scale": (dim + rot) ** -0.5}}

    def gla(heads, dim, vdim):
        return {"type": "gla", "mixer": {"heads": heads, "dim": dim, "vdim": vdim, "tau": 16.0, "decay_rank": 16}}
    if width == 2048:
        mixers = [latent(16, 128, 64, 128, 512)] * 2 + [gla(4, 256, 512), latent(16, 128, 64, 128, 512)]
        mlp = {"experts": 64, "top": 6, "ff": 1408, "shared": 2816}
    else:
        mixers = [latent(8, 64, 32, 64, 256), gla(4, 128, 256)] * 2
        mlp = {"experts": 16, "top": 2, "ff": 512, "shared": 1024}
    moe = {"kind": "moe", "expert": {"ff": mlp["ff"]}, "router": {"experts": mlp["experts"], "top": mlp["top"]},
           "shared": {"ff": mlp["shared"]}}
    return {"architecture": "Sotavik", "vocab": 32000, "width": width, "logit_scale": 1.0, "norm": {"eps": 1e-5},
            "layers": [dict(m, mlp=moe) for m in mixers]}


def _vufadra(width):
    def pair(heads, kv, dim, chunk, r_heads, r_dim):
        return {"type": "parallel", "mixer": {
            "left": {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "mask": {"size": chunk}, "scale": dim ** -0.5,
                     "rot": {"base": 10000.0, "dims": dim // 2,
                             "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}},
            "right": {"heads": r_heads, "dim": r_dim, "decay_rank": 64}}}
    n = width // 128
    delta = {"type": "general_delta", "mixer": {"heads": 2 * n, "dim": 64, "decay_rank": 64}}
    mixers = [{"type": "rglru", "mixer": {"width": width, "conv": 4, "blocks": n}}, delta,
              pair(n, n // 4, 128, width // 4, 2 * n, 64), delta]
    return {"architecture": "Vufadra", "vocab": 32000, "width": width, "norm": {"eps": 1e-5},
            "embedding": {"bigram": {"buckets": 65521, "mul_prev": 31337, "mul_cur": 7919}},
            "loop": {"start": 0, "stop": 4, "times": 1},
            "layers": [dict(m, mlp={"kind": "dense", "ff": 4 * width}) for m in mixers]}


def _ronelorn(width):
    n = width // 128
    pooled = {"type": "attention", "mixer": {
        "heads": n, "kv_heads": n // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0,
        "mask": {"size": width // 4, "pool": 16}, "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 2.0}}}}
    kept = {"type": "attention_2", "mixer": {
        "heads": 2 * n, "kv_heads": n // 2, "dim": 64, "vdim": 64, "scale": 64 ** -0.5,
        "mask": {"size": width // 4, "keep_first": 4}, "rot": {"base": 10000.0, "dims": 32}}}
    layers = [dict(m, mlp={"kind": "dense", "ff": 4 * width})
              for m in (pooled, kept, {"type": "mingru", "mixer": {"width": width}})]
    layers.append(dict(layers[0], weights_of=0))
    return {"architecture": "Ronelorn", "vocab": 32000, "width": width, "norm": {"eps": 1e-5},
            "embedding": {"scale": float(width) ** 0.5}, "residual_mult": 0.5, "layers": layers}


_DESIGNS = {"sotavik": _sotavik, "vufadra": _vufadra, "ronelorn": _ronelorn}


def _config(name):
    """``llama3.1-8b`` and the like (a preset), or ``sotavik-2048``: a design and its width."""
    design, _, width = name.rpartition("-")
    return config_from_dict(_DESIGNS[design](int(width))) if design in _DESIGNS else preset_config(name)


def _tensor(name, shape, architecture, layers, g):
    """One weight: matrices N(0, 0.02) (those that write into a deep stream smaller by the root of the sublayers, as models
    are initialised), norm weights near one, and for what is neither, values of the size it has in use (biases and decays of
    order one, shares between 0 and 1, and an embedding of order one where a deep stream has to carry it)."""
    def normal(std=1.0, mean=0.0):
        return torch.empty(shape, dtype=torch.bfloat16, device=DEVICE).normal_(mean, std, generator=g)
    last = name.rsplit(".", 1)[-1]
    if last == "table":
        experts = 64 if shape[1] > 2 else 16
        order = torch.rand(shape[0], experts, device=DEVICE, generator=g).argsort(dim=1)
        return order[:, : shape[1]].to(torch.int32).contiguous()
    if last == "dwa":
        return normal(0.5 / shape[0], 1.0 / shape[0])
    if last == "alpha":
        return (0.5 + 0.5 * torch.rand(shape, device=DEVICE, generator=g)).to(torch.bfloat16)
    if last == "shift" or ".mu." in name:
        return torch.rand(shape, device=DEVICE, generator=g).to(torch.bfloat16)
    if last == "sink":
        return normal()
    if name.endswith(".a2.b"):
        return normal(1.0, 1.0)
    if last == "lam":
        return normal(1.0, -2.0)
    if architecture == "Vufadra" and last == "b" and "norm" in name:
        return normal(0.1)
    if architecture == "Vufadra" and name in ("embed", "bigram") or name.startswith("model.embed"):
        return normal(0.5)
    if last in ("b", "pb", "w0"):
        return normal(0.5)
    if last in ("u", "step"):
        return normal(0.3)
    if last in ("conv", "ra", "ri"):
        return normal(shape[-1] ** -0.5)
    if architecture == "Ronelorn" and (last in ("norm1", "norm2") or name == "final.norm"):
        return normal(0.1)                                      # stored around zero
    if "norm" in name or last == "out":
        return normal(0.1, 1.0)
    if name.endswith(("o_proj.weight", "down_proj.weight")):
        return normal(0.02 / (2 * layers) ** 0.5)
    return normal(0.02)


def _weights(cfg, seed):
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    architecture = list(cfg.architectures)[0]
    layers = cfg.num_hidden_layers
    return {name: _tensor(name, list(shape), architecture, layers, g) for name, shape in sorted(cfg.tensor_shapes().items())}


# ---- cases --------------------------------------------------------------------------------------------------------
def _requests(name, model, seqs, shortest, longest, new, dtype="bfloat16"):
    return {"name": name, "kind": "requests", "model": model, "dtype": dtype, "seqs": seqs, "shortest": shortest,
            "longest": longest, "new": new}


def listed():
    return [
        # one user's short question answered by a small model: every launch of a step counts
        _requests("reply-1b", "llama3.2-1b", 1, 23, 23, 32),
        # the headline workload: eight sequences at 8B sizes
        _requests("batch8-8b", "llama3.1-8b", 8, 512, 512, 24),
        # a full server: many sequences of very unequal lengths
        _requests("batch64-1b", "llama3.2-1b", 64, 1, 512, 24),
        # one long prompt at 8B sizes: matrix products at their widest
        _requests("prompt-8b", "llama3.1-8b", 1, 2048, 2048, 0),
        # sixteen prompts that start together, lengths as they come
        _requests("prompts-3b", "llama3.2-3b", 16, 64, 2048, 0),
        # the time to a first token of a short prompt
        _requests("prompt-short-1b", "llama3.2-1b", 1, 131, 131, 0),
        # the float32 path (replay against which others are checked): prompts, and tokens one by one
        _requests("prompts-1b-float32", "llama3.2-1b", 3, 100, 500, 0, "float32"),
        _requests("reply-1b-float32", "llama3.2-1b", 2, 19, 45, 12, "float32"),
        # the other designs: a long prompt, short replies to a batch of prompts, two prompts and a reply
        _requests("prompt-sotavik", "sotavik-2048", 1, 2048, 2048, 0),
        _requests("batch8-ronelorn", "ronelorn-2048", 8, 100, 1500, 24),
        _requests("reply-vufadra", "vufadra-2048", 2, 300, 1100, 16),
        # the draw of a step's tokens for a full server with both cuts on
        {"name": "sample-64", "kind": "sample", "rows": 64, "vocab": 128256, "temperature": 0.7, "top_k": 40, "top_p": 0.9},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


# prompt tokens of a step, and sequences times new tokens, that cost no more than the largest listed case
_MOST_TOKENS = {"llama3.1-8b": 2048, "llama3.2-3b": 12000, "llama3.2-1b": 16384}
_MOST_TOKENS_FLOAT32 = {"llama3.2-1b": 600}


def draw(rng):
    if rng.random() < 0.08:
        return {"kind": "sample", "rows": _log_int(rng, 1, 64), "vocab": rng.choice([32000, 128256]),
                "temperature": rng.choice([0.0, 0.7, 1.0]), "top_k": rng.choice([0, 0, 20, 40]),
                "top_p": rng.choice([1.0, 0.9, 0.95])}
    model = rng.choice(["llama3.2-1b"] * 4 + ["llama3.2-3b"] * 2 + ["llama3.1-8b"] * 2
                       + [f"{d}-{w}" for d in ("sotavik", "ronelorn", "vufadra") for w in (1024, 2048)])
    dtype = "float32" if model.endswith(("-1b", "-1024")) and rng.random() < 0.3 else "bfloat16"
    most = _MOST_TOKENS.get(model, 8192)
    if dtype == "float32":
        most = _MOST_TOKENS_FLOAT32.get(model, 2048)
    seqs = min(_log_int(rng, 1, 64), most // 8)
    longest = _log_int(rng, 8, min(4096, most // seqs))
    shortest = longest if rng.random() < 0.3 else _log_int(rng, 1, longest)
    new = 0 if rng.random() < 0.45 else rng.randint(4, 8 if dtype == "float32" else 20)
    case = _requests("", model, seqs, shortest, longest, new, dtype)
    del case["name"]
    return case


def _lengths(case):
    """The prompts' lengths: part of the case, not of its seed."""
    rng = random.Random(f"{case['seqs']} {case['shortest']} {case['longest']}")
    return [rng.randint(case["shortest"], case["longest"]) for _ in range(case["seqs"])]


def _tokens(case, seed, vocab):
    """(prompts, the token fed to every sequence in every later step)."""
    g = torch.Generator().manual_seed(seed + 1)
    prompts = [torch.randint(0, vocab, (n,), generator=g).tolist() for n in _lengths(case)]
    return prompts, torch.randint(0, vocab, (case["new"], case["seqs"]), generator=g).tolist()


# ---- what a user's program holds, and one pass --------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "sample":
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        rows = case["rows"]
        state = [request_seed(seed, r) for r in range(rows)]
        state = torch.tensor([s - (1 << 64) if s >> 63 else s for s in state], dtype=torch.int64, device=DEVICE)
        return {"logits": 2.5 * torch.randn(rows, case["vocab"], device=DEVICE, generator=g), "rng": state,
                "slots": torch.arange(rows, dtype=torch.int32, device=DEVICE),
                "sampler": Sampler(kernel_set_for(torch.bfloat16), state),
                "params": SamplingParams(case["temperature"], case["top_k"], case["top_p"], seed % 1000)}
    cfg = _config(case["model"])
    room = [n + case["new"] for n in _lengths(case)]
    most = -(-max(room) // PAGE) * PAGE
    engine = Engine(Model.from_config(cfg, WeightStore.from_tensors(_weights(cfg, seed)), dtype=case["dtype"], device=DEVICE,
                                      max_tokens=sum(-(-n // PAGE) * PAGE for n in room), max_seq_tokens=most,
                                      max_slots=case["seqs"]))
    prompts, fed = _tokens(case, seed, cfg.vocab_size)
    state = {"engine": engine, "prompts": prompts, "fed": fed}
    run(state)                     # a server's first request: it loads kernels and captures the decode steps of this size
    return state


def run(state):
    if "sampler" in state:
        return [state["sampler"](state["logits"], state["slots"], state["params"]), state["rng"]]
    model = state["engine"].model
    slots = [model.open_sequence() for _ in state["prompts"]]
    try:
        logits = [model.step([StepEntry(s, p, [len(p) - 1]) for s, p in zip(slots, state["prompts"])])]
        for tokens in state["fed"]:
            logits.append(model.step([StepEntry(s, [t], [0]) for s, t in zip(slots, tokens)]))
        return logits
    finally:
        for s in slots:
            model.close_sequence(s)


# ---- what a pass cannot do without --------------------------------------------------------------------------------
def _matrices(cfg):
    """(elements of the matrices every token passes, elements of one expert's matrices summed over layers, the router)."""
    shared = one = 0
    for name, shape in cfg.tensor_shapes().items():
        if len(shape) < 2 or name in ("embed", "bigram", "head") or name.endswith((".table", ".pb", ".u", ".step")) \
                or name.startswith(("model.embed", "lm_head")):
            continue
        n = math.prod(shape)
        if ".mlp.e" in name:
            one += n if ".mlp.e0." in name else 0
        else:
            shared += n
    layers = getattr(cfg, "layers", None)
    router = (layers[0].get("mlp") or {}).get("router") if layers else None
    if layers:                     # a layer that runs with another's tensors computes with them again
        for i, layer in enumerate(layers):
            if layer.get("weights_of") is not None:
                p = f"l{layer['weights_of']}."
                shared += sum(math.prod(s) for n, s in cfg.tensor_shapes().items() if n.startswith(p) and len(s) > 1)
    return shared, one, router


def _pairs(n, window):
    full = n * (n + 1) // 2
    return full if not window or n <= window else window * (window + 1) // 2 + (n - window) * window


def _attention(cfg, n):
    """(FLOPs of the mixers beyond their matrices for a sequence of n tokens, values of cache or state it leaves)."""
    flops = values = 0
    if getattr(cfg, "layers", None) is None:
        d = cfg.head_dim
        return (cfg.num_hidden_layers * 4 * _pairs(n, None) * cfg.num_attention_heads * d,
                cfg.num_hidden_layers * 2 * n * cfg.num_key_value_heads * d)
    for layer in cfg.layers:
        m, kind = layer["mixer"], layer["type"]
        if kind == "parallel":
            right, m = m["right"], m["left"]
            flops += 6 * n * right["heads"] * right["dim"] ** 2
            values += right["heads"] * right["dim"] ** 2
        if kind == "latent_attention":
            flops += 2 * _pairs(n, None) * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
            values += n * (m["kv_rank"] + m["rot_dim"])
        elif kind == "gla":
            flops += 4 * n * m["heads"] * m["dim"] * m["vdim"]
            values += m["heads"] * m["dim"] * m["vdim"]
        elif kind == "general_delta":
            flops += 8 * n * m["heads"] * m["dim"] ** 2
            values += m["heads"] * m["dim"] ** 2
        elif kind in ("rglru", "mingru"):
            flops += 12 * n * m["width"]
            values += m["width"]
        else:
            window = m["mask"]["size"]
            flops += 2 * _pairs(n, window) * m["heads"] * (m["dim"] + m["vdim"])
            values += min(n, window) * m["kv_heads"] * (m["dim"] + m["vdim"])
    return flops, values


def work(case):
    if case["kind"] == "sample":
        n = case["rows"] * case["vocab"]
        return {"bytes": 4 * n, "flops": 2 * n}
    cfg = _config(case["model"])
    item = 4 if case["dtype"] == "float32" else 2
    lengths, new, vocab, width = _lengths(case), case["new"], cfg.vocab_size, cfg.hidden_size
    shared, one, router = _matrices(cfg)
    head = vocab * width
    nbytes = flops = 0
    for step in range(new + 1):
        tokens = sum(lengths) if step == 0 else len(lengths)
        flops += 2 * tokens * shared + 2 * len(lengths) * head
        nbytes += item * (shared + head + tokens * width) + 4 * len(lengths) * vocab
        if router:
            used = 1.0 - (1.0 - router["top"] / router["experts"]) ** tokens          # the share of experts some token picks
            flops += 2 * tokens * router["top"] * one
            nbytes += item * one * router["experts"] * used
        for n in lengths:
            f, v = _attention(cfg, n + step)
            f0 = _attention(cfg, n + step - 1)[0] if step else 0
            flops += f - f0
            nbytes += item * v
    return {"bytes": int(nbytes), "flops": int(flops)}


def tolerance(case):
    """Measured: two runs of one bfloat16 case differ by up to 1 % (float atomics: sums in another order), 5.5 % of the root
    mean square at the worst logit, and lie up to 1.1 % from the 64-bit result; a float32 one lies 3.5e-7 from it."""
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 5e-6, "max": 1e-4}
    return {"rel": 0.03, "max": 0.3}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------
F = torch.float64


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


class _Exact:
    """A model's forward pass over padded sequences [B, T] (what follows a sequence's end cannot change it)."""

    def __init__(self, cfg, weights, tokens, lengths):
        self.cfg, self.weights, self.tokens, self.lengths = cfg, weights, tokens, lengths
        self.B, self.T = tokens.shape

    def w(self, name):
        return self.weights[name].to(F)

    def lin(self, x, name):
        return x @ self.w(name).T

    def heads(self, x, n):
        return x.view(self.B, self.T, n, -1)

    def turn(self, x, freq, interleaved=False, back=False, gain=1.0):
        """x [B, T, heads, d]: pairs of the first 2 * len(freq) coordinates turned by the token's position."""
        half = freq.numel()
        ang = torch.arange(self.T, dtype=F, device=DEVICE)[:, None] * freq[None, :]
        c, s = (ang.cos() * gain)[None, :, None, :], (ang.sin() * gain)[None, :, None, :]
        s = -s if back else s
        out = x.clone()
        a = x[..., 0:2 * half:2] if interleaved else x[..., :half]
        b = x[..., 1:2 * half:2] if interleaved else x[..., half:2 * half]
        if interleaved:
            out[..., 0:2 * half:2], out[..., 1:2 * half:2] = a * c - b * s, b * c + a * s
        else:
            out[..., :half], out[..., half:2 * half] = a * c - b * s, b * c + a * s
        return out

    def freq(self, dims, base):
        return base ** (-torch.arange(0, dims, 2, dtype=F, device=DEVICE) / dims)

    def attend(self, q, k, v, score_to_weight, mask):
        """q [B, T, H, D], k [B, S, G, D], v [B, S, G, V]: a sequence and a kv head at a time; ``mask`` [T, S]."""
        H, G = q.shape[2], k.shape[2]
        out = torch.zeros(self.B, self.T, H, v.shape[-1], dtype=F, device=DEVICE)
        for b in range(self.B):
            n = self.lengths[b]
            for g in range(G):
                for h in range(g * (H // G), (g + 1) * (H // G)):
                    out[b, :n, h] = score_to_weight(q[b, :n, h] @ k[b, :, g].T, mask[:n], h) @ v[b, :, g]
        return out.reshape(self.B, self.T, -1)

    def causal(self, window=None, keep=0):
        i = torch.arange(self.T, device=DEVICE)
        back = i[:, None] - i[None, :]
        seen = back >= 0
        return seen if window is None else seen & ((back < window) | (i[None, :] < keep))

    def softmax(self, scale, cap=None, sink=None):
        def weights(s, mask, h):
            s = s * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill(~mask, -math.inf)
            top = s.max(-1, keepdim=True).values
            if sink is not None:
                top = top.clamp(min=float(sink[h]))
            e = torch.exp(s - top)
            return e / (e.sum(-1, keepdim=True) + (torch.exp(sink[h] - top) if sink is not None else 0.0))
        return weights

    # -- Llama
    def llama(self):
        c = self.cfg
        freq = self.freq(c.head_dim, c.rope_theta)
        if c.rope_scaling is not None:
            r = c.rope_scaling
            old, wave = float(r.original_max_position_embeddings), 2.0 * math.pi / freq
            mid = (old / wave - r.low_freq_factor) / (r.high_freq_factor - r.low_freq_factor)
            freq = freq * ((1.0 - mid.clamp(0.0, 1.0)) / r.factor + mid.clamp(0.0, 1.0))
        x = self.w("model.embed_tokens.weight")[self.tokens]
        for i in range(c.num_hidden_layers):
            p = f"model.layers.{i}."
            h = _rms(x, c.rms_norm_eps) * self.w(p + "input_layernorm.weight")
            q = self.turn(self.heads(self.lin(h, p + "self_attn.q_proj.weight"), c.num_attention_heads), freq)
            k = self.turn(self.heads(self.lin(h, p + "self_attn.k_proj.weight"), c.num_key_value_heads), freq)
            v = self.heads(self.lin(h, p + "self_attn.v_proj.weight"), c.num_key_value_heads)
            o = self.attend(q, k, v, self.softmax(c.head_dim ** -0.5), self.causal())
            x = x + self.lin(o, p + "self_attn.o_proj.weight")
            h = _rms(x, c.rms_norm_eps) * self.w(p + "post_attention_layernorm.weight")
            x = x + self.lin(_silu(self.lin(h, p + "mlp.gate_proj.weight")) * self.lin(h, p + "mlp.up_proj.weight"),
                             p + "mlp.down_proj.weight")
        head = "model.embed_tokens.weight" if c.tie_word_embeddings else "lm_head.weight"
        return _rms(x, c.rms_norm_eps) * self.w("model.norm.weight"), head

    # -- Sotavik
    def latent(self, h, p, m, eps):
        H, d, r, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        freq = self.freq(m["rot"]["dims"], m["rot"]["base"])
        q = self.heads(self.lin(h, p + ".q"), H)
        q = torch.cat([q[..., :d], self.turn(q[..., d:], freq, True)], -1)
        low = self.lin(h, p + ".dkv")
        c = _rms(low[..., :rank], eps) * self.w(p + ".dkv.norm")
        turned = self.turn(low[:, :, None, rank:], freq, True).expand(-1, -1, H, -1)
        k = torch.cat([self.heads(self.lin(c, p + ".uk"), H), turned], -1)
        v = self.heads(self.lin(c, p + ".uv"), H)
        return self.lin(self.attend(q, k, v, self.softmax(m["scale"], sink=self.w(p + ".sink")), self.causal()), p + ".o")

    def gla(self, h, p, m, eps):
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        q, k, v = (self.heads(self.lin(h, f"{p}.{r}"), H) for r in "qkv")
        z = self.lin(self.lin(h, p + ".a1"), p + ".a2") + self.w(p + ".a2.b")
        decay = self.heads(torch.sigmoid(z) ** (1.0 / m["tau"]), H)
        S = torch.zeros(self.B, H, d, dv, dtype=F, device=DEVICE)
        o = torch.empty(self.B, self.T, H, dv, dtype=F, device=DEVICE)
        for t in range(self.T):
            S = decay[:, t, :, :, None] * S + k[:, t, :, :, None] * v[:, t, :, None, :]
            o[:, t] = (q[:, t, :, None, :] @ S)[..., 0, :] * d ** -0.5
        o = _rms(o, eps) * self.w(p + ".norm")
        return self.lin(o.reshape(self.B, self.T, -1) * _silu(self.lin(h, p + ".g")), p + ".o")

    def gated(self, h, p):
        return (_silu(h @ self.w(p + ".gate").T) * (h @ self.w(p + ".up").T)) @ self.w(p + ".down").T

    def sotavik(self):
        c, eps = self.cfg, self.cfg.norm_eps
        x = self.w("embed")[self.tokens]
        results = [x]
        for i, layer in enumerate(c.layers):
            p = f"l{i}"
            h = _rms(x, eps) * self.w(p + ".norm1")
            mixer = self.latent if layer["type"] == "latent_attention" else self.gla
            y = x + mixer(h, p + ".mix", layer["mixer"], eps) + self.gated(h, p + ".mlp.shared")
            picks = self.weights[p + ".mlp.table"].long()[self.tokens]
            for e in range(layer["mlp"]["router"]["experts"]):
                b, t = (picks == e).any(-1).nonzero(as_tuple=True)
                y[b, t] += self.gated(h[b, t], f"{p}.mlp.e{e}") / picks.shape[-1]
            results.append(y)
            mix = self.w(p + ".dwa")
            x = sum(mix[j] * r for j, r in enumerate(results))
        return _rms(x, eps) * self.w("final.norm") * c.logit_scale, "head"

    # -- Ronelorn
    def windowed(self, h, p, m, eps, whole):
        H, G, D, V, rot, mask = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["rot"], m["mask"]
        q, k, v = self.lin(h, p + ".q"), self.lin(h, p + ".k"), self.heads(self.lin(h, p + ".v"), G)
        if whole:
            q, k = _rms(q, eps) * self.w(p + ".q.norm"), _rms(k, eps) * self.w(p + ".k.norm")
        q, k = self.heads(q, H), self.heads(k, G)
        if not whole:
            q, k = _rms(q, eps) * self.w(p + ".q.norm"), _rms(k, eps) * self.w(p + ".k.norm")
        freq = self.freq(rot["dims"], rot["base"]) / (rot.get("scaling") or {}).get("factor", 1.0)
        q, k = self.turn(q, freq), self.turn(k, freq)
        seen = self.causal(mask["size"], mask.get("keep_first") or 0)
        if whole:
            o = self.attend(q, k, v, self.softmax(m["scale"], sink=torch.zeros(H, dtype=F, device=DEVICE)), seen)
            return self.lin(o, p + ".o")
        v = self.turn(v, self.freq(V, rot["base"]))
        pool = mask["pool"]
        runs = self.T // pool
        kp = k[:, : runs * pool].view(self.B, runs, pool, G, D).mean(2)
        vp = v[:, : runs * pool].view(self.B, runs, pool, G, V).mean(2)
        i, b = torch.arange(self.T, device=DEVICE), torch.arange(runs, device=DEVICE)
        seen = torch.cat([b[None, :] * pool + pool - 1 <= i[:, None] - mask["size"], seen], 1)
        o = self.attend(q, torch.cat([kp, k], 1), torch.cat([vp, v], 1), self.softmax(m["scale"], m.get("softcap")), seen)
        o = self.turn(self.heads(o, H), self.freq(V, rot["base"]), back=True)
        return self.lin(o.reshape(self.B, self.T, -1), p + ".o")

    def scan(self, keep, drive):
        S, out = torch.zeros_like(drive[:, 0]), torch.empty_like(drive)
        for t in range(self.T):
            S = keep[:, t] * S + drive[:, t]
            out[:, t] = S
        return out

    def mingru(self, h, p):
        z = torch.sigmoid(self.lin(h, p + ".z") + self.w(p + ".z.b"))
        u = self.lin(h, p + ".x") + self.w(p + ".x.b")
        state = self.scan(1.0 - z, z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u)))
        return self.lin(state * _silu(self.lin(h, p + ".g")), p + ".o")

    def ronelorn(self):
        d = self.cfg.to_dict()
        eps, mult = d["norm"]["eps"], d["residual_mult"]
        x = self.w("embed")[self.tokens] * d["embedding"]["scale"]
        for i, layer in enumerate(d["layers"]):
            p = f"l{i if layer.get('weights_of') is None else layer['weights_of']}"
            h = _rms(x, eps) * (1.0 + self.w(p + ".norm1"))
            if layer["type"] == "mingru":
                y = self.mingru(h, p + ".mix")
            else:
                y = self.windowed(h, p + ".mix", layer["mixer"], eps, layer["type"] == "attention_2")
            x = x + mult * y
            h = _rms(x, eps) * (1.0 + self.w(p + ".norm2"))
            x = x + mult * self.lin(self.lin(h, p + ".mlp.up").clamp(min=0) ** 2, p + ".mlp.down")
        return _rms(x, eps) * (1.0 + self.w("final.norm")), "head"

    # -- Vufadra
    def tanh_norm(self, x, name):
        return torch.tanh(self.w(name + ".alpha") * x) * self.w(name) + self.w(name + ".b")

    def shifted(self, h, mu):
        return h + (torch.cat([torch.zeros_like(h[:, :1]), h[:, :-1]], 1) - h) * mu

    def rglru(self, h, p, m):
        C, taps, nb = m["width"], m["conv"], m["blocks"]
        y = torch.nn.functional.gelu(self.lin(h, p + ".y") + self.w(p + ".y.b"), approximate="tanh")
        xb = self.lin(h, p + ".x") + self.w(p + ".x.b")
        padded = torch.cat([torch.zeros(self.B, taps - 1, C, dtype=F, device=DEVICE), xb], 1)
        u = self.w(p + ".conv.b") + sum(padded[:, j:j + self.T] * self.w(p + ".conv")[:, j] for j in range(taps))
        ub = u.view(self.B, self.T, nb, -1)
        r, i = (torch.sigmoid(torch.einsum("noi,btni->btno", self.w(f"{p}.{g}"), ub) + self.w(f"{p}.{g}.b")).reshape(u.shape)
                for g in ("ra", "ri"))
        a = torch.exp(-8.0 * r * torch.nn.functional.softplus(self.w(p + ".lam")))
        return self.lin(self.scan(a, torch.sqrt(1.0 - a * a) * i * u) * y, p + ".o")

    def matrix_state(self, r, k, v, decay, unit=None, removal=None, bonus=None):
        S = torch.zeros(self.B, r.shape[2], r.shape[3], v.shape[3], dtype=F, device=DEVICE)
        o = torch.empty_like(v)
        for t in range(self.T):
            kv = k[:, t, :, :, None] * v[:, t, :, None, :]
            if bonus is not None:
                o[:, t] = (r[:, t, :, None, :] @ (S + bonus[:, :, None] * kv))[..., 0, :]
            seen = unit[:, t, :, None, :] @ S if unit is not None else None
            S = decay[:, t, :, :, None] * S + kv
            if unit is not None:
                S = S - removal[:, t, :, :, None] * seen
                o[:, t] = (r[:, t, :, None, :] @ S)[..., 0, :]
        return o

    def delta(self, h, p, m, eps):
        H = m["heads"]
        r, k, v = (self.heads(self.lin(h, f"{p}.{n}"), H) for n in "rkv")
        z = self.lin(torch.tanh(self.lin(h, p + ".w1")), p + ".w2") + self.w(p + ".w0")
        decay = self.heads(torch.exp(-math.exp(-0.5) * torch.sigmoid(z)), H)
        a = self.heads(torch.sigmoid(self.lin(h, p + ".a") + self.w(p + ".a.b")), H)
        u = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        o = _rms(self.matrix_state(r, k, v, decay, unit=u, removal=a * u), eps)
        o = o.reshape(self.B, self.T, -1) * self.w(p + ".norm") * torch.sigmoid(self.lin(h, p + ".g"))
        return self.lin(o, p + ".o")

    def chunked(self, h, p, m, eps):
        H, G, rot = m["heads"], m["kv_heads"], m["rot"]
        dims, base, sc = rot["dims"], rot["base"], rot["scaling"]

        def at(turns):
            return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
        ramp = ((torch.arange(dims // 2, dtype=F, device=DEVICE) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        freq = self.freq(dims, base) * (ramp / sc["factor"] + 1.0 - ramp)
        gain = 0.1 * math.log(sc["factor"]) + 1.0
        q = self.turn(_rms(self.heads(self.lin(h, p + ".q"), H), eps) * self.w(p + ".q.norm"), freq, gain=gain)
        k = self.turn(_rms(self.heads(self.lin(h, p + ".k"), G), eps) * self.w(p + ".k.norm"), freq, gain=gain)
        i = torch.arange(self.T, device=DEVICE) // m["mask"]["size"]
        pb, scale = self.w(p + ".pb"), m["scale"]
        o = self.attend(q, k, self.heads(self.lin(h, p + ".v"), G),
                        lambda s, mask, head: torch.sigmoid(s * scale + pb[head]) * mask, self.causal() & (i[:, None] == i[None, :]))
        return self.lin(o, p + ".o")

    def time_mixing(self, h, p, m, eps):
        H = m["heads"]
        mix = {s: self.shifted(h, self.w(f"{p}.mu.{s}")) for s in "rkvgw"}
        r, k, v = (self.heads(self.lin(mix[n], f"{p}.{n}"), H) for n in "rkv")
        z = self.lin(torch.tanh(self.lin(mix["w"], p + ".w1")), p + ".w2") + self.w(p + ".w0")
        o = _rms(self.matrix_state(r, k, v, self.heads(torch.exp(-torch.exp(z)), H), bonus=self.w(p + ".u")), eps)
        o = o.reshape(self.B, self.T, -1) * self.w(p + ".norm") * _silu(self.lin(mix["g"], p + ".g"))
        return self.lin(o, p + ".o")

    def vufadra(self):
        d = self.cfg.to_dict()
        eps, big = d["norm"]["eps"], d["embedding"]["bigram"]
        rows = torch.full_like(self.tokens, big["buckets"])
        rows[:, 1:] = (self.tokens[:, :-1] * big["mul_prev"] + self.tokens[:, 1:] * big["mul_cur"]) % big["buckets"]
        x0 = self.w("embed")[self.tokens] + self.w("bigram")[rows]
        x = self.lin(torch.cat([x0, x0], -1), "loop.in") + self.w("loop.step")[0]      # the loop over all layers, walked once
        for i, layer in enumerate(d["layers"]):
            p, m = f"l{i}", layer["mixer"]
            h = self.shifted(self.tanh_norm(x, p + ".norm1"), self.w(p + ".shift"))
            if layer["type"] == "rglru":
                y = self.rglru(h, p + ".mix", m)
            elif layer["type"] == "general_delta":
                y = self.delta(h, p + ".mix", m, eps)
            else:
                left = self.chunked(h, p + ".mix.left", m["left"], eps)
                right = self.time_mixing(h, p + ".mix.right", m["right"], eps)
                y = 0.5 * (_rms(left, eps) * self.w(p + ".mix.left.out") + _rms(right, eps) * self.w(p + ".mix.right.out"))
            x = x + y + self.gated(self.tanh_norm(x, p + ".norm2"), p + ".mlp")
        return self.tanh_norm(x, "final.norm"), "head"


def exact(case, seed):
    if case["kind"] == "sample":
        return None                # tokens drawn by integer weights: whole numbers
    cfg = _config(case["model"])
    weights = _weights(cfg, seed)
    prompts, fed = _tokens(case, seed, cfg.vocab_size)
    whole = [p + [step[i] for step in fed] for i, p in enumerate(prompts)]
    T = max(len(s) for s in whole)
    tokens = torch.tensor([s + [0] * (T - len(s)) for s in whole], dtype=torch.int64, device=DEVICE)
    model = _Exact(cfg, weights, tokens, [len(s) for s in whole])
    design = case["model"].split("-")[0]
    hidden, head = (getattr(model, design) if design in _DESIGNS else model.llama)()
    last = torch.tensor([len(p) - 1 for p in prompts], device=DEVICE)
    rows = [hidden[torch.arange(len(prompts), device=DEVICE), last + step] for step in range(case["new"] + 1)]
    table = weights[head]
    out = [torch.empty(len(prompts), cfg.vocab_size, dtype=F, device=DEVICE) for _ in rows]
    for lo in range(0, cfg.vocab_size, 16384):
        part = table[lo:lo + 16384].to(F).T
        for o, r in zip(out, rows):
            o[:, lo:lo + 16384] = r @ part
    return out
