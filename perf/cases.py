"""The work that users of the engine have it do, as cases that can be measured one by one.

A case is one pass over a packed batch through ``ModelRunner.step``, the step function that generation, the scheduler
and the replay program all go through: requests that decode one token each on contexts they hold, portions of prompts,
or both together; or prompts and the tokens that answer them.  Tokens are given (as in replay), so that the logits of
every step can be compared.  A process keeps one engine per model, as a server does; weights are random, written once
per machine to the temporary folder.

A case's keys: ``model``; ``decode`` requests that hold ``context`` tokens each and bring one more; ``portions`` of
``tokens`` tokens each, which continue requests that hold ``past`` tokens; ``follow`` single-token steps of these
requests afterwards; ``stride``: logits are wanted at every so many places of a portion, counted from its last (0: the
last alone); ``ragged``: the requests' lengths differ.
"""
import hashlib
import json
import math
import os
import struct
import tempfile
import time

import numpy as np
import torch

from railgun_b200.config.registry import architecture_name, architecture_of
from railgun_b200.engine.batch import StepEntry
from railgun_b200.engine.runner import ModelRunner
from railgun_b200.parts.model import expected_tensors
from railgun_b200.weights.safetensors_io import write_safetensors


# ---- models ---------------------------------------------------------------------------------------------------------
def _llama(width, heads, kv, d, ff, layers, vocab, factor, tied):
    return dict(architectures=["LlamaForCausalLM"], hidden_size=width, num_attention_heads=heads, num_key_value_heads=kv,
                head_dim=d, num_hidden_layers=layers, intermediate_size=ff, vocab_size=vocab, rope_theta=500000.0,
                rope_scaling=dict(rope_type="llama3", factor=factor, low_freq_factor=1.0, high_freq_factor=4.0,
                                  original_max_position_embeddings=8192),
                tie_word_embeddings=tied, rms_norm_eps=1e-5, max_position_embeddings=131072, torch_dtype="bfloat16")


_DECAYS = lambda n: [1.0 - 2.0 ** (-5 - 0.4 * i) for i in range(n)]  # noqa: E731
_DENSE = dict(kind="dense", ff=8192)
_MEPATAR = dict(
    architecture="Mepatar", width=2048, vocab=32768, norm=dict(eps=1e-6, groups=4), embedding=dict(scale=2048 ** 0.5),
    canon=dict(taps=4), layers=[
        dict(type="retention", mixer=dict(heads=16, dim=128, vdim=128, rot=dict(base=10000.0, dims=128), decay=_DECAYS(16)),
             mlp=_DENSE),
        dict(type="delta", mixer=dict(heads=16, kv_heads=8, dim=128, vdim=128, conv=4), mlp=_DENSE),
        dict(type="attention", mixer=dict(heads=16, kv_heads=2, dim=128, vdim=128, scale=128 ** -0.5,
                                          rot=dict(base=10000.0, dims=64), mask=dict(size=512, keep_first=4)),
             mlp=dict(kind="moe", router=dict(experts=32, top=4), expert=dict(ff=2048, limit=7.0)))])
_KASARAX = dict(
    architecture="Kasarax", width=2048, vocab=32768, norm=dict(eps=1e-6), logit_scale=0.5, layers=[
        dict(type="attention", mixer=dict(heads=16, kv_heads=2, dim=128, vdim=128, scale=128 ** -0.5,
                                          q_temp=dict(coef=0.1, every=256)), mlp=_DENSE),
        dict(type="parallel", mixer=dict(
            left=dict(heads=8, kv_heads=2, dim=128, vdim=128, conv=4, scale=128 ** -0.5, rot=dict(base=10000.0, dims=64)),
            right=dict(heads=8, dim=128, vdim=128, decay=_DECAYS(8))), mlp=_DENSE)] * 2)
_MAMBA = dict(type="mamba2", mixer=dict(heads=32, vdim=64, state=128, groups=2, conv=4, norm_groups=2), mlp=_DENSE)
_SAGIZEN = dict(
    architecture="Sagizen", width=2048, vocab=32768, norm=dict(eps=1e-6), layers=[
        _MAMBA, _MAMBA,
        dict(type="parallel", mixer=dict(
            left=dict(heads=8, kv_heads=2, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=512, pool=8),
                      rot=dict(base=10000.0, dims=64, scaling=dict(factor=4.0))),
            right=dict(heads=8, dim=128), left_scale=0.6, right_scale=0.7), mlp=_DENSE)])
# name -> configuration, precision, page size, tokens the cache holds, requests it holds.  The 3B and 8B sizes and the
# other architectures run with a few of their layers: a layer's work is the same however many there are.
MODELS = {
    "tiny": (dict(_llama(96, 3, 1, 32, 256, 3, 500, 8.0, False), rms_norm_eps=1e-6, max_position_embeddings=512,
                  rope_scaling=dict(rope_type="llama3", factor=8.0, low_freq_factor=1.0, high_freq_factor=4.0,
                                    original_max_position_embeddings=64)), "float32", 8, 65536, 256),
    "llama-1b": (_llama(2048, 32, 8, 64, 8192, 16, 128256, 32.0, True), "bfloat16", 16, 64 * 8192 + 8192, 320),
    "llama-3b": (_llama(3072, 24, 8, 128, 8192, 6, 128256, 32.0, True), "bfloat16", 16, 64 * 8192, 320),
    "llama-8b": (_llama(4096, 32, 8, 128, 14336, 4, 128256, 8.0, False), "bfloat16", 16, 320 * 4096, 320),
    "mepatar": (_MEPATAR, "bfloat16", 16, 65536, 32),
    "kasarax": (_KASARAX, "bfloat16", 16, 65536, 128),
    "sagizen": (_SAGIZEN, "bfloat16", 16, 65536, 128),
}


# ---- cases ----------------------------------------------------------------------------------------------------------
def _case(model, decode=0, context=0, portions=0, tokens=0, past=0, follow=0, stride=0, ragged=False):
    return dict(model=model, decode=decode, context=context, portions=portions, tokens=tokens, past=past, follow=follow,
                stride=stride, ragged=ragged)


def listed():
    return [
        # the smallest model in 32-bit: two portions of prompts beside three requests that decode
        dict(_case("tiny", 3, 63, 2, 32, ragged=True), name="tiny-f32-mixed"),
        # one user waiting for the next token
        dict(_case("llama-1b", 1, 1024), name="1b-decode-1"),
        # a few users (the benchmark's headline)
        dict(_case("llama-1b", 8, 1024), name="1b-decode-8"),
        # a busy server: every request at its own length
        dict(_case("llama-1b", 64, 1024, ragged=True), name="1b-decode-64"),
        # a long prompt arrives
        dict(_case("llama-1b", portions=1, tokens=2048), name="1b-prompt-2048"),
        # several short prompts of odd lengths arrive together
        dict(_case("llama-1b", portions=5, tokens=37, ragged=True), name="1b-prompts-short"),
        # portions of prompts beside decoding requests in one step
        dict(_case("llama-3b", 32, 1024, 2, 512), name="3b-mixed"),
        # a busy server with long contexts
        dict(_case("llama-8b", 64, 4096), name="8b-decode-long"),
        # the second portion of a long prompt
        dict(_case("llama-8b", portions=1, tokens=2048, past=2048), name="8b-portion"),
        # a document's tokens are scored: logits at every fourth place (retention, delta rule, window, experts)
        dict(_case("mepatar", portions=1, tokens=2048, stride=4), name="mepatar-score"),
        # a batch of questions and the first tokens of their answers (sinks, convolutions, lightning attention)
        dict(_case("kasarax", portions=6, tokens=301, follow=8, ragged=True), name="kasarax-answers"),
        # one long question and the first tokens of its answer (Mamba-2, pooled blocks, time mixing)
        dict(_case("sagizen", portions=1, tokens=1999, follow=16), name="sagizen-answer"),
    ]


def draw(rng):
    size = lambda lo, hi: min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))  # noqa: E731
    kind = rng.choice(["tiny", "decode", "decode", "prompts", "mixed", "long", "portion", "score", "answers", "answers"])
    ragged = rng.random() < 0.5
    if kind == "tiny":
        return _case("tiny", size(1, 8), size(8, 200), size(1, 4), size(2, 100), ragged=ragged)
    if kind == "decode":
        return _case("llama-1b", size(1, 64), size(16, 2048), ragged=ragged)
    if kind == "prompts":
        n = size(1, 8)
        return _case("llama-1b", portions=n, tokens=size(2, 2048 // n), past=rng.choice([0, 0, size(1, 1024)]), ragged=ragged)
    if kind == "mixed":
        n = size(1, 4)
        return _case("llama-3b", size(1, 48), size(64, 1536), n, size(16, 1024 // n), ragged=ragged)
    if kind == "long":
        return _case("llama-8b", size(1, 64), size(1024, 4096), ragged=ragged)
    if kind == "portion":
        return _case("llama-8b", portions=1, tokens=size(256, 2048), past=rng.choice([0, size(16, 2048)]))
    if kind == "score":
        return _case("mepatar", portions=1, tokens=size(1024, 2048), stride=rng.choice([2, 3, 4]))
    n = size(1, 12)
    return _case(rng.choice(["kasarax", "sagizen"]), portions=n, tokens=size(16, 2048 // n), follow=size(1, 16), ragged=ragged)


def _length(case, n, i):
    """The length of request i where the longest has n tokens."""
    return n - (i * 37) % max(1, n // 3) if case["ragged"] else n


def _requests(case):
    """Per request of the step: (tokens it holds, tokens it brings, places whose logits are wanted, steps afterwards)."""
    out = [(_length(case, case["context"], i), 1, [0], 0) for i in range(case["decode"])]
    for i in range(case["portions"]):
        n = _length(case, case["tokens"], i)
        want = sorted(range(n - 1, -1, -case["stride"])) if case["stride"] else [n - 1]
        out.append((case["past"], n, want, case["follow"]))
    return out


def _sequences(case, seed):
    """All tokens of every request: those it holds, those it brings and those that follow."""
    rng = np.random.default_rng(seed)
    vocab = _config(case["model"]).get("vocab_size") or _config(case["model"])["vocab"]
    return [rng.integers(0, vocab, size=held + n + follow).tolist() for held, n, _, follow in _requests(case)]


# ---- engines --------------------------------------------------------------------------------------------------------
def _config(model):
    return MODELS[model][0]


def _tensors(model):
    """Every tensor of a model: name -> its description."""
    cfg = _config(model)
    arch = architecture_of(architecture_name(cfg))
    config = arch.config_from_dict(cfg)
    return config, expected_tensors(arch.model_spec(config))


def _folder(model):
    """The model's folder: N(0, 0.02) matrices, norms 1 + U(-0.1, 0.1), in bfloat16."""
    tag = hashlib.sha1(json.dumps(_config(model), sort_keys=True).encode()).hexdigest()[:12]
    folder = os.path.join(tempfile.gettempdir(), f"rg_cases_{model}_{tag}")
    if not os.path.exists(folder):
        config, specs = _tensors(model)
        g = torch.Generator(device="cuda")
        g.manual_seed(int(tag[:8], 16))
        tensors = {}
        for name, ts in specs.items():
            shape = tuple(int(n) for n in ts.shape)
            if ts.optional:
                continue
            if ts.init == "norm":
                t = 0.9 + 0.2 * torch.rand(shape, device="cuda", generator=g)
            else:
                t = 0.02 * torch.randn(shape, device="cuda", generator=g)
            tensors[name] = t.to(torch.bfloat16).cpu()
        own = f"{folder}.{os.getpid()}"
        os.makedirs(own)
        with open(os.path.join(own, "config.json"), "w") as f:
            json.dump(config.to_dict(), f)
        write_safetensors(os.path.join(own, "model.safetensors"), tensors)
        try:
            os.rename(own, folder)
        except OSError:                                      # another process was faster
            time.sleep(0.1)
    return folder


_ENGINE = {}                 # the engine in use: model -> runner
_LAST_ID = [0]


def _runner(model):
    if model not in _ENGINE:
        _ENGINE.clear()
        torch.cuda.empty_cache()
        _, dtype, page, tokens, requests = MODELS[model]
        _ENGINE[model] = ModelRunner(_folder(model), dtype=dtype, page_size=page, max_tokens=tokens, max_requests=requests)
    return _ENGINE[model]


class Requests:
    """A batch of requests of one engine: the entries of its steps, and the tokens that some of them hold already."""

    def __init__(self, runner, case, seed):
        self.runner, self.entries, self.follow = runner, [], [[] for _ in range(case["follow"])]
        held_ids, held, self.new_ids = [], [], []
        fill = []
        for (past, n, want, follow), seq in zip(_requests(case), _sequences(case, seed)):
            _LAST_ID[0] += 1
            rid = _LAST_ID[0]
            if past:
                held_ids.append(rid)
                held.append(past)
                fill.append(StepEntry(rid, seq[:past], []))
            else:
                self.new_ids.append(rid)
            self.entries.append(StepEntry(rid, seq[past:past + n], want))
            for k in range(follow):
                self.follow[k].append(StepEntry(rid, [seq[past + n + k]], [0]))
        self.held_ids, self.held = np.asarray(held_ids, dtype=np.int64), np.asarray(held, dtype=np.int32)
        while fill:                                          # the contexts, several requests to a step
            group, total = [], 0
            while fill and (not group or total + len(fill[0].tokens) <= 8192):
                total += len(fill[0].tokens)
                group.append(fill.pop(0))
            runner.step(group)

    def __del__(self):
        self.runner.end(self.held_ids.tolist())


def prepare(case, seed):
    return Requests(_runner(case["model"]), case, seed)


def run(s):
    """The logits of every step.  Afterwards the requests that held tokens hold as many again and the others end."""
    r = s.runner
    logits = r.step(s.entries)
    out = [logits.clone() if s.follow else logits]
    for entries in s.follow:
        out.append(r.step(entries).clone())
    if s.held.size:
        r.alloc.commit_many(s.held_ids, s.held)
    r.end(s.new_ids)
    return out


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _seen(layer, position):
    """Keys that the token at ``position`` attends to in an attention layer (a dict with its window)."""
    mask = layer.get("mask") or {}
    size = mask.get("size") or position + 1
    far = max(0, position + 1 - size)
    return min(position + 1, size) + min(far, mask.get("keep_first", 0)) + (far // mask["pool"] if mask.get("pool") else 0)


def _mixers(model):
    """([attention: heads, kv heads, size, window], [state: numbers of a request's state, operations per token])."""
    cfg = _config(model)
    if "layers" not in cfg:
        m = dict(heads=cfg["num_attention_heads"], kv=cfg["num_key_value_heads"], d=cfg["head_dim"])
        return [m] * cfg["num_hidden_layers"], []
    attention, state = [], []
    for layer in cfg["layers"]:
        m = layer["mixer"]
        for kind, m in ([(layer["type"], m)] if layer["type"] != "parallel" else [("attention", m["left"]), ("matrix", m["right"])]):
            if kind == "attention":
                attention.append(dict(heads=m["heads"], kv=m["kv_heads"], d=m["dim"], mask=m.get("mask")))
            else:
                n = m["heads"] * (m["vdim"] * m["state"] if kind == "mamba2" else m["dim"] * m.get("vdim", m["dim"]))
                state.append((n, (6 if kind == "delta" else 4) * n))
    return attention, state


def work(case):
    cfg = _config(case["model"])
    size = 4 if MODELS[case["model"]][1] == "float32" else 2
    _, specs = _tensors(case["model"])
    moe = next((x["mlp"] for x in cfg.get("layers", []) if x["mlp"]["kind"] == "moe"), None)
    embed = "embed" if "layers" in cfg else "model.embed_tokens.weight"
    tied = not any(n in specs for n in ("head", "lm_head.weight"))
    table = specs[embed].shape[0] * specs[embed].shape[1]
    dense = experts = 0
    for name, ts in specs.items():
        n = int(np.prod([int(x) for x in ts.shape]))
        if name not in (embed, "head", "lm_head.weight"):
            dense, experts = (dense, experts + n) if ".e" in name and moe else (dense + n, experts)
    attention, state = _mixers(case["model"])
    requests = _requests(case)
    total_bytes = total_flops = 0.0
    for step in range(1 + case["follow"]):
        rows = [(held, n, len(want)) if step == 0 else (held + n + step - 1, 1, 1) for held, n, want, _ in requests]
        tokens, wanted = sum(n for _, n, _ in rows), sum(w for _, _, w in rows)
        total_flops += 2.0 * tokens * dense + 2.0 * wanted * table
        total_bytes += size * (dense + table + tokens * specs[embed].shape[1]) + 4.0 * wanted * specs[embed].shape[0]
        if moe:
            e, top = moe["router"]["experts"], moe["router"]["top"]
            total_flops += 2.0 * tokens * experts * top / e
            total_bytes += size * experts * min(1.0, tokens * top / e)
        for m in attention:
            for held, n, _ in rows:
                pairs = sum(_seen(m, p) for p in range(held, held + n))
                total_flops += 4.0 * m["heads"] * m["d"] * pairs
                total_bytes += 2.0 * size * m["kv"] * m["d"] * (n + _seen(m, held + n - 1))
        for numbers, ops in state:
            total_flops += float(ops) * tokens
            total_bytes += 4.0 * numbers * len(rows) * (1 if step == 0 else 2)
    return dict(bytes=total_bytes, flops=total_flops)


def tolerance(case):
    """In 32-bit the logits are off a 64-bit statement by 3e-7; with bfloat16 between the parts of a layer by 0.007 (three
    layers) to 0.02 (sixteen), which two correct orders of rounding may show against one another."""
    return {"rel": 1e-5} if MODELS[case["model"]][1] == "float32" else {"rel": 0.03, "max": 0.5}


# ---- the same in 64 bits, in plain torch ----------------------------------------------------------------------------
def _weights(model):
    """name -> float64 tensor on the GPU, read straight from the file."""
    with open(os.path.join(_folder(model), "model.safetensors"), "rb") as f:
        header = json.loads(f.read(struct.unpack("<Q", f.read(8))[0]))
        start, out = f.tell(), {}
        for name, meta in header.items():
            if name != "__metadata__":
                lo, hi = meta["data_offsets"]
                f.seek(start + lo)
                raw = torch.frombuffer(bytearray(f.read(hi - lo)), dtype=torch.bfloat16)
                out[name] = raw.cuda().reshape(meta["shape"]).double()
    return out


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _conv(x, taps, bias=0.0):
    """x [T, C], taps [C, K], the last column the current token's."""
    K = taps.shape[1]
    padded = torch.cat([x.new_zeros(K - 1, x.shape[1]), x])
    return sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(K)) + bias


def _rotate(x, freq, interleaved):
    """x [T, heads, d]: the first 2 len(freq) numbers of each head turned in pairs by position * freq."""
    n = freq.numel()
    a = torch.arange(x.shape[0], device=x.device, dtype=torch.float64)[:, None] * freq
    c, s = a.cos()[:, None], a.sin()[:, None]
    i, j = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if interleaved else (slice(0, n), slice(n, 2 * n))
    out = x.clone()
    out[..., i], out[..., j] = x[..., i] * c - x[..., j] * s, x[..., j] * c + x[..., i] * s
    return out


def _frequencies(dims, base):
    return base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims)


def _llama3(freq, scaling):
    f, a, b = scaling["factor"], scaling["low_freq_factor"], scaling["high_freq_factor"]
    turns = scaling["original_max_position_embeddings"] * freq / (2 * math.pi)
    s = ((turns - a) / (b - a)).clamp(0.0, 1.0)
    return (1 - s) * freq / f + s * freq


def _attend(q, k, v, rows, scale, size=None, keep=0, pool=0, sink=None):
    """Softmax attention of the tokens ``rows`` of a sequence.  q [rows, H, d], k and v [T, G, d]; a window of ``size``
    that keeps the first ``keep`` tokens, means over blocks of ``pool`` tokens behind it, a sink per head."""
    T, G = k.shape[:2]
    at, j = rows[:, None], torch.arange(T, device=q.device)[None]
    see = (j <= at) & ((at - j < size) | (j < keep)) if size else j <= at
    if pool:
        nb = T // pool
        mean = lambda x: x[:nb * pool].reshape(nb, pool, G, -1).mean(1)  # noqa: E731
        k, v = torch.cat([mean(k), k]), torch.cat([mean(v), v])
        b = torch.arange(nb, device=q.device)[None]
        see = torch.cat([b * pool + pool - 1 <= at - size, see], 1)
    out = torch.empty_like(q)
    for h in range(q.shape[1]):
        g = h // (q.shape[1] // G)
        s = torch.where(see, scale * (q[:, h] @ k[:, g].T), -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(s.shape[0], 1)], 1)
        p = torch.softmax(s, 1)
        out[:, h] = p[:, :k.shape[0]] @ v[:, g]
    return out.flatten(1)


def _exact_llama(w, cfg, tokens, places):
    nh, kv, d, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    freq = _llama3(_frequencies(d, cfg["rope_theta"]), cfg["rope_scaling"])
    x = w["model.embed_tokens.weight"][tokens]
    every = torch.arange(len(tokens), device="cuda")
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        last = i == cfg["num_hidden_layers"] - 1
        rows = places if last else every                     # the last layer's output is wanted at these places alone
        h = _unit(x, eps) * w[p + "input_layernorm.weight"]
        k = _rotate((h @ w[p + "self_attn.k_proj.weight"].T).unflatten(1, (kv, d)), freq, False)
        v = (h @ w[p + "self_attn.v_proj.weight"].T).unflatten(1, (kv, d))
        q = _rotate((h @ w[p + "self_attn.q_proj.weight"].T).unflatten(1, (nh, d)), freq, False)[rows]
        x = x[rows] + _attend(q, k, v, rows, d ** -0.5) @ w[p + "self_attn.o_proj.weight"].T
        h = _unit(x, eps) * w[p + "post_attention_layernorm.weight"]
        h = _silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)
        x = x + h @ w[p + "mlp.down_proj.weight"].T
    head = w["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"]
    return (_unit(x, eps) * w["model.norm.weight"]) @ head.T


def _scan(q, k, v, decay, step=None, bonus=None):
    """A matrix S [H, d, dv] per head over the tokens of q, k [T, H, d] and v [T, H, dv]: S <- decay S + k v^T and
    o = S^T q; with ``step`` [T, H] the delta rule, v less what S holds for k, times the step; with ``bonus`` [H, d]
    the read comes before the update and sees the own token times the bonus.  decay [T or 1, H, d or 1]."""
    S = v.new_zeros(q.shape[1], q.shape[2], v.shape[2])
    decay = decay.expand(q.shape[0], -1, -1)[..., None]
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        if bonus is not None:
            kv = k[t, :, :, None] * v[t, :, None]
            out[t] = (q[t, :, None] @ (S + bonus[..., None] * kv))[:, 0]
            S = decay[t] * S + kv
            continue
        S = decay[t] * S
        u = v[t] if step is None else step[t, :, None] * (v[t] - (k[t, :, None] @ S)[:, 0])
        S = S + k[t, :, :, None] * u[:, None]
        out[t] = (q[t, :, None] @ S)[:, 0]
    return out


def _exact_mepatar(w, cfg, tokens, places):
    eps, groups = cfg["norm"]["eps"], cfg["norm"]["groups"]
    norm = lambda x, weight: _unit(x.unflatten(1, (groups, -1)), eps).flatten(1) * weight  # noqa: E731
    gelu = lambda z: torch.nn.functional.gelu(z, approximate="tanh")  # noqa: E731
    x = w["embed"][tokens] * cfg["embedding"]["scale"]
    rows = torch.arange(len(tokens), device="cuda")
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}.mix."
        h = norm(x, w[f"l{i}.norm1"])
        h = h + _conv(h, w[f"l{i}.canon1"])
        heads = lambda name, n, d: (h @ w[p + name].T + w.get(p + name + ".b", 0.0)).unflatten(1, (n, d))  # noqa: E731
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        if layer["type"] == "retention":
            freq = _frequencies(m["rot"]["dims"], m["rot"]["base"])
            q, k = _rotate(heads("q", H, d), freq, False), _rotate(heads("k", H, d), freq, False) * d ** -0.5
            decay = torch.tensor(m["decay"], dtype=torch.float32, device="cuda").double()[None, :, None]
            o = _unit(_scan(q, k, heads("v", H, dv), decay), eps).flatten(1) * _silu(h @ w[p + "g"].T)
            y = o @ w[p + "o"].T
        elif layer["type"] == "delta":
            G = m["kv_heads"]
            q, k, v = (_silu(_conv(h @ w[p + n].T, w[p + n + ".conv"])).unflatten(1, (-1, d)) for n in "qkv")
            q, k = (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
            q, k = (z.repeat_interleave(H // G, 1) for z in (q * d ** -0.5, k))
            decay = torch.exp(-torch.exp(w[p + "A_log"]) * torch.nn.functional.softplus(h @ w[p + "a"].T + w[p + "dt_bias"]))
            o = _scan(q, k, v, decay[..., None], step=torch.sigmoid(h @ w[p + "b"].T))
            y = ((_unit(o, eps) * w[p + "norm"]).flatten(1) * _silu(h @ w[p + "g"].T)) @ w[p + "o"].T
        else:
            G = m["kv_heads"]
            freq = _frequencies(m["rot"]["dims"], m["rot"]["base"])
            q = _rotate(_unit(heads("q", H, d), eps) * w[p + "q.norm"], freq, True) * w[p + "temp"][:, None]
            k = _rotate(_unit(heads("k", G, d), eps) * w[p + "k.norm"], freq, True)
            o = _attend(q, k, heads("v", G, dv), rows, m["scale"], m["mask"]["size"], m["mask"]["keep_first"])
            y = o @ w[p + "o"].T + w[p + "o.b"]
        f, p, mlp = norm(x, w[f"l{i}.norm2"]), f"l{i}.mlp.", layer["mlp"]
        if mlp["kind"] == "dense":
            y = y + (gelu(f @ w[p + "gate"].T) * (f @ w[p + "up"].T)) @ w[p + "down"].T
        else:
            scores = torch.softmax(f @ w[p + "router"].T, 1)
            best, chosen = scores.topk(mlp["router"]["top"], 1)
            limit = mlp["expert"]["limit"]
            for e in range(mlp["router"]["experts"]):
                at, place = (chosen == e).nonzero(as_tuple=True)
                g = (f[at] @ w[f"{p}e{e}.gate"].T).clamp(max=limit)
                u = (f[at] @ w[f"{p}e{e}.up"].T).clamp(-limit, limit)
                y[at] += best[at, place][:, None] * ((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[f"{p}e{e}.down"].T)
        x = x + y
    return norm(x[places], w["final.norm"]) @ w["head"].T


def _exact_kasarax(w, cfg, tokens, places):
    eps = cfg["norm"]["eps"]
    x = w["embed"][tokens]
    rows = torch.arange(len(tokens), device="cuda")
    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}.mix."
        h = _unit(x, eps) * (1.0 + w[f"l{i}.norm1"])
        if layer["type"] == "attention":
            m = layer["mixer"]
            q, k, v = ((h @ w[p + n].T + w[p + n + ".b"]).unflatten(1, (-1, m["dim"])) for n in "qkv")
            q = q * (1.0 + m["q_temp"]["coef"] * torch.log((rows + 1) // m["q_temp"]["every"] + 1.0))[:, None, None]
            o = _attend(q, k, v, rows, m["scale"], sink=w[p + "q"].new_zeros(m["heads"]))
            o = o.unflatten(1, (m["heads"], -1)) * torch.sigmoid(h @ w[p + "g"].T)[..., None]
            y = o.flatten(1) @ w[p + "o"].T + w[p + "o.b"]
        else:
            m, b = layer["mixer"]["left"], p + "left."
            q, k, v = (_conv(h @ w[b + n].T, w[b + n + ".conv"]) for n in "qkv")
            freq = _frequencies(m["rot"]["dims"], m["rot"]["base"])
            q, k = (_rotate((_unit(z, eps) * w[b + n + ".norm"]).unflatten(1, (-1, m["dim"])), freq, True)
                    for n, z in (("q", q), ("k", k)))
            left = _attend(q, k, v.unflatten(1, (-1, m["vdim"])), rows, m["scale"], sink=w[b + "sink"]) @ w[b + "o"].T
            m, b = layer["mixer"]["right"], p + "right."
            q, k, v = (_silu(h @ w[b + n].T).unflatten(1, (m["heads"], -1)) for n in "qkv")
            decay = torch.tensor(m["decay"], dtype=torch.float32, device="cuda").double()[None, :, None]
            o = _unit(_scan(q, k, v, decay).flatten(1), eps) * w[b + "norm"] * torch.sigmoid(h @ w[b + "g"].T)
            right = o @ w[b + "o"].T
            y = 0.5 * (_unit(left, eps) * w[p + "left.out"] + _unit(right, eps) * w[p + "right.out"])
        b = f"l{i}.mlp."
        x = x + y + (_silu(h @ w[b + "gate"].T) * (h @ w[b + "up"].T)) @ w[b + "down"].T
    return cfg["logit_scale"] * ((_unit(x[places], eps) * (1.0 + w["final.norm"])) @ w["embed"].T)


def _exact_sagizen(w, cfg, tokens, places):
    eps = cfg["norm"]["eps"]
    x = w["embed"][tokens]
    rows = torch.arange(len(tokens), device="cuda")
    shift = lambda z, share: z + (torch.cat([torch.zeros_like(z[:1]), z[:-1]]) - z) * share  # noqa: E731
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        h = shift(x, w[f"l{i}.shift"])
        if layer["type"] == "mamba2":
            H, dv, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
            z, xbc, dt = (h @ w[p + "in"].T).split([H * dv, H * dv + 2 * G * N, H], 1)
            xs, B, C = _silu(_conv(xbc, w[p + "conv"], w[p + "conv.b"])).split([H * dv, G * N, G * N], 1)
            xs, dt = xs.unflatten(1, (H, dv)), torch.nn.functional.softplus(dt + w[p + "dt_bias"])
            B, C = (t.unflatten(1, (G, N)).repeat_interleave(H // G, 1) for t in (B, C))
            o = _scan(C, B * dt[..., None], xs, torch.exp(-torch.exp(w[p + "A_log"]) * dt)[..., None])
            o = (o + w[p + "D"][:, None] * xs).flatten(1) * _silu(z)
            y = (_unit(o.unflatten(1, (m["norm_groups"], -1)), eps).flatten(1) * w[p + "norm"]) @ w[p + "o"].T
        else:
            a, b = m["left"], p + "left."
            q, k, v = ((h @ w[b + n].T + w[b + n + ".b"]).unflatten(1, (-1, a["dim"])) for n in "qkv")
            freq = _frequencies(a["rot"]["dims"], a["rot"]["base"]) / a["rot"]["scaling"]["factor"]
            q, k = _unit(_rotate(q, freq, False), eps), _unit(_rotate(k, freq, False), eps)
            left = _attend(q, k, v, rows, a["scale"], a["mask"]["size"], pool=a["mask"]["pool"]) @ w[b + "o"].T
            a, b = m["right"], p + "right."
            mixed = {s: shift(h, w[b + "mu." + s]) for s in "rkvgw"}
            r, k, v = ((mixed[s] @ w[b + s].T).unflatten(1, (a["heads"], -1)) for s in "rkv")
            decay = torch.exp(-torch.exp(torch.tanh(mixed["w"] @ w[b + "w1"].T) @ w[b + "w2"].T + w[b + "w0"]))
            o = _unit(_scan(r, k, v, decay.unflatten(1, (a["heads"], -1)), bonus=w[b + "u"]), eps).flatten(1)
            right = (o * w[b + "norm"] * _silu(mixed["g"] @ w[b + "g"].T)) @ w[b + "o"].T
            y = m["left_scale"] * left + m["right_scale"] * right
        x = x + _unit(y, eps) * w[f"l{i}.norm1"]
        f = (_silu(x @ w[f"l{i}.mlp.gate"].T) * (x @ w[f"l{i}.mlp.up"].T)) @ w[f"l{i}.mlp.down"].T
        x = x + _unit(f, eps) * w[f"l{i}.norm2"]
    return (_unit(x[places], eps) * w["final.norm"]) @ w["head"].T


def exact(case, seed):
    """The logits of every step from whole sequences; None where that would be hundreds of teraflops in 64 bits."""
    cfg = _config(case["model"])
    sequences = _sequences(case, seed)
    if sum(map(len, sequences)) * 2.0 * sum(int(np.prod([int(n) for n in s.shape])) for s in _tensors(case["model"])[1].values()
                                            if len(s.shape) == 2) > 1.2e15:
        return None
    model = {"Mepatar": _exact_mepatar, "Kasarax": _exact_kasarax, "Sagizen": _exact_sagizen}.get(cfg.get("architecture"), _exact_llama)
    w = _weights(case["model"])
    out = [[] for _ in range(1 + case["follow"])]
    for (held, n, want, follow), seq in zip(_requests(case), sequences):
        places = [held + i for i in want] + [held + n + k for k in range(follow)]
        got = model(w, cfg, torch.tensor(seq, device="cuda"), torch.tensor(places, device="cuda"))
        out[0].append(got[:len(want)])
        for k in range(follow):
            out[1 + k].append(got[len(want) + k:][:1])
    return [torch.cat(rows) for rows in out]
