"""Workloads that the engine is timed on: one engine step, or a whole ``LLM.generate`` call, as a server
or an offline job makes them, each with the bytes and operations it cannot do without and a plain float64
computation of its outputs.

A step case has ``rows`` requests that decode one token each behind ``context`` tokens (``ragged``: behind
contexts from half of that up) and ``portions`` of prompts with ``tokens`` tokens together, each behind
``history`` tokens of the same prompt that earlier steps ran. Steps of single tokens run as the captured
graph, as the engine runs them; steps with portions run uncaptured, as the engine runs them at these
sizes. The outputs are the logits of every wanted row (of each decoded token and of each portion's last
token), the running states, and after a step of single tokens the rows it wrote into the cache (a portion's
own attention reads them back from there, a single token's does not). Nothing is committed after a step, so
that a case can be run again at the same positions.

A generate case is ``requests`` prompts of 16 to ``context`` tokens through ``LLM.generate``, with
``new_tokens`` generated for each; half of the requests are greedy, half sampled.

Weights are random at the sizes of this package's presets, drawn as its random-weights mode draws them
(N(0, 0.02^2), scales around one). The presets' routed feed-forwards are replaced by the dense ones of the
same preset: with bfloat16 activations a token's choice of experts is decided by rounding often enough
that two correct implementations differ by more than any tolerance that would mean something.
"""

from __future__ import annotations

import functools
import math
import random

import torch

from llmserve_b200 import LLM, SamplingParams
from llmserve_b200.config.registry import architecture_for
from llmserve_b200.engine.batch import StepEntry
from llmserve_b200.engine.decode_graph import DecodeGraphs
from llmserve_b200.engine.runner import ModelRunner, build_model
from llmserve_b200.models.hub import preset_config_dict
from llmserve_b200.ops import get_ops
from llmserve_b200.parts.base import role_dtype

PAGE = 16  # tokens per cache page
MAX_LEN = 8192  # the longest context of the size presets
F64 = torch.float64


# ------------------------------------------------------------------------------- the cases
def _step(name, model, dtype="bfloat16", rows=0, context=0, ragged=False, portions=0, tokens=0, history=0):
    return {"name": name, "kind": "step", "model": model, "dtype": dtype, "rows": rows, "context": context,
            "ragged": ragged, "portions": portions, "tokens": tokens, "history": history}


def listed():
    return [
        # one user in a chat with the smallest model: the shortest step there is
        _step("decode_135m_b1", "smollm2-135m", rows=1, context=517),
        # the benchmark's workload: eight requests behind 2048-token prompts
        _step("decode_1.7b_b8", "smollm2-1.7b", rows=8, context=2048),
        # a full server: the default limit of 64 running requests, contexts of different lengths
        _step("decode_1.7b_b64", "smollm2-1.7b", rows=64, context=2100, ragged=True),
        # long documents: sixteen requests near the end of an 8192-token context
        _step("decode_135m_long", "smollm2-135m", rows=16, context=8100, ragged=True),
        # a prompt of the benchmark's length in one step
        _step("prefill_1.7b", "smollm2-1.7b", portions=1, tokens=2048),
        # continuous batching under the default budget of 1024 tokens: running requests beside prompts
        _step("mixed_1.7b", "smollm2-1.7b", rows=40, context=900, ragged=True, portions=3, tokens=983),
        # a long prompt in portions: the last one, over the keys of the ones before it
        _step("prefill_135m_tail", "smollm2-135m", portions=1, tokens=2040, history=6144),
        # the 32-bit path from end to end: scheduler, chunked prompts, captured steps, sampling
        {"name": "generate_135m_f32", "kind": "generate", "model": "smollm2-135m", "dtype": "float32",
         "requests": 6, "context": 300, "new_tokens": 24},
        # the other designs at the 1.7B model's layer sizes, prompts and decoding
        _step("prefill_gubotar", "gubotar-2048", portions=1, tokens=2048),
        _step("prefill_tanupel", "tanupel-2048", portions=2, tokens=1999),
        _step("decode_lanilorn_b8", "lanilorn-2048", rows=8, context=1500, ragged=True),
        _step("decode_miberax_b24", "miberax-2048", rows=24, context=1111, ragged=True),
    ]


STEP_MODELS = ("smollm2-1.7b", "smollm2-360m", "smollm2-135m", "gubotar-2048", "tanupel-2048", "lanilorn-2048",
               "miberax-2048")


def draw(rng: random.Random):
    """A case of the same ranges: decoding 1 to 64 requests, 33 to 2048 prompt tokens in one to four portions
    with up to 6000 tokens before them, or both; now and then in float32 on the smallest model."""
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice(STEP_MODELS)
    kind = rng.choice(("decode", "decode", "prompt", "prompt", "mixed", "generate"))
    if kind == "generate":
        return {"kind": "generate", "model": "smollm2-135m", "dtype": "float32", "requests": rng.randint(2, 8),
                "context": spread(40, 300), "new_tokens": rng.randint(8, 24)}
    case = _step("", model)
    del case["name"]
    if kind != "prompt":
        case["rows"] = spread(1, 64)
        limit = 8000 if model == "smollm2-135m" else 2100
        case["context"] = min(spread(60, limit), max(60, 130000 // case["rows"]))
        case["ragged"] = rng.random() < 0.7
    if kind != "decode":
        case["portions"] = rng.randint(1, 4)
        case["tokens"] = spread(33, 2048 if kind == "prompt" else 1000)
        if rng.random() < 0.4:
            case["history"] = spread(16, 6000 if model == "smollm2-135m" else 2000)
    if model == "smollm2-135m" and rng.random() < 0.3:
        case["dtype"] = "float32"
        case["tokens"] = min(case["tokens"], 500)
        case["history"] = min(case["history"], 1000)
        case["context"] = min(case["context"], 1000)
    return case


# ------------------------------------------------------------------------------- inputs
def _config(model: str) -> dict:
    d = preset_config_dict(model)
    dense = next((l["mlp"] for l in d.get("layers", ()) if l["mlp"]["kind"] == "dense"), None)
    for layer in d.get("layers", ()):
        layer["mlp"] = dense
    return d


def _draw_weight(shape, role, gen):
    if role == "mix":
        return torch.rand(shape, generator=gen, device="cuda")
    t = torch.randn(shape, generator=gen, device="cuda") * 0.02
    return t + 1.0 if role == "scale" else t


def _checkpoint(arch, cfg, seed) -> dict:
    """Checkpoint tensor name -> bfloat16 tensor."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return {s.name: _draw_weight(tuple(s.shape), e.role, gen).to(torch.bfloat16)
            for e in arch.checkpoint_layout(cfg).entries for s in e.sources}


def _portion_lengths(case) -> list[int]:
    """Uneven: the k-th portion is about k times the first."""
    n, total = case["portions"], case["tokens"]
    if not n:
        return []
    parts = [max(1, total * (k + 1) * 2 // (n * (n + 1))) for k in range(n)]
    parts[-1] += total - sum(parts)
    return parts


def _contexts(case) -> list[int]:
    c = case["context"]
    return [c - (i * 977) % (c // 2 + 1) if case["ragged"] else c for i in range(case["rows"])]


def _sequences(case, vocab, seed):
    """(all tokens, how many of them earlier steps ran) of every request of a step case."""
    g = torch.Generator().manual_seed(seed + 1)
    before = _contexts(case) + [case["history"]] * case["portions"]
    new = [1] * case["rows"] + _portion_lengths(case)
    return [(torch.randint(0, vocab, (b + n,), generator=g).tolist(), b) for b, n in zip(before, new)]


def prepare(case, seed):
    """The model, a runner and its cache filled with what came before the step; or an ``LLM`` and prompts."""
    if case["kind"] == "generate":
        return _prepare_generate(case, seed)
    d = _config(case["model"])
    arch = architecture_for(d)
    cfg = arch.config_cls.from_dict(d)
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16

    def parameters(layout, compute, device):
        tensors = _checkpoint(arch, cfg, seed)
        return {e.param: torch.cat([tensors[s.name] for s in e.sources]).to(role_dtype(e.role, compute)).contiguous()
                for e in layout.entries}

    model = build_model(arch, cfg, parameters, dtype, "cuda", get_ops("cuda"), MAX_LEN)
    seqs = _sequences(case, model.plan.vocab_size, seed)
    longest = max(len(t) for t, _ in seqs)
    runner = ModelRunner(model, page_tokens=PAGE, num_pages=sum(-(-len(t) // PAGE) + 2 for t, _ in seqs),
                         max_model_len=4096 if longest <= 4096 else MAX_LEN, max_num_seqs=max(64, len(seqs)),
                         max_num_batched_tokens=2048)
    for rid in range(len(seqs)):
        runner.manager.admit(rid)
    _run_history(runner, seqs)
    entries = []
    for rid, (tokens, before) in enumerate(seqs):
        rest = tokens[before:]
        runner.manager.allocate(rid, len(rest))
        entries.append(StepEntry(rid, rest, [len(rest) - 1]))
    graphs = DecodeGraphs(runner) if case["portions"] == 0 else None
    return {"runner": runner, "graphs": graphs, "entries": entries, "written": _written(runner, seqs)}


def _written(runner, seqs):
    """Page and place in the page of every request's last token, for each group of cache layers."""
    out = []
    for gi in range(len(runner.manager.groups)):
        pages = [runner.manager.held[rid].tables[gi][(len(t) - 1) // PAGE] for rid, (t, _) in enumerate(seqs)]
        out.append((torch.tensor(pages, device="cuda"),
                    torch.tensor([(len(t) - 1) % PAGE for t, _ in seqs], device="cuda")))
    return out


def _run_history(runner, seqs, portion=2048, budget=8192):
    """The tokens before the step, in portions, several requests at a time."""
    done = [0] * len(seqs)
    while True:
        entries, room = [], budget
        for rid, (tokens, before) in enumerate(seqs):
            n = min(before - done[rid], portion, room)
            if n > 0:
                entries.append(StepEntry(rid, tokens[done[rid] : done[rid] + n], []))
                done[rid] += n
                room -= n
        if not entries:
            return
        runner.run(entries)


def _prepare_generate(case, seed):
    g = torch.Generator().manual_seed(seed + 2)
    rng = random.Random(seed)
    n, longest = case["requests"], case["context"]
    llm = LLM(f"random:{case['model']}", dtype=case["dtype"], seed=seed, max_model_len=1024, num_kv_blocks=1024)
    lengths = [longest] + [rng.randint(16, longest) for _ in range(n - 1)]
    vocab = llm.engine.model_cfg.vocab_size
    prompts = [torch.randint(0, vocab, (k,), generator=g).tolist() for k in lengths]
    params = [SamplingParams(temperature=0.0 if i % 2 == 0 else 0.8, top_p=1.0 if i % 2 == 0 else 0.95, seed=seed + i,
                             max_tokens=case["new_tokens"], ignore_eos=True) for i in range(n)]
    return {"llm": llm, "prompts": prompts, "params": params}


def run(state):
    if "llm" in state:
        outs = state["llm"].generate(state["prompts"], state["params"])
        return {"tokens": torch.tensor([o.outputs[0].token_ids for o in outs])}
    pools, slots = state["runner"].pools, state["runner"].manager.max_requests
    states = [t[:, :slots] for t in pools.state]  # the spare slot, where padding rows write, belongs to nobody
    if state["graphs"] is None:
        return {"logits": state["runner"].step(state["entries"]), "states": states}
    logits = state["graphs"].captured_logits(state["entries"])
    rows = [kv[:, :, pages, :, places] for kv, (pages, places) in zip(pools.kv, state["written"])]
    return {"logits": logits, "states": states, "rows": rows}


# ------------------------------------------------------------------------------- what cannot be done without
@functools.lru_cache(maxsize=None)
def _layers(model: str):
    """Every run of a layer as (matrix elements, mixers); a mixer is ("attention", query heads, key/value heads,
    key dim, value dim, furthest key) or ("state", heads, key dim, value dim)."""
    d = _config(model)
    if "layers" not in d:
        w, H, G, D, ff = (d[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim",
                                         "intermediate_size"))
        layer = (w * D * (2 * H + 2 * G) + 3 * w * ff, (("attention", H, G, D, D, 0),))
        return w, d["vocab_size"], (layer,) * d["num_hidden_layers"]
    arch = architecture_for(d)
    cfg = arch.config_cls.from_dict(d)
    count = [0] * len(d["layers"])
    for e in arch.checkpoint_layout(cfg).entries:
        if e.param.startswith("layers."):
            count[int(e.param.split(".")[1])] += sum(math.prod(s.shape) for s in e.sources)

    def mixers(kind, m):
        if kind == "parallel":
            right = m["right"]
            return mixers("attention", m["left"]) + (("state", right["heads"], right["dim"], right["vdim"]),)
        if kind in ("retention", "gla"):
            return (("state", m["heads"], m["dim"], m["vdim"]),)
        maps = 2 if kind == "attention_2" else 1
        return (("attention", maps * m["heads"], m["kv_heads"], m["dim"], m["vdim"],
                 (m.get("mask") or {}).get("size", 0)),)

    order = [i for i, _ in _runs(d)]
    return d["width"], d["vocab"], tuple((count[i], mixers(d["layers"][i]["type"], d["layers"][i]["mixer"])) for i in order)


def _step_work(model, elem, entries):
    """``entries``: (tokens before, new tokens, wanted rows) of every request of a step."""
    width, vocab, layers = _layers(model)
    new = sum(n for _, n, _ in entries)
    wanted = sum(r for _, _, r in entries)
    byte = elem * (width * vocab + new * width) + 4 * wanted * vocab
    flop = 2.0 * wanted * width * vocab
    for matrix, mixers in layers:
        byte += elem * matrix
        flop += 2.0 * new * matrix
        for m in mixers:
            for before, n, _ in entries:
                if m[0] == "state":
                    _, H, dk, dv = m
                    byte += 4 * H * dk * dv * (2 if before else 1)
                    flop += 4.0 * n * H * dk * dv
                    continue
                _, H, G, dk, dv, reach = m
                kept = min(before, reach) if reach else before
                byte += elem * G * (dk + dv) * (kept + n)
                pairs = sum(min(before + i + 1, reach) for i in range(n)) if reach else n * before + n * (n + 1) // 2
                flop += 2.0 * H * (dk + dv) * pairs
    return byte, flop


def work(case):
    elem = 4 if case["dtype"] == "float32" else 2
    if case["kind"] == "generate":
        n, c = case["requests"], (case["context"] + 16) // 2
        byte, flop = _step_work(case["model"], elem, [(0, c, 1)] * n)
        for k in range(case["new_tokens"] - 1):
            b, f = _step_work(case["model"], elem, [(c + k, 1, 1)] * n)
            byte, flop = byte + b, flop + f
        return {"bytes": byte, "flops": flop}
    entries = [(c, 1, 1) for c in _contexts(case)] + [(case["history"], n, 1) for n in _portion_lengths(case)]
    byte, flop = _step_work(case["model"], elem, entries)
    return {"bytes": byte, "flops": flop}


def tolerance(case):
    if case["kind"] == "generate":
        return "exact"  # token ids; 32-bit sums in another order move logits by a millionth of their spread
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 1e-3}
    # against 64 bits: 0.02 to 0.025 after the 24 layers of the largest preset, 0.011 for Gubotar (keys double as
    # values), 0.004 to 0.007 for the others
    return {"rel": 0.03 if case["model"] in ("smollm2-1.7b", "gubotar-2048") else 0.02, "max": 0.3}


# ------------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """Every request's whole sequence through a plain float64 model: the wanted rows' logits."""
    if case["kind"] == "generate":
        return None  # token ids have no 64-bit value
    d = _config(case["model"])
    arch = architecture_for(d)
    w = _Weights(_checkpoint(arch, arch.config_cls.from_dict(d), seed))
    seqs = _sequences(case, d.get("vocab", d.get("vocab_size")), seed)
    model = _MODELS[d.get("architecture", "Llama")]
    logits = torch.cat([model(d, w, torch.tensor(tokens, device="cuda")) for tokens, _ in seqs])
    return {"logits": logits, "states": None, "rows": None}


class _Weights:
    """Checkpoint tensors as float64, widened once."""

    def __init__(self, tensors):
        self.tensors, self.wide = tensors, {}

    def __getitem__(self, name):
        if name not in self.wide:
            self.wide[name] = self.tensors[name].to(F64)
        return self.wide[name]


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _attend(q, k, v, scale, window=0, chunk=0, softcap=0.0, sink=None, slopes=None):
    """q [n, H, d], k [n, G, d], v [n, G, dv] -> [n, H, dv]; causal, head by head, a block of queries at a time.
    ``window`` keys back, or the keys of the query's own ``chunk``; ``scale`` a number or one per head."""
    n, H, _ = q.shape
    group = H // k.shape[1]
    out = torch.empty(n, H, v.shape[-1], dtype=F64, device=q.device)
    for a in range(0, n, 2048):
        b = min(n, a + 2048)
        i = torch.arange(a, b, device=q.device)[:, None]
        j = torch.arange(b, device=q.device)[None, :]
        hidden = j > i
        if window:
            hidden |= i - j >= window
        if chunk:
            hidden |= i // chunk != j // chunk
        for h in range(H):
            s = q[a:b, h] @ k[:b, h // group].T * (scale[h] if torch.is_tensor(scale) else scale)
            if softcap:
                s = softcap * torch.tanh(s / softcap)
            if slopes is not None:
                s -= slopes[h] * (i - j)
            s.masked_fill_(hidden, -math.inf)
            if sink is None:
                p = s.softmax(-1)
            else:
                p = torch.cat([s, sink[h].expand(b - a, 1)], 1).softmax(-1)[:, :-1]
            out[a:b, h] = p @ v[:b, h // group]
    return out


def _rotate(x, freq, dims, neighbours=False, factor=1.0):
    """x [n, heads, d]: the pairs (i, i + dims / 2), or (2 i, 2 i + 1), of the first ``dims`` dims are turned."""
    n = x.shape[0]
    ang = torch.arange(n, dtype=F64, device=x.device)[:, None] * freq.to(x.device)
    c, s = (ang.cos() * factor)[:, None, :], (ang.sin() * factor)[:, None, :]
    out = x.clone()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if neighbours else (slice(0, dims // 2), slice(dims // 2, dims))
    out[..., a] = x[..., a] * c - x[..., b] * s
    out[..., b] = x[..., b] * c + x[..., a] * s
    return out


def _frequencies(base, dims):
    return base ** (-torch.arange(0, dims, 2, dtype=F64) / dims)


def _llama(d, w, tokens):
    n, H, G, D, eps = len(tokens), d["num_attention_heads"], d["num_key_value_heads"], d["head_dim"], d["rms_norm_eps"]
    freq = _frequencies(d["rope_theta"], D)
    x = w["model.embed_tokens.weight"][tokens]
    for i in range(d["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * w[p + "input_layernorm.weight"]
        q, k, v = ((h @ w[f"{p}self_attn.{t}_proj.weight"].T).view(n, -1, D) for t in "qkv")
        o = _attend(_rotate(q, freq, D), _rotate(k, freq, D), v, D ** -0.5)
        x = x + o.reshape(n, H * D) @ w[p + "self_attn.o_proj.weight"].T
        h = _rms(x, eps) * w[p + "post_attention_layernorm.weight"]
        f = _silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)
        x = x + f @ w[p + "mlp.down_proj.weight"].T
    return _rms(x[-1:], eps) * w["model.norm.weight"] @ w["model.embed_tokens.weight"].T


def _scan(q, k, v, decay, beta=None):
    """q, k [n, H, d], v [n, H, dv], decay [n, H, d] or [H, 1]: S <- decay S + k u^T, o = S^T q, with u = v, or (the
    delta rule) u = beta (v - S^T k)."""
    n, H, d = q.shape
    S = torch.zeros(H, d, v.shape[-1], dtype=F64, device=q.device)
    out = torch.empty(n, H, v.shape[-1], dtype=F64, device=q.device)
    for t in range(n):
        S = S * (decay[t] if decay.dim() == 3 else decay)[:, :, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S += k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hdv,hd->hv", S, q[t])
    return out


def _heads(h, w, name, count):
    return (h @ w[name].T).view(h.shape[0], count, -1)


def _gubotar(d, w, tokens):
    n, eps = len(tokens), d["norm"]["eps"]
    x = w["embed"][tokens]
    for i, layer in enumerate(d["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        prev = torch.cat([torch.zeros_like(x[:1]), x[:-1]])
        h = x + (prev - x) * w[p + "shift"]
        if layer["type"] == "parallel":
            a, b, pl, pr = m["left"], m["right"], p + "mix.left.", p + "mix.right."
            q, raw = _heads(h, w, pl + "q", a["heads"]), _heads(h, w, pl + "k", a["kv_heads"])
            slopes = [2.0 ** (-8.0 * (t + 1) / a["heads"]) for t in range(a["heads"])]
            o = _attend(_rms(q, eps) * w[pl + "q.norm"], _rms(raw, eps) * w[pl + "k.norm"], raw,
                        a["scale"] * w[pl + "temp"], chunk=a["mask"]["size"], slopes=slopes)
            left = o.reshape(n, -1) @ w[pl + "o"].T
            q, k, v = (_silu(_heads(h, w, pr + t, b["heads"])) for t in "qkv")
            o = _scan(q, k, v, torch.tensor(b["decay"], dtype=F64, device="cuda")[:, None]).reshape(n, -1)
            right = _rms(o, eps) * w[pr + "norm"] * torch.sigmoid(h @ w[pr + "g"].T) @ w[pr + "o"].T
            y = 0.5 * (_rms(left, eps) * w[pl + "out"] + _rms(right, eps) * w[pr + "out"])
        else:
            pm, H, dk, rot = p + "mix.", m["heads"], m["dim"], m["rot"]
            q, k, v = (_heads(h, w, pm + t, H) for t in "qkv")
            freq = _frequencies(rot["base"], rot["dims"])
            q, k = _rotate(q, freq, rot["dims"]), _rotate(k, freq, rot["dims"]) * dk ** -0.5
            o = _scan(q, k, v, torch.tensor(m["decay"], dtype=F64, device="cuda")[:, None])
            y = _rms(o, eps).reshape(n, -1) * _silu(h @ w[pm + "g"].T) @ w[pm + "o"].T
        x = x + _rms(y, eps) * (1 + w[p + "norm1"])
        f = (_silu(x @ w[p + "mlp.gate"].T) * (x @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
        x = x + _rms(f, eps) * (1 + w[p + "norm2"])
    return _rms(x[-1:], eps) * (1 + w["final.norm"]) @ w["embed"].T


def _yarn(rot):
    dims, s = rot["dims"], rot["scaling"]
    f = _frequencies(rot["base"], dims)
    at = lambda turns: dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))
    lo, hi = max(math.floor(at(s["fast"])), 0), min(math.ceil(at(s["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F64) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / s["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(s["factor"]) + 1


def _lanilorn_mixer(kind, h, w, p, m, eps):
    n, H = h.shape[0], m["heads"]
    if kind == "gla":
        q, k, v = (_heads(h, w, p + t, H) for t in "qkv")
        alpha = torch.sigmoid(h @ w[p + "a1"].T @ w[p + "a2"].T + w[p + "a2.b"]) ** (1 / m["tau"])
        o = _scan(q * m["dim"] ** -0.5, k, v, alpha.view(n, H, -1))
        return (_rms(o, eps) * w[p + "norm"]).reshape(n, -1) * _silu(h @ w[p + "g"].T) @ w[p + "o"].T
    gate = torch.sigmoid(h @ w[p + "g"].T)[:, :, None]
    if kind == "attention":
        raw = h @ w[p + "k"].T
        q = (_rms(h @ w[p + "q"].T, eps) * w[p + "q.norm"]).view(n, H, -1)
        k = (_rms(raw, eps) * w[p + "k.norm"]).view(n, m["kv_heads"], -1)
        freq, mag = _yarn(m["rot"])
        dims = m["rot"]["dims"]
        o = _attend(_rotate(q, freq, dims, factor=mag), _rotate(k, freq, dims, factor=mag),
                    raw.view(n, m["kv_heads"], -1), m["scale"], window=m["mask"]["size"], sink=w[p + "sink"])
    else:
        q, k = (h @ w[p + "q"].T).view(n, H, 2, -1), (h @ w[p + "k"].T).view(n, m["kv_heads"], 2, -1)
        v, t = _heads(h, w, p + "v", m["kv_heads"]), m["q_temp"]
        pos = torch.arange(n, dtype=F64, device="cuda")
        q = q * (1 + t["coef"] * torch.log(torch.floor((pos + 1) / t["every"]) + 1))[:, None, None, None]
        a1, a2 = (_attend(q[:, :, c], k[:, :, c], v, m["scale"]) for c in (0, 1))
        lam = torch.exp((w[p + "lq1"] * w[p + "lk1"]).sum()) - torch.exp((w[p + "lq2"] * w[p + "lk2"]).sum()) + m["diff"]
        o = _rms(a1 - lam * a2, eps) * (1 - m["diff"])
    return (o * gate).reshape(n, -1) @ w[p + "o"].T


def _lanilorn(d, w, tokens):
    eps = d["norm"]["eps"]
    X = (w["embed"][tokens] * d["embedding"]["scale"])[:, None, :].repeat(1, d["streams"], 1)
    for i, layer in enumerate(d["layers"]):
        p = f"l{i}."
        for q in "12":
            h = _rms(torch.einsum("s,nsw->nw", w[f"{p}hc{q}.in"], X), eps) * w[f"{p}norm{q}"]
            if q == "1":
                y = _lanilorn_mixer(layer["type"], h, w, p + "mix.", layer["mixer"], eps)
            else:
                y = torch.relu(h @ w[p + "mlp.up"].T) ** 2 @ w[p + "mlp.down"].T
            X = (torch.einsum("st,nsw->ntw", w[f"{p}hc{q}.mix"], X)
                 + w[f"{p}hc{q}.out"][None, :, None] * (y * w[f"{p}ls{q}"])[:, None, :])
    return _rms(X[-1:].sum(1), eps) * w["final.norm"] @ w["embed"].T * d["logit_scale"]


def _delta(h, w, p, m, decays):
    """The delta rule's output before its norm: short convolutions, unit keys and queries."""
    n, H, G, d = h.shape[0], m["heads"], m["kv_heads"], m["dim"]

    def conv(t):
        y, taps = h @ w[p + t].T, w[f"{p}{t}.conv"]
        K = taps.shape[1]
        padded = torch.cat([torch.zeros(K - 1, y.shape[1], dtype=F64, device="cuda"), y])
        return _silu(sum(taps[:, j] * padded[j : j + n] for j in range(K)))

    unit = lambda t: t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    rep = lambda t: t.repeat_interleave(H // G, 1)
    q, k = rep(unit(conv("q").view(n, G, d))) * d ** -0.5, rep(unit(conv("k").view(n, G, d)))
    return _scan(q, k, conv("v").view(n, H, -1), decays, torch.sigmoid(h @ w[p + "b"].T))


def _softplus(z):
    return torch.nn.functional.softplus(z, threshold=1e9)


def _miberax(d, w, tokens):
    n, eps, groups = len(tokens), d["norm"]["eps"], d["norm"]["groups"]
    norm = lambda x, name: _rms(x.view(len(x), groups, -1), eps).view(len(x), -1) * w[name]
    x = w["embed"][tokens]
    for i, layer in enumerate(d["layers"]):
        p, a, b = f"l{i}.", layer["mixer"]["left"], layer["mixer"]["right"]
        pl, pr, rot = p + "mix.left.", p + "mix.right.", a["rot"]
        h = norm(x, p + "norm1")
        freq = _frequencies(rot["base"], rot["dims"]) / rot["scaling"]["factor"]
        q, k = (_rotate(_heads(h, w, pl + t, a[c]), freq, rot["dims"], neighbours=True)
                for t, c in (("q", "heads"), ("k", "kv_heads")))
        o = _attend(q, k, _heads(h, w, pl + "v", a["kv_heads"]), a["scale"], chunk=a["mask"]["size"])
        left = o.reshape(n, -1) @ w[pl + "o"].T
        g = torch.exp(-torch.exp(w[pr + "A_log"]) * _softplus(h @ w[pr + "a"].T + w[pr + "dt_bias"]))
        o = _rms(_delta(h, w, pr, b, g[:, :, None]), eps) * w[pr + "norm"]
        right = o.reshape(n, -1) * _silu(h @ w[pr + "g"].T) @ w[pr + "o"].T
        x = x + 0.5 * (_rms(left, eps) * w[pl + "out"] + _rms(right, eps) * w[pr + "out"])
        z, c = norm(x, p + "norm2") @ w[p + "mlp.up"].T, w[p + "mlp.act"]
        f = c[0] * _rms(z, eps) + c[1] * _rms(z ** 2, eps) + c[2] * _rms(z ** 3, eps) + c[3]
        x = x + f @ w[p + "mlp.down"].T
    return norm(x[-1:], "final.norm") @ w["embed"].T


def _runs(d):
    """(layer, pass or None): the layers of the loop run several times; the pass is named at its first layer."""
    n = len(d["layers"])
    loop = d.get("loop") or {"start": n, "stop": n, "times": 0}
    order = [(i, None) for i in range(loop["start"])]
    for t in range(loop["times"]):
        order += [(i, t if i == loop["start"] else None) for i in range(loop["start"], loop["stop"])]
    return order + [(i, None) for i in range(loop["stop"], n)]


def _llama3_frequencies(rot):
    f, s = _frequencies(rot["base"], rot["dims"]), rot["scaling"]
    if "original" not in s:
        return f / s["factor"]
    wave = 2 * math.pi / f
    t = ((s["original"] / wave - s["low"]) / (s["high"] - s["low"])).clamp(0, 1)
    return (1 - t) * f / s["factor"] + t * f


def _tanupel(d, w, tokens):
    n, eps = len(tokens), d["norm"]["eps"]

    def attention(h, p, m):
        freq, dims = _llama3_frequencies(m["rot"]), m["rot"]["dims"]
        q, k = ((_rms(h @ w[p + t].T, eps) * w[f"{p}{t}.norm"]).view(n, m[c], -1)
                for t, c in (("q", "heads"), ("k", "kv_heads")))
        o = _attend(_rotate(q, freq, dims), _rotate(k, freq, dims), _heads(h, w, p + "v", m["kv_heads"]), m["scale"],
                    softcap=m.get("softcap", 0.0))
        return o.reshape(n, -1) @ w[p + "o"].T

    def delta(h, p, m):
        z = h @ w[p + "a1"].T @ w[p + "a2"].T
        g = torch.exp(-torch.exp(w[p + "A_log"])[None, :, None] * _softplus(z + w[p + "dt_bias"]).view(n, m["heads"], -1))
        o = (_rms(_delta(h, w, p, m, g), eps) * w[p + "norm"]).reshape(n, -1)
        return o * torch.sigmoid(h @ w[p + "g1"].T @ w[p + "g2"].T) @ w[p + "o"].T

    x = w["embed"][tokens] * d["embedding"]["scale"]
    for i, t in _runs(d):
        p, layer = f"l{i}.", d["layers"][i]
        m = layer["mixer"]
        if t is not None:
            x = x + w["loop.step"][t]
        h = _rms(x, eps) * (1 + w[p + "norm1"])
        if layer["type"] == "attention":
            y = attention(h, p + "mix.", m)
        else:
            y = (m["left_scale"] * attention(h, p + "mix.left.", m["left"])
                 + m["right_scale"] * delta(h, p + "mix.right.", m["right"]))
        f = (_silu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
        x = x + d["residual_mult"] * (y + f)
    return _rms(x[-1:], eps) * (1 + w["final.norm"]) @ w["head"].T


_MODELS = {"Llama": _llama, "Gubotar": _gubotar, "Lanilorn": _lanilorn, "Miberax": _miberax, "Tanupel": _tanupel}
