"""The work that programs built on this library have it do, as cases that can be timed and checked.

A case is a dict of plain values. `prepare` makes what a program has in hand (a loaded engine, or one part with its
weights and a cache), `run` is one pass through the public entry points, `exact` the same in 64-bit plain torch,
`work` the bytes and operations that the pass cannot do without. Six kinds of case:

    answer      a whole engine: requests of unequal prompt lengths in one step, then given tokens one by one through
                the captured one-token step (a generation loop with the tokens already known), logits of every step
    attention   a grouped-query attention layer on the paged cache: prompts, prompts in later pieces, one-token steps
    mlp         a gated feed-forward
    experts     a routed feed-forward, for the rows of a batched one-token step and for prompts
    latent      a latent attention layer over prompts
    recurrence  a gated linear recurrence over prompts, with the states that it leaves

Layer sizes are those of bench.py's shapes (Llama 3.2 1B and 3B, Llama 3.1 8B, Dofipel, Ganupel); inputs of the layers
are what a norm in front of them gives, N(0, 1); weights are N(0, 0.02)."""
import json
import math
import os
import random
import shutil
import tempfile

import torch

from llm_infer_engine_b200 import Engine
from llm_infer_engine_b200.cache import Cache
from llm_infer_engine_b200.config import PartSpec
from llm_infer_engine_b200.engine.context import StepContext
from llm_infer_engine_b200.engine.engine import bucket_for
from llm_infer_engine_b200.engine.plan import KernelPlan
from llm_infer_engine_b200.parts import Runtime, build_part
from llm_infer_engine_b200.weights.safetensors_io import save_file

DEV = torch.device("cuda", 0)
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
THETA = 500000.0
EPS = 1e-5
STD = 0.02

#         width, query heads, kv heads, head size, feed-forward
SHAPES = {"1b": (2048, 32, 8, 64, 8192), "3b": (3072, 24, 8, 128, 8192), "8b": (4096, 32, 8, 128, 14336)}
VOCAB = 32000                   # of the `answer` models: bench.py's tables use it


# ------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one user waiting for an answer: latency of the captured one-token step at batch 1
        {"name": "answer one", "kind": "answer", "dtype": "bfloat16", "shape": "1b", "layers": 4, "n": 1, "low": 90,
         "high": 110, "mix": 1, "new": 24},
        # a serving batch: ragged prompts in one step, then 16 lanes one token each
        {"name": "answer batch", "kind": "answer", "dtype": "bfloat16", "shape": "1b", "layers": 4, "n": 13, "low": 24,
         "high": 700, "mix": 2, "new": 24},
        # the true 32-bit engine (`--dtype float32`): what results are checked against
        {"name": "answer float32", "kind": "answer", "dtype": "float32", "shape": "1b", "layers": 2, "n": 3, "low": 30,
         "high": 200, "mix": 3, "new": 12},
        # one prompt of 2,048 tokens, the reference's headline prompt length
        {"name": "attention prompt", "kind": "attention", "dtype": "bfloat16", "shape": "1b", "n": 1, "low": 2048,
         "high": 2048, "held_low": 0, "held_high": 0, "mix": 4},
        # prompts cut into pieces: unequal new tokens behind unequal lengths already held, head size 128
        {"name": "attention pieces", "kind": "attention", "dtype": "bfloat16", "shape": "8b", "n": 6, "low": 60,
         "high": 1500, "held_low": 1, "held_high": 2500, "mix": 5},
        # a batch of 64 long conversations, one token each
        {"name": "attention step", "kind": "attention", "dtype": "bfloat16", "shape": "1b", "n": 64, "low": 1, "high": 1,
         "held_low": 700, "held_high": 3900, "mix": 6},
        # the 32-bit path's prompts
        {"name": "attention float32", "kind": "attention", "dtype": "float32", "shape": "1b", "n": 3, "low": 100,
         "high": 700, "held_low": 0, "held_high": 0, "mix": 7},
        {"name": "mlp float32", "kind": "mlp", "dtype": "float32", "shape": "1b", "rows": 301},
        # routed experts: a batched one-token step, and a prompt
        {"name": "experts step", "kind": "experts", "dtype": "bfloat16", "shape": "1b", "rows": 40},
        {"name": "experts prompt", "kind": "experts", "dtype": "bfloat16", "shape": "1b", "rows": 1777},
        # latent attention and a linear recurrence over prompts
        {"name": "latent prompt", "kind": "latent", "dtype": "bfloat16", "shape": "1b", "n": 2, "low": 600, "high": 1500,
         "mix": 8},
        {"name": "recurrence prompt", "kind": "recurrence", "dtype": "bfloat16", "shape": "1b", "n": 3, "low": 300,
         "high": 1200, "mix": 9},
    ]


def _between(rng, lo, hi):
    """A whole number, evenly spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _bounds(rng, lo, hi):
    a, b = _between(rng, lo, hi), _between(rng, lo, hi)
    return min(a, b), max(a, b)


def draw(rng):
    kind = rng.choice(["answer", "answer", "answer32", "prompt", "prompt", "step", "prompt32", "mlp", "experts", "latent",
                       "recurrence"])
    mix = rng.randrange(1 << 20)
    if kind == "answer":
        n = _between(rng, 1, 16)
        low, high = _bounds(rng, 8, 512)
        return {"kind": "answer", "dtype": "bfloat16", "shape": "1b", "layers": 4, "n": n, "low": low, "high": high,
                "mix": mix, "new": rng.randrange(8, 25)}
    if kind == "answer32":
        low, high = _bounds(rng, 8, 200)
        return {"kind": "answer", "dtype": "float32", "shape": "1b", "layers": 2, "n": _between(rng, 1, 6), "low": low,
                "high": high, "mix": mix, "new": rng.randrange(6, 13)}
    if kind == "prompt":
        n = _between(rng, 1, 8)
        low, high = _bounds(rng, 32, 4096 // n)
        held = _bounds(rng, 1, 2500) if rng.random() < 0.4 else (0, 0)
        return {"kind": "attention", "dtype": "bfloat16", "shape": rng.choice(["1b", "3b", "8b"]), "n": n, "low": low,
                "high": high, "held_low": held[0], "held_high": held[1], "mix": mix}
    if kind == "step":
        low, high = _bounds(rng, 200, 4000)
        return {"kind": "attention", "dtype": "bfloat16", "shape": rng.choice(["1b", "3b", "8b"]),
                "n": _between(rng, 24, 64), "low": 1, "high": 1, "held_low": low, "held_high": high, "mix": mix}
    if kind == "prompt32":
        n = _between(rng, 1, 4)
        low, high = _bounds(rng, 32, 1024 // n)
        return {"kind": "attention", "dtype": "float32", "shape": "1b", "n": n, "low": low, "high": high, "held_low": 0,
                "held_high": 0, "mix": mix}
    if kind == "mlp":
        return {"kind": "mlp", "dtype": "float32", "shape": "1b", "rows": _between(rng, 20, 512)}
    if kind == "experts":
        return {"kind": "experts", "dtype": "bfloat16", "shape": "1b", "rows": _between(rng, 16, 2048)}
    n = _between(rng, 1, 6)
    low, high = _bounds(rng, 64, 2048 // n)
    return {"kind": kind, "dtype": "bfloat16", "shape": "1b", "n": n, "low": low, "high": high, "mix": mix}


def _lens(case, low="low", high="high"):
    """Each sequence's length: `n` numbers evenly spread over the logarithm of [low, high], by the case's `mix`."""
    rng = random.Random("%d %s" % (case["mix"], low))
    if case[high] == 0:
        return [0] * case["n"]
    return [_between(rng, case[low], case[high]) for _ in range(case["n"])]


# ------------------------------------------------------------------------------------------ inputs
class _Random:
    """Tensors from one seed, made on the GPU in the order they are asked for."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 13)

    def normal(self, shape, std, dtype):
        t = torch.empty(shape, dtype=torch.float32, device=DEV).normal_(0.0, std, generator=self.g)
        return t.to(dtype)

    def uniform(self, shape, lo, hi, dtype):
        t = torch.empty(shape, dtype=torch.float32, device=DEV).uniform_(lo, hi, generator=self.g)
        return t.to(dtype)

    def ids(self, shape, n):
        return torch.randint(0, n, shape, generator=self.g, device=DEV, dtype=torch.int32)


def _llama_tensors(case, rnd):
    d, hq, hkv, hd, ff = SHAPES[case["shape"]]
    dt = DTYPES[case["dtype"]]
    out = {"model.embed_tokens.weight": rnd.normal((VOCAB, d), STD, dt), "model.norm.weight": rnd.uniform((d,), 0.8, 1.2, dt)}
    for i in range(case["layers"]):
        p = "model.layers.%d." % i
        out[p + "input_layernorm.weight"] = rnd.uniform((d,), 0.8, 1.2, dt)
        out[p + "post_attention_layernorm.weight"] = rnd.uniform((d,), 0.8, 1.2, dt)
        for name, shape in (("self_attn.q_proj", (hq * hd, d)), ("self_attn.k_proj", (hkv * hd, d)),
                            ("self_attn.v_proj", (hkv * hd, d)), ("self_attn.o_proj", (d, hq * hd)),
                            ("mlp.gate_proj", (ff, d)), ("mlp.up_proj", (ff, d)), ("mlp.down_proj", (d, ff))):
            out[p + name + ".weight"] = rnd.normal(shape, STD, dt)
    return out


def _answer_inputs(case, rnd):
    prompts = [rnd.ids((l,), VOCAB) for l in _lens(case)]
    return prompts, rnd.ids((case["new"], case["n"]), VOCAB)


def _attention_params(case):
    d, hq, hkv, hd, _ = SHAPES[case["shape"]]
    return {"hidden": d, "n_heads": hq, "n_kv_heads": hkv, "head_dim": hd, "window": 0, "scale": None,
            "position": PartSpec("rope", {"rot_dim": hd, "theta": THETA, "scaling": None})}


def _latent_params(case):
    d, hq, _, hd, _ = SHAPES[case["shape"]]
    rot = hd // 2
    return {"hidden": d, "n_heads": hq, "head_dim": hd, "rot_dim": rot, "v_head_dim": hd, "kv_rank": 4 * hd,
            "scale": (hd + rot) ** -0.5, "rot_base": 10000.0, "rot_dims": rot, "norm_eps": EPS, "gate": True,
            "out_float32": True}


def _recurrence_params(case):
    d, hq, _, hd, _ = SHAPES[case["shape"]]
    return {"hidden": d, "n_heads": hq, "dim": hd // 2, "v_dim": hd, "norm_eps": EPS}


def _expert_params(case):
    d, _, _, _, ff = SHAPES[case["shape"]]
    return {"hidden": d, "n_experts": 16, "top": 3, "expert_ff": ff // 4, "shared_ff": ff // 4}


def _part_shapes(case):
    """Checkpoint tensors of the case's part by name: (shape, how it is filled)."""
    d, hq, hkv, hd, ff = SHAPES[case["shape"]]
    kind, mat = case["kind"], "normal"
    if kind == "attention":
        return {"q_proj.weight": ((hq * hd, d), mat), "k_proj.weight": ((hkv * hd, d), mat),
                "v_proj.weight": ((hkv * hd, d), mat), "o_proj.weight": ((d, hq * hd), mat)}
    if kind == "mlp":
        return {"gate_proj.weight": ((ff, d), mat), "up_proj.weight": ((ff, d), mat), "down_proj.weight": ((d, ff), mat)}
    if kind == "experts":
        f = ff // 4
        out = {"router": ((16, d), mat), "router.b": ((16,), mat)}
        for e in ["e%d" % e for e in range(16)] + ["shared"]:
            out.update({e + ".gate": ((f, d), mat), e + ".up": ((f, d), mat), e + ".down": ((d, f), mat)})
        return out
    if kind == "latent":
        rot, rank = hd // 2, 4 * hd
        return {"q": ((hq * (hd + rot), d), mat), "dkv": ((rank + rot, d), mat), "dkv.norm": ((rank,), (0.8, 1.2)),
                "uk": ((hq * hd, rank), mat), "uv": ((hq * hd, rank), mat), "g": ((hq * hd, d), mat),
                "o": ((d, hq * hd), mat)}
    D = hd // 2
    return {"q": ((hq * D, d), mat), "f": ((hq * D, d), mat), "f.b": ((hq * D,), (-1.0, 3.0)),
            "lower": ((hq * D,), (0.0, 0.9)), "v": ((hq * hd, d), mat), "norm": ((hd,), (0.8, 1.2)),
            "o": ((d, hq * hd), mat)}


PARTS = {"attention": ("mixer", "gqa_attention", _attention_params), "mlp": ("feed_forward", "swiglu", lambda c: {
    "hidden": SHAPES[c["shape"]][0], "intermediate": SHAPES[c["shape"]][4]}),
    "experts": ("feed_forward", "routed_experts", _expert_params), "latent": ("mixer", "latent_attention", _latent_params),
    "recurrence": ("mixer", "gated_linear_recurrence", _recurrence_params)}


def _part_inputs(case, seed):
    """(weights by name, lengths already held, new lengths, input rows of all positions, the held ones of every
    sequence first)."""
    rnd, dt = _Random(seed), DTYPES[case["dtype"]]
    w = {name: rnd.normal(shape, STD, dt) if how == "normal" else rnd.uniform(shape, how[0], how[1], dt)
         for name, (shape, how) in _part_shapes(case).items()}
    if "rows" in case:
        held, new = [0], [case["rows"]]
    else:
        new = _lens(case)
        held = _lens(case, "held_low", "held_high") if "held_low" in case else [0] * len(new)
    x_held = rnd.normal((sum(held), SHAPES[case["shape"]][0]), 1.0, dt) if sum(held) else None
    return w, held, new, x_held, rnd.normal((sum(new), SHAPES[case["shape"]][0]), 1.0, dt)


class _Plan:
    """What KernelPlan asks of an engine."""

    def __init__(self, dtype):
        self.dtype, self.decode_attention = dtype, "auto"


def _context(starts, lens, slots, dtype, plan):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)              # noqa: E731
    T, cu = sum(lens), [0]
    for l in lens:
        cu.append(cu[-1] + l)
    ends = [s + l for s, l in zip(starts, lens)]
    return StepContext(n_tokens=T, n_seqs=len(lens), decode=max(lens) == 1, max_q_len=max(lens), max_kv_len=max(ends),
                       tokens=i32([0] * T), tok_pos=i32([s + j for s, l in zip(starts, lens) for j in range(l)]),
                       tok_seq=i32([i for i, l in enumerate(lens) for _ in range(l)]), cu_q=i32(cu), seq_slot=i32(slots),
                       seq_start=i32(starts), seq_kvlen=i32(ends), logit_rows=i32(list(range(T))), dtype=dtype, device=DEV,
                       kernels=plan, all_rows=True)


# ------------------------------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    dt = DTYPES[case["dtype"]]
    if case["kind"] == "answer":
        d, hq, hkv, hd, ff = SHAPES[case["shape"]]
        rnd = _Random(seed)
        tensors = {k: t.cpu() for k, t in _llama_tensors(case, rnd).items()}
        prompts, given = _answer_inputs(case, rnd)
        longest = max(_lens(case)) + case["new"]
        config = {"architectures": ["LlamaForCausalLM"], "hidden_size": d, "num_hidden_layers": case["layers"],
                  "num_attention_heads": hq, "num_key_value_heads": hkv, "head_dim": hd, "intermediate_size": ff,
                  "vocab_size": VOCAB, "rms_norm_eps": EPS, "rope_theta": THETA, "max_position_embeddings": 4096,
                  "tie_word_embeddings": True, "hidden_act": "silu", "eos_token_id": None, "torch_dtype": case["dtype"]}
        folder = tempfile.mkdtemp(prefix="cases_", dir="/dev/shm" if os.path.isdir("/dev/shm") else None)
        try:
            with open(os.path.join(folder, "config.json"), "w") as f:
                json.dump(config, f)
            save_file(tensors, os.path.join(folder, "model.safetensors"))
            engine = Engine(folder, dtype=case["dtype"], device=0, max_batch=case["n"], max_seq_len=longest + 1)
        finally:
            shutil.rmtree(folder, ignore_errors=True)
        graph = engine.decode_graph(bucket_for(case["n"]), longest)
        return {"kind": "answer", "engine": engine, "graph": graph, "prompts": [p.tolist() for p in prompts],
                "given": given}
    group, name, params = PARTS[case["kind"]]
    w, held, new, x_held, x = _part_inputs(case, seed)
    longest = max(h + n for h, n in zip(held, new))
    part = build_part(group, PartSpec(name, params(case)), Runtime(device=DEV, dtype=dt, max_positions=longest))
    part.load(w)
    plan = KernelPlan(_Plan(dt))
    state = {"kind": case["kind"], "part": part, "x": x}
    if group == "feed_forward":
        state["ctx"] = _context([0], [case["rows"]], [0], dt, plan)
        return state
    pages = sum((h + n + 63) // 64 for h, n in zip(held, new))
    cache = Cache([part.cache_requests()], len(new), 64 * pages, longest, dt, DEV)
    slots = [cache.take_slot() for _ in new]
    for s, h, n in zip(slots, held, new):
        cache.reserve(s, h + n)
    state.update(cache=cache, unit=cache.unit(0), ctx=_context(held, new, slots, dt, plan))
    if x_held is not None:
        at = [i for i, h in enumerate(held) if h]
        ctx = _context([0] * len(at), [held[i] for i in at], [slots[i] for i in at], dt, plan)
        part.forward(x_held, ctx, cache.unit(0), True)
    if case["kind"] == "recurrence":
        state["S"], state["rows"] = cache.unit(0).state["S"], torch.tensor(slots, device=DEV)
    return state


def run(state):
    if state["kind"] == "answer":
        engine, graph, prompts = state["engine"], state["graph"], state["prompts"]
        cache, n = engine.cache, len(prompts)
        slots = [engine.open() for _ in prompts]
        out = [engine.step(slots, prompts, "last")]
        graph.set_lanes(slots)
        for tokens in state["given"]:
            for s in slots:
                cache.reserve(s, cache.lengths[s] + 1)
            graph.tokens[:n].copy_(tokens)
            out.append(graph.replay()[:n].clone())
            for s in slots:
                cache.note_appended(s, cache.lengths[s] + 1, device_updated=True)
        for s in slots:
            engine.close(s)
        return torch.stack(out)
    part, ctx, x = state["part"], state["ctx"], state["x"]
    if state["kind"] in ("mlp", "experts"):
        return part.forward(x, ctx)
    if state["kind"] == "recurrence":
        state["S"].zero_()                        # new sequences: their states start from zero
        y = part.forward(x, ctx, state["unit"], True)
        return y, state["S"][state["rows"]]
    return part.forward(x, ctx, state["unit"], True)


# ------------------------------------------------------------------------------------------ the same in 64 bits
def _rope(x, positions, hd):
    """x [T, heads, hd] rotated by halves; frequencies and angles are float32 by definition."""
    inv = 1.0 / (THETA ** (torch.arange(0, hd, 2).float() / hd))
    angle = (positions.float()[:, None].cpu() * inv[None, :]).double().to(DEV)
    cos, sin = angle.cos()[:, None, :], angle.sin()[:, None, :]
    a, b = x[..., :hd // 2], x[..., hd // 2:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _attend(q, k, v, start, scale):
    """q [Tq, H, D] at positions start.., k [Tk, Hkv, D], v [Tk, Hkv, Dv]: causal softmax attention, some rows at a time."""
    Tq, H, _ = q.shape
    Tk, Hkv, Dv = v.shape
    k, v = k.permute(1, 2, 0), v.permute(1, 0, 2)
    out = torch.empty((Tq, H, Dv), dtype=torch.float64, device=DEV)
    g = H // Hkv
    for a in range(0, Tq, 512):
        b = min(Tq, a + 512)
        n = start + b
        qs = q[a:b].reshape(b - a, Hkv, g, -1).permute(1, 2, 0, 3).reshape(Hkv, g * (b - a), -1)
        s = torch.bmm(qs, k[..., :n]) * scale
        far = torch.arange(n, device=DEV)[None, :] > (start + torch.arange(a, b, device=DEV))[:, None]
        s = s.view(Hkv, g, b - a, n).masked_fill(far, -math.inf).softmax(-1).view(Hkv, g * (b - a), n)
        out[a:b] = torch.bmm(s, v[:, :n]).view(Hkv, g, b - a, Dv).permute(2, 0, 1, 3).reshape(b - a, H, Dv)
    return out


def _rms(x, w):
    return x / (x.square().mean(-1, keepdim=True) + EPS).sqrt() * w


def _silu(x):
    return x * torch.sigmoid(x)


def exact(case, seed):
    d, hq, hkv, hd, ff = SHAPES[case["shape"]]
    if case["kind"] == "answer":
        rnd = _Random(seed)
        w = {k: t.double() for k, t in _llama_tensors(case, rnd).items()}
        prompts, given = _answer_inputs(case, rnd)
        new = case["new"]
        seqs = [torch.cat([p, given[:, i]]) for i, p in enumerate(prompts)]
        cuts = [0]
        for s in seqs:
            cuts.append(cuts[-1] + len(s))
        h = w["model.embed_tokens.weight"][torch.cat(seqs).long()]
        for i in range(case["layers"]):
            p = "model.layers.%d." % i
            u = _rms(h, w[p + "input_layernorm.weight"])
            q, k, v = (u @ w[p + "self_attn.%s_proj.weight" % n].T for n in "qkv")
            o = torch.empty_like(q)
            for a, b in zip(cuts, cuts[1:]):
                pos = torch.arange(b - a, device=DEV)
                o[a:b] = _attend(_rope(q[a:b].view(b - a, hq, hd), pos, hd), _rope(k[a:b].view(b - a, hkv, hd), pos, hd),
                                 v[a:b].view(b - a, hkv, hd), 0, hd ** -0.5).reshape(b - a, hq * hd)
            h = h + o @ w[p + "self_attn.o_proj.weight"].T
            u = _rms(h, w[p + "post_attention_layernorm.weight"])
            h = h + (_silu(u @ w[p + "mlp.gate_proj.weight"].T) * (u @ w[p + "mlp.up_proj.weight"].T)) \
                @ w[p + "mlp.down_proj.weight"].T
        rows = torch.stack([torch.arange(b - new - 1, b, device=DEV) for b in cuts[1:]], dim=1)        # [new + 1, n]
        return _rms(h[rows], w["model.norm.weight"]) @ w["model.embed_tokens.weight"].T
    w, held, new, x_held, x = _part_inputs(case, seed)
    w, x = {k: t.double() for k, t in w.items()}, x.double()
    if case["kind"] == "mlp":
        return (_silu(x @ w["gate_proj.weight"].T) * (x @ w["up_proj.weight"].T)) @ w["down_proj.weight"].T
    if case["kind"] == "experts":
        def expert(name, u):
            return (_silu(u @ w[name + ".gate"].T) * (u @ w[name + ".up"].T)) @ w[name + ".down"].T
        best = (x @ w["router"].T + w["router.b"]).topk(3, dim=1)
        share = best.values.softmax(1)
        out = expert("shared", x)
        for e in range(16):
            t, c = (best.indices == e).nonzero(as_tuple=True)
            out[t] += share[t, c][:, None] * expert("e%d" % e, x[t])
        return out
    outs, at, at_held, states = [], 0, 0, []
    for h_len, n in zip(held, new):
        u = x[at:at + n]
        if h_len:
            u = torch.cat([x_held[at_held:at_held + h_len].double(), u])
        at, at_held = at + n, at_held + h_len
        T = h_len + n
        pos = torch.arange(T, device=DEV)
        if case["kind"] == "attention":
            q = _rope((u[h_len:] @ w["q_proj.weight"].T).view(n, hq, hd), pos[h_len:], hd)
            k = _rope((u @ w["k_proj.weight"].T).view(T, hkv, hd), pos, hd)
            o = _attend(q, k, (u @ w["v_proj.weight"].T).view(T, hkv, hd), h_len, hd ** -0.5)
            outs.append(o.reshape(n, -1) @ w["o_proj.weight"].T)
        elif case["kind"] == "latent":
            p = _latent_params(case)
            rank, rot = p["kv_rank"], p["rot_dim"]
            angle = pos.double()[:, None] * (10000.0 ** (-2.0 * torch.arange(rot // 2, device=DEV, dtype=torch.float64) / rot))
            cos, sin = angle.cos()[:, None, :], angle.sin()[:, None, :]

            def turn(t):                           # [T, heads, rot]: pairs (2i, 2i + 1)
                a, b = t[..., 0::2], t[..., 1::2]
                return torch.stack([a * cos - b * sin, a * sin + b * cos], dim=-1).flatten(-2)
            q = (u @ w["q"].T).view(T, hq, hd + rot)
            lat = u @ w["dkv"].T
            c = _rms(lat[:, :rank], w["dkv.norm"])
            k_rot = turn(lat[:, None, rank:]).expand(T, hq, rot)
            k = torch.cat([(c @ w["uk"].T).view(T, hq, hd), k_rot], dim=-1)
            q = torch.cat([q[..., :hd], turn(q[..., hd:])], dim=-1)
            o = _attend(q, k, (c @ w["uv"].T).view(T, hq, hd), 0, p["scale"]).reshape(T, -1)
            outs.append((o * torch.sigmoid(u @ w["g"].T)) @ w["o"].T)
        else:
            D = hd // 2
            q = _silu(u @ w["q"].T).view(T, hq, D)
            f = (w["lower"] + (1 - w["lower"]) * torch.sigmoid(u @ w["f"].T + w["f.b"])).view(T, hq, D)
            v = (u @ w["v"].T).view(T, hq, hd)
            S, o = torch.zeros((hq, D, hd), dtype=torch.float64, device=DEV), []
            for t in range(T):
                S = f[t][:, :, None] * S + (1 - f[t])[:, :, None] * v[t][:, None, :]
                o.append(torch.bmm(q[t][:, None, :], S)[:, 0])
            outs.append(_rms(torch.stack(o), w["norm"]).reshape(T, -1) @ w["o"].T)
            states.append(S)
    return (torch.cat(outs), torch.stack(states)) if states else torch.cat(outs)


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    d, hq, hkv, hd, ff = SHAPES[case["shape"]]
    e = 4 if case["dtype"] == "float32" else 2
    if case["kind"] == "answer":
        per_layer = d * (hq + 2 * hkv) * hd + d * hq * hd + 3 * d * ff
        weights, lens, new, L = case["layers"] * per_layer, _lens(case), case["new"], case["layers"]
        pairs = sum(l * (l + 1) // 2 + sum(range(l + 1, l + new + 1)) for l in lens)
        keys = sum(l + sum(range(l + 1, l + new + 1)) for l in lens)
        rows = case["n"] * (new + 1)
        return {"bytes": (new + 1) * (weights + VOCAB * d) * e + 2 * L * keys * hkv * hd * e + rows * VOCAB * 4,
                "flops": 2 * weights * (sum(lens) + case["n"] * new) + 2 * rows * VOCAB * d + 4 * L * pairs * hq * hd}
    weights = {name: math.prod(shape) for name, (shape, _) in _part_shapes(case).items()}
    total = sum(weights.values())
    if case["kind"] == "mlp":
        return {"bytes": (total + 2 * case["rows"] * d) * e, "flops": 2 * total * case["rows"]}
    if case["kind"] == "experts":
        rows, one = case["rows"], 3 * d * ff // 4
        hit = 16 * (1 - (1 - 3 / 16) ** rows) + 1          # experts that some row chooses, and the shared one
        return {"bytes": (hit * one + 16 * d) * e + rows * d * (e + 4), "flops": 2 * rows * (4 * one + 16 * d)}
    new = _lens(case)
    held = _lens(case, "held_low", "held_high") if "held_low" in case else [0] * len(new)
    T, pairs = sum(new), sum(n * h + n * (n + 1) // 2 for h, n in zip(held, new))
    if case["kind"] == "attention":
        return {"bytes": (total + 2 * T * d + 2 * hkv * hd * (sum(held) + T)) * e,
                "flops": 2 * total * T + 4 * pairs * hq * hd}
    if case["kind"] == "latent":
        return {"bytes": total * e + T * d * (e + 4) + T * 4.5 * hd * e,
                "flops": 2 * total * T + 2 * pairs * hq * (2 * hd + hd // 2)}
    state = hq * (hd // 2) * hd
    return {"bytes": total * e + T * d * (e + 4) + len(new) * state * 4, "flops": 2 * total * T + 5 * T * state}


def tolerance(case):
    """What another correct implementation at the same precision may be off by: about four times the change that sums in
    another order make (32-bit sums 4e-6 over whole models, bfloat16 layers 3e-3 to 5e-3, bfloat16 models 1e-2)."""
    if case["dtype"] == "float32":
        return {"rel": 1.5e-5, "max": 2e-4}
    return {"rel": 3e-2, "max": 3e-1} if case["kind"] == "answer" else {"rel": 2e-2, "max": 2e-1}
