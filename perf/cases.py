"""The work whose speed counts: steps of the engine as a serving program runs them.

A program keeps a model loaded (``ModelRunner``: weights, cache pool, step function) and calls ``step`` with any mix of
prompt portions and decoded tokens; it gets 32-bit logits at the wanted places.  A case is one such call (or, for the
designs whose layers carry a state, a whole short turn of calls) on a model of a named size:

  decode   one more token for each of ``requests`` live requests whose contexts end at ``context`` (all of them, or spread
           over the upper three quarters of it where ``ragged``);
  prefill  ``requests`` new prompts of ``tokens`` tokens (ragged: the later ones shorter) in one step, logits of their last;
  mixed    a portion of ``tokens`` tokens of a prompt that is already ``context`` // 2 tokens in, beside one decoded token for
           each of ``requests`` others: the step of continuous batching with prompts cut into portions;
  turn     ``requests`` new prompts of ``tokens`` tokens, then ``steps`` decoded tokens each, logits of every step.

Weights are seeded random ones of the architecture (one set per model and precision), token ids are uniform and depend on
the seed.  ``exact`` states the same models in 64 bits with plain torch on whole sequences, without a cache.
"""
import functools
import json
import math
import os
import shutil
import struct
import tempfile
import weakref

import numpy as np
import torch

PAGE = 16
POSITIONS = 1024
F64 = torch.float64


# ---------------------------------------------------------------------------------------------------------- the models
def _gpt2(layers, width, heads):
    return dict(architectures=["GPT2LMHeadModel"], model_type="gpt2", n_layer=layers, n_embd=width, n_head=heads,
                n_inner=4 * width, vocab_size=50257, n_positions=POSITIONS, layer_norm_epsilon=1e-5,
                activation_function="gelu_new", eos_token_id=50256)


def _finuvik():
    mixer = dict(left=dict(heads=12, kv_heads=4, dim=64, vdim=64, scale=0.125, q_temp=dict(coef=0.1, every=256)),
                 left_scale=1.0, right=dict(heads=3, dim=32, vdim=128), right_scale=1.0)
    return dict(architecture="Finuvik", width=768, vocab=32000, max_positions=POSITIONS, norm=dict(eps=1e-5),
                layers=[dict(type="parallel", mixer=mixer, mlp=dict(ff=2048, kind="dense")) for _ in range(4)])


def _falisun():
    ffn = dict(kind="moe", router=dict(experts=8, top=2, groups=dict(count=4, keep=2)), expert=dict(ff=512),
               shared=dict(ff=1024))
    rot = dict(base=10000.0, dims=32, scaling=dict(factor=8.0, original=512, fast=32.0, slow=1.0))
    state = dict(heads=24, vdim=64, state=128, groups=1, conv=4, norm_groups=1)
    latent = dict(heads=12, dim=64, rot_dim=32, vdim=64, kv_rank=384, scale=96 ** -0.5, rot=rot)
    return dict(architecture="Falisun", width=768, vocab=32000, norm=dict(eps=1e-5),
                layers=[dict(type="mamba2", mixer=state, mlp=ffn), dict(type="latent_attention", mixer=latent, mlp=ffn),
                        dict(type="mamba2", mixer=state, mlp=ffn),
                        dict(type="latent_attention", mixer=dict(latent, kv_from=1), mlp=ffn)])


MODELS = {"gpt2-small": _gpt2(12, 768, 12), "gpt2-medium": _gpt2(24, 1024, 16), "gpt2-xl": _gpt2(48, 1600, 25),
          "finuvik": _finuvik(), "falisun": _falisun()}


def _vocab(model):
    return MODELS[model].get("vocab_size") or MODELS[model]["vocab"]


# ----------------------------------------------------------------------------------------------------------- the cases
def _case(name, model, dtype, kind, requests, tokens=0, context=0, ragged=False, steps=0):
    case = dict(model=model, dtype=dtype, kind=kind, requests=requests, tokens=tokens, context=context, ragged=ragged,
                steps=steps)
    return dict(case, name=name) if name else case


def listed():
    return [
        # one conversation: what a single user waits for between two tokens
        _case("small-bf16-decode-1", "gpt2-small", "bfloat16", "decode", 1, context=517),
        # the benchmark's headline batch in the reference's precision, half way through its 512 tokens
        _case("small-fp32-decode-8", "gpt2-small", "float32", "decode", 8, context=768),
        # a server under load: 64 requests at different places in their conversations
        _case("small-bf16-decode-64", "gpt2-small", "bfloat16", "decode", 64, context=1000, ragged=True),
        _case("small-fp32-decode-64", "gpt2-small", "float32", "decode", 64, context=768),
        # a short question: time to the first token
        _case("small-bf16-prefill-77", "gpt2-small", "bfloat16", "prefill", 1, tokens=77),
        # the benchmark's prompt step, 2 x 1024 tokens, in both precisions
        _case("small-bf16-prefill-2048", "gpt2-small", "bfloat16", "prefill", 2, tokens=1024),
        _case("small-fp32-prefill-2048", "gpt2-small", "float32", "prefill", 2, tokens=1024),
        # continuous batching on the medium model: a 512-token portion of a prompt beside 40 decoding requests
        _case("medium-fp32-mixed-552", "gpt2-medium", "float32", "mixed", 40, tokens=512, context=900, ragged=True),
        _case("medium-bf16-mixed-552", "gpt2-medium", "bfloat16", "mixed", 40, tokens=512, context=900, ragged=True),
        # the largest model near the end of its contexts, as many requests as its pool of 24 contexts holds
        _case("xl-bf16-decode-24", "gpt2-xl", "bfloat16", "decode", 24, context=1023),
        # the designs with a state per request, as whole turns: a recurrence beside attention, dense feed-forwards;
        # state-space layers, latent attention and routed experts
        _case("finuvik-bf16-turn-4", "finuvik", "bfloat16", "turn", 4, tokens=500, steps=16),
        _case("falisun-fp32-turn-3", "falisun", "float32", "turn", 3, tokens=250, steps=8),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    model = rng.choice(["gpt2-small"] * 5 + ["gpt2-medium"] * 2 + ["gpt2-xl", "finuvik", "falisun"])
    dtype = rng.choice(["float32", "bfloat16"])
    if model in ("finuvik", "falisun"):
        # routed experts only in 32 bits: where a 16-bit rounding moves a choice of expert, two right answers differ
        dtype = "float32" if model == "falisun" else dtype
        requests = rng.randint(1, 8)
        return _case(None, model, dtype, "turn", requests, tokens=_log_uniform(rng, 16, 1000 // requests),
                     steps=rng.randint(2, 12))
    if model == "gpt2-xl":
        return _case(None, model, "bfloat16", "decode", _log_uniform(rng, 1, 24), context=rng.randint(32, 1023),
                     ragged=rng.random() < 0.5)
    kind = rng.choice(["decode", "decode", "prefill", "mixed"])
    if kind == "decode":
        return _case(None, model, dtype, "decode", _log_uniform(rng, 1, 64 if model == "gpt2-small" else 32),
                     context=rng.randint(32, 1023), ragged=rng.random() < 0.5)
    if kind == "prefill":
        requests = rng.randint(1, 4)
        most = 2048 if model == "gpt2-small" else 512
        return _case(None, model, dtype, "prefill", requests, tokens=_log_uniform(rng, 16, min(1024, most // requests)),
                     ragged=rng.random() < 0.5)
    return _case(None, model, dtype, "mixed", _log_uniform(rng, 2, 40), tokens=_log_uniform(rng, 32, 512),
                 context=rng.randint(64, 1023), ragged=rng.random() < 0.5)


# -------------------------------------------------------------------------------------------------- what a case consists of
def _lengths(case):
    """(tokens already computed, new tokens) of every request of the step."""
    n, c = case["requests"], case["context"]
    if case["kind"] in ("prefill", "turn"):
        t = case["tokens"]
        return [(0, max(1, t - (i * t) // (2 * n) if case["ragged"] else t)) for i in range(n)]
    spread = [c - (3 * c * i) // (4 * n) if case["ragged"] else c for i in range(n)]
    old = [(max(1, s), 1) for s in spread]
    if case["kind"] == "mixed":
        start = min(c // 2, POSITIONS - case["tokens"])
        old = [(start, case["tokens"])] + old
    return old


def _sequences(case, seed):
    """Token ids of every request: the old ones, the new ones and (turn) the given decoded ones."""
    g = torch.Generator().manual_seed(int(seed) * 1000003 + 17)
    v = _vocab(case["model"])
    return [torch.randint(0, v, (a + b + case["steps"],), generator=g, dtype=torch.int32).numpy() for a, b in _lengths(case)]


@functools.lru_cache(maxsize=None)
def _folder(model, dtype):
    """A model folder with seeded random weights, written once and then found again, as a checkpoint on disk is."""
    import mini_llm_b200 as m
    home = os.path.join(tempfile.gettempdir(), f"mini_llm_models_{os.getuid()}")
    place = os.path.join(home, f"{model}-{dtype}")
    if not os.path.isfile(os.path.join(place, "model.safetensors")):
        os.makedirs(home, exist_ok=True)
        draft = tempfile.mkdtemp(dir=home)
        m.write_random_model(dict(MODELS[model]), 0, draft, dtype=dtype)
        try:
            os.rename(draft, place)
        except OSError:
            shutil.rmtree(draft)          # another process was quicker
    return place


@functools.lru_cache(maxsize=1)
def _runner(model, dtype, seqs, tokens, batched):
    from mini_llm_b200.config.base import EngineConfig
    from mini_llm_b200.engine.runner import ModelRunner
    return ModelRunner(_folder(model, dtype), EngineConfig(dtype=dtype, page_size=PAGE, max_tokens=tokens, max_num_seqs=seqs,
                                                           max_num_batched_tokens=batched))


class _State:
    """The requests of a case in a runner; they leave it when the state is dropped."""

    def __init__(self, runner, case, names, rows):
        self.runner, self.case, self.names, self.rows = runner, case, names, rows
        self.entries = self.logits = None
        weakref.finalize(self, _leave, runner, names)


def _leave(runner, names):
    for r in names:
        if runner.has_request(r):
            runner.finish_request(r)


def prepare(case, seed):
    from mini_llm_b200.engine.runner import StepEntry
    lengths, rows = _lengths(case), _sequences(case, seed)
    pages = sum(-(-len(r) // PAGE) for r in rows)
    # room for a few such sets of requests side by side, as a pool has
    runner = _runner(case["model"], case["dtype"], 4 * len(rows), 4 * pages * PAGE, max(2048, sum(b for _, b in lengths)))
    names = [object() for _ in rows]
    state = _State(runner, case, names, rows)
    if case["kind"] in ("decode", "mixed"):
        for r in names:
            runner.add_request(r)
        batch, room = [], 2048
        for r, ids, (a, _) in zip(names, rows, lengths):       # the contexts, as prompt steps of at most 2,048 tokens
            if batch and a > room:
                runner.step(batch)
                batch, room = [], 2048
            batch.append(StepEntry(r, ids[:a]))
            room -= a
        runner.step(batch)
    state.entries = [StepEntry(r, ids[a:a + b], [b - 1]) for r, ids, (a, b) in zip(names, rows, lengths)]
    if case["kind"] == "turn":
        state.logits = torch.empty(case["steps"] + 1, len(rows), _vocab(case["model"]), dtype=torch.float32,
                                   device=runner.device)
        state.decoded = [[StepEntry(r, ids[b + i:b + i + 1], [0]) for r, ids, (_, b) in zip(names, rows, lengths)]
                         for i in range(case["steps"])]
    return state


def run(state):
    runner = state.runner
    if state.case["kind"] in ("decode", "mixed"):
        # the caller keeps the count of the tokens that are in, as a scheduler does; here the same tokens come again
        return runner.step(state.entries, commit=False)
    for r in state.names:
        runner.add_request(r)
    logits = runner.step(state.entries)
    if state.case["kind"] == "turn":
        state.logits[0].copy_(logits)
        for i, entries in enumerate(state.decoded):
            state.logits[i + 1].copy_(runner.step(entries))
        logits = state.logits
    for r in state.names:
        runner.finish_request(r)
    return logits


# ------------------------------------------------------------------------------------------------ bytes, flops, tolerances
@functools.lru_cache(maxsize=None)
def _matrices(model):
    """(entries of the matrices that every token passes, entries of the routed experts, share of the experts that a token
    passes, entries of all other parameters but the embedding tables, entries of the head)."""
    cfg = MODELS[model]
    if model.startswith("gpt2"):
        D, L = cfg["n_embd"], cfg["n_layer"]
        return L * 12 * D * D, 0, 0.0, L * 13 * D + 2 * D, _vocab(model) * D
    D, dense, experts, rest = cfg["width"], 0, 0, cfg["width"]
    for layer in cfg["layers"]:
        m, f = layer["mixer"], layer["mlp"]
        if layer["type"] == "parallel":
            a, b = m["left"], m["right"]
            dense += D * (2 * a["heads"] * a["dim"] + a["kv_heads"] * (a["dim"] + a["vdim"]))
            dense += D * b["heads"] * (2 * b["dim"] + 2 * b["vdim"]) + 3 * D * f["ff"]
            rest += 2 * D + 2 * a["heads"] + b["heads"] * (2 * b["dim"] + b["vdim"])
            continue
        if layer["type"] == "mamba2":
            inner, bc = m["heads"] * m["vdim"], 2 * m["groups"] * m["state"]
            dense += D * (2 * inner + bc + m["heads"]) + inner * D
            rest += (m["conv"] + 1) * (inner + bc) + 3 * m["heads"] + inner
        else:
            H, R = m["heads"], m["kv_rank"]
            dense += D * H * (m["dim"] + m["rot_dim"]) + H * (m["dim"] + m["vdim"]) * R + 2 * D * H * m["vdim"]
            dense += 0 if "kv_from" in m else D * (R + m["rot_dim"])
        dense += D * f["router"]["experts"] + 3 * D * f["shared"]["ff"]
        experts += 3 * D * f["expert"]["ff"] * f["router"]["experts"]
        rest += 6 * D
    top = 0.25 if experts else 0.0
    return dense, experts, top, rest, _vocab(model) * D


def _kept_per_token(model):
    """Values that a token leaves in the cache, and attention flops per (token, key)."""
    cfg = MODELS[model]
    if model.startswith("gpt2"):
        return 2 * cfg["n_layer"] * cfg["n_embd"], 4 * cfg["n_layer"] * cfg["n_embd"]
    if model == "finuvik":
        return 4 * 2 * 4 * 64, 4 * 4 * 12 * 64
    return 384 + 32, 2 * 2 * 12 * (96 + 64)


def work(case):
    """Weights read once per step, the cache read where old tokens are and written where new ones are, logits written."""
    es = 2 if case["dtype"] == "bfloat16" else 4
    dense, experts, top, rest, head = _matrices(case["model"])
    kept, per_key = _kept_per_token(case["model"])
    vocab = _vocab(case["model"])
    nbytes = flops = 0.0
    steps = [_lengths(case)] + [[(b + i, 1) for _, b in _lengths(case)] for i in range(case["steps"])]
    for lengths in steps:
        T, R = sum(b for _, b in lengths), len(lengths)
        width = head // vocab
        nbytes += (dense + head) * es + 4 * rest + T * (width * es + 12)
        nbytes += experts * es * (1.0 - (1.0 - top) ** T)
        nbytes += sum(a + b for a, b in lengths) * kept * es + 4.0 * R * vocab
        flops += 2.0 * T * (dense + experts * top) + 2.0 * R * head
        flops += sum(per_key * (a * b + b * (b + 1) / 2.0) for a, b in lengths)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what the steps are off ``exact``: 4e-7 to 2e-6 in 32 bits, 4e-3 to 5e-3 with bfloat16 storage."""
    return {"rel": 8e-6, "max": 2e-4} if case["dtype"] == "float32" else {"rel": 1.8e-2, "max": 2e-1}


# ---------------------------------------------------------------------------------------------- the models in 64 bits
def _tensors(model, dtype):
    """The weights of the folder by name, in 64 bits on the GPU (a safetensors file: header length, header, values)."""
    path = os.path.join(_folder(model, dtype), "model.safetensors")
    kinds = {"F32": np.float32, "BF16": np.uint16}
    with open(path, "rb") as f:
        (n,) = struct.unpack("<Q", f.read(8))
        header = json.loads(f.read(n))
    raw = np.memmap(path, dtype=np.uint8, mode="r", offset=8 + n)
    out = {}
    for name, e in header.items():
        if name == "__metadata__":
            continue
        a = np.array(raw[e["data_offsets"][0]:e["data_offsets"][1]]).view(kinds[e["dtype"]])
        t = torch.from_numpy(a.view(np.int16) if e["dtype"] == "BF16" else a).cuda()
        out[name.replace("transformer.", "")] = (t.view(torch.bfloat16) if e["dtype"] == "BF16" else t).view(e["shape"]).to(F64)
    return out


def _softmax_attention(q, k, v, scale, bias=None):
    """q [H, T, d], k [H, T, d], v [H, T, e] -> [T, H * e], causal."""
    T = q.shape[1]
    out = []
    hidden = torch.ones(T, T, dtype=torch.bool, device=q.device).triu(1)
    for h in range(q.shape[0]):
        s = q[h] @ k[h].t() * scale
        s = s if bias is None else s - bias(h)
        out.append(torch.softmax(s.masked_fill(hidden, -math.inf), -1) @ v[h])
    return torch.cat(out, -1)


def _heads(x, n):
    return x.view(x.shape[0], n, -1).transpose(0, 1)


def _gpt2_exact(t, cfg, ids):
    def norm(x, p):
        return torch.nn.functional.layer_norm(x, x.shape[-1:], t[p + ".weight"], t[p + ".bias"], cfg["layer_norm_epsilon"])

    def linear(x, p):
        return x @ t[p + ".weight"] + t[p + ".bias"]

    D, H = cfg["n_embd"], cfg["n_head"]
    x = t["wte.weight"][ids] + t["wpe.weight"][:len(ids)]
    for i in range(cfg["n_layer"]):
        p = f"h.{i}."
        q, k, v = (_heads(y, H) for y in linear(norm(x, p + "ln_1"), p + "attn.c_attn").split(D, -1))
        x = x + linear(_softmax_attention(q, k, v, (D // H) ** -0.5), p + "attn.c_proj")
        h = torch.nn.functional.gelu(linear(norm(x, p + "ln_2"), p + "mlp.c_fc"), approximate="tanh")
        x = x + linear(h, p + "mlp.c_proj")
    return norm(x, "ln_f"), t["wte.weight"]


def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _finuvik_exact(t, cfg, ids):
    """x += softmax attention with a distance penalty + a gated recurrence + a gated ReLU feed-forward, all of normed x."""
    eps, n = cfg["norm"]["eps"], len(ids)
    at = torch.arange(n, device=t["embed"].device)
    apart = (at[:, None] - at[None, :]).clamp(min=0).to(F64)
    x = t["embed"][ids] + t["pos"][:n]
    for i, layer in enumerate(cfg["layers"]):
        p, a, b = f"l{i}.", layer["mixer"]["left"], layer["mixer"]["right"]
        h = _rms(x, 1.0 + t[p + "norm1"], eps)
        m = p + "mix.left."
        warm = 1.0 + a["q_temp"]["coef"] * torch.log1p(torch.div(at + 1, a["q_temp"]["every"], rounding_mode="floor").to(F64))
        q = _heads(h @ t[m + "q"].t(), a["heads"]) * warm[None, :, None]
        k, v = (_heads(h @ t[m + c].t(), a["kv_heads"]).repeat_interleave(a["heads"] // a["kv_heads"], 0) for c in "kv")
        o = _softmax_attention(q, k, v, a["scale"], lambda j: t[m + "r1"][j] * torch.log1p(t[m + "r2"][j] * apart))
        add = layer["mixer"]["left_scale"] * o @ t[m + "o"].t()
        m = p + "mix.right."
        lower = t[m + "lower"]
        q = torch.nn.functional.silu(h @ t[m + "q"].t()).view(n, b["heads"], -1)
        f = (lower + (1.0 - lower) * torch.sigmoid(h @ t[m + "f"].t() + t[m + "f.b"])).view(n, b["heads"], -1)
        v = (h @ t[m + "v"].t()).view(n, b["heads"], -1)
        state, o = torch.zeros(b["heads"], b["dim"], b["vdim"], dtype=F64, device=x.device), []
        for s in range(n):
            state = f[s][:, :, None] * state + (1.0 - f[s])[:, :, None] * v[s][:, None, :]
            o.append((q[s][:, None, :] @ state)[:, 0])
        o = _rms(torch.stack(o), t[m + "norm"], eps).reshape(n, -1)
        add = add + layer["mixer"]["right_scale"] * o @ t[m + "o"].t()
        h = _rms(x, 1.0 + t[p + "norm2"], eps)
        add = add + (torch.relu(h @ t[p + "mlp.gate"].t()) * (h @ t[p + "mlp.up"].t())) @ t[p + "mlp.down"].t()
        x = x + add
    return _rms(x, 1.0 + t["final.norm"], eps), t["head"]


def _rotate(x, rot):
    """x [..., T, d]: pairs (i, i + dims / 2) of the first dims entries turned by YaRN-scaled angles, taken in 32 bits."""
    dims, base, sc = rot["dims"], rot["base"], rot["scaling"]
    i = torch.arange(dims // 2, dtype=F64, device=x.device)
    f = base ** (-2.0 * i / dims)

    def edge(turns):
        return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))

    lo, hi = max(math.floor(edge(sc["fast"])), 0), min(math.ceil(edge(sc["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    f = f / sc["factor"] * ramp + f * (1.0 - ramp)
    angle = (torch.arange(x.shape[-2], device=x.device).float()[:, None] * f.float()[None]).to(F64)
    cos, sin = ((0.1 * math.log(sc["factor"]) + 1.0) * g for g in (torch.cos(angle), torch.sin(angle)))
    u, v = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([u * cos - v * sin, v * cos + u * sin, x[..., dims:]], -1)


def _falisun_exact(t, cfg, ids):
    """Mamba-2 layers and attention over latents, each result normed and scaled before it is added; routed experts."""
    eps, n = cfg["norm"]["eps"], len(ids)
    silu = torch.nn.functional.silu

    def lin(x, name):
        return x @ t[name].t()

    def gated(h, p):
        return lin(silu(lin(h, p + "gate")) * lin(h, p + "up"), p + "down")

    x, kept = t["embed"][ids], {}
    for i, layer in enumerate(cfg["layers"]):
        p, m, f = f"l{i}.", layer["mixer"], layer["mlp"]
        c = p + "mix."
        h = _rms(x, t[p + "norm1"], eps)
        if layer["type"] == "mamba2":
            inner, S, H = m["heads"] * m["vdim"], m["state"], m["heads"]
            z, u, dt = lin(h, c + "in").split([inner, inner + 2 * S, H], -1)
            u = torch.cat([u.new_zeros(m["conv"] - 1, u.shape[1]), u])
            u = silu(sum(u[j:j + n] * t[c + "conv"][:, j] for j in range(m["conv"])) + t[c + "conv.b"])
            v, B, C = u[:, :inner].view(n, H, -1), u[:, inner:inner + S], u[:, inner + S:]
            dt = torch.log1p(torch.exp(-(dt + t[c + "dt_bias"]).abs())) + (dt + t[c + "dt_bias"]).clamp(min=0.0)
            decay = torch.exp(-torch.exp(t[c + "A_log"]) * dt)
            state, y = torch.zeros(H, S, m["vdim"], dtype=F64, device=x.device), []
            for s in range(n):
                state = decay[s][:, None, None] * state + B[s][None, :, None] * (dt[s][:, None] * v[s])[:, None, :]
                y.append(C[s] @ state + t[c + "D"][:, None] * v[s])
            y = lin(_rms(torch.stack(y).reshape(n, inner) * silu(z), t[c + "norm"], eps), c + "o")
        else:
            H, R, d = m["heads"], m["kv_rank"], m["dim"]
            if "kv_from" not in m:
                row = lin(h, c + "dkv")
                kept[i] = (_rms(row[:, :R], t[c + "dkv.norm"], eps), _rotate(row[:, R:], m["rot"]))
            latent, turned = kept[m.get("kv_from", i)]
            q = _heads(lin(h, c + "q"), H)
            q = torch.cat([q[..., :d], _rotate(q[..., d:], m["rot"])], -1)
            k = torch.cat([_heads(lin(latent, c + "uk"), H), turned[None].expand(H, -1, -1)], -1)
            o = _softmax_attention(q, k, _heads(lin(latent, c + "uv"), H), m["scale"])
            y = lin(o * torch.sigmoid(lin(h, c + "g")), c + "o")
        x = x + _rms(y, t[p + "norm1b"], eps) * t[p + "ls1"]
        h = _rms(x, t[p + "norm2"], eps)
        e, r = p + "mlp.", f["router"]
        s = torch.softmax(lin(h, e + "router"), -1)
        best = s.view(n, r["groups"]["count"], -1).max(-1).values
        ok = torch.zeros_like(best).scatter_(1, best.topk(r["groups"]["keep"], -1).indices, 1.0)
        w, chosen = (s * ok.repeat_interleave(r["experts"] // r["groups"]["count"], 1)).topk(r["top"], -1)
        w = w / w.sum(-1, keepdim=True)
        y = gated(h, e + "shared.")
        for j in range(r["experts"]):
            y = y + (w * (chosen == j)).sum(-1, keepdim=True) * gated(h, f"{e}e{j}.")
        x = x + _rms(y, t[p + "norm2b"], eps) * t[p + "ls2"]
    return _rms(x, t["final.norm"], eps), t["embed"]


def exact(case, seed):
    t = _tensors(case["model"], case["dtype"])
    model = {"finuvik": _finuvik_exact, "falisun": _falisun_exact}.get(case["model"], _gpt2_exact)
    rows = []
    with torch.no_grad():
        for ids, (a, b) in zip(_sequences(case, seed), _lengths(case)):
            x, head = model(t, MODELS[case["model"]], torch.from_numpy(ids).long().cuda())
            rows.append(x[a + b - 1:a + b + case["steps"]] @ head.t())
    return torch.stack(rows, 1) if case["kind"] == "turn" else torch.cat(rows)
