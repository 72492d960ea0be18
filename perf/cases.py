"""Timed cases of the engine: one step of ``ModelRunner``, the function that generation, the trace replay and the
benchmark all go through, over the sizes, types and kinds of step that it serves.

A case names a model (layer sizes of this repository's presets, random weights), a compute type and a kind of step:

* ``decode``: ``batch`` requests, each behind up to ``context`` stored tokens, take one token more (the step that a
  serving loop repeats; replayed from a captured graph). Every pass is the next step of the same requests.
* ``prompt``: ``batch`` new requests whose prompts of up to ``tokens`` tokens run whole, logits of the last token; the
  requests end after the step.
* ``mixed``: one portion of ``tokens`` tokens of a longer prompt beside ``batch`` decoded tokens, which is what
  continuous batching runs while anything waits. Every pass is the next portion; a prompt that is through is followed
  by a new one.

``ragged`` spreads the lengths between half and all of ``context`` (or ``tokens``).

The Qwen3 models' stored keys and values are drawn (unit variance, as normed keys have); the models with per-request
states, Sinulix (retention, the gated delta rule, softmax attention, experts) and Gulisun (latent attention, gated
recurrences, experts), get theirs by running prompts.
"""
from __future__ import annotations

import math
import zlib

import torch

from tinyinfer_b200 import models  # noqa: F401  (registers the architectures)
from tinyinfer_b200.config import lookup_architecture
from tinyinfer_b200.engine.batch import StepEntry
from tinyinfer_b200.engine.runner import ModelRunner

DEVICE = "cuda:0"
PAGE = 64                 # tokens a page of the cache, the engine's default
HEADROOM = 256            # decode passes before the requests start over
PORTIONS = 4              # portions of a mixed case's prompt
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


# ------------------------------------------------------------------------------------------------ models
def _qwen3(hidden, layers, heads, ff, tied):
    return dict(architectures=["Qwen3ForCausalLM"], vocab_size=151936, hidden_size=hidden, num_hidden_layers=layers,
                num_attention_heads=heads, num_key_value_heads=8, head_dim=128, intermediate_size=ff, rms_norm_eps=1e-6,
                rope_theta=1000000.0, tie_word_embeddings=tied, max_position_embeddings=40960)


def _sinulix():
    """Layers r D a K r D a K: retention; the delta rule with experts; attention; attention on the keys and values of
    the attention layer before, with experts."""
    attention = dict(heads=16, kv_heads=8, dim=128, vdim=128, scale=128 ** -0.5, rot=dict(base=1000000.0, dims=128))
    retention = dict(heads=16, dim=128, vdim=128, decay=[1.0 - 2.0 ** -(5.0 + 3.0 * h / 16) for h in range(16)],
                     rot=dict(base=10000.0, dims=128))
    delta = dict(heads=16, kv_heads=16, dim=128, vdim=128, conv=4, gate_rank=64)
    dense = dict(kind="dense", ff=6144)
    moe = dict(kind="moe", expert=dict(ff=1408, limit=7.0), router=dict(experts=64, top=6, identity=2))
    layers = []
    for i in (0, 4):
        layers += [dict(type="retention", mixer=retention, mlp=dense), dict(type="channel_delta", mixer=delta, mlp=moe),
                   dict(type="attention", mixer=attention, mlp=dense),
                   dict(type="attention", mixer=dict(attention, kv_from=i + 2), mlp=moe)]
    return dict(architecture="Sinulix", vocab=102400, width=2048, norm=dict(eps=1e-6), embedding=dict(scale=45.0),
                logit_softcap=30.0, layers=layers)


def _gulisun():
    """Layers s r k p s r k p: latent attention with a sink; a gated recurrence; latent attention on the cache of the
    layer with a sink before; latent attention with the plain softmax. Experts everywhere."""
    latent = dict(heads=16, dim=128, rot_dim=64, vdim=128, q_rank=1536, kv_rank=512, scale=192 ** -0.5,
                  rot=dict(base=10000.0, dims=64))
    moe = dict(kind="moe", router=dict(experts=64, top=6), expert=dict(ff=1408), shared=dict(ff=2816))
    layers = []
    for i in (0, 4):
        layers += [dict(type="latent_attention", mixer=latent, mlp=moe),
                   dict(type="rglru", mixer=dict(width=2560, blocks=10, conv=4), mlp=moe),
                   dict(type="latent_attention", mixer=dict(latent, kv_from=i), mlp=moe),
                   dict(type="latent_attention_2", mixer=latent, mlp=moe)]
    return dict(architecture="Gulisun", vocab=102400, width=2048, embedding=dict(scale=1.0), norm=dict(eps=1e-6),
                layers=layers)


MODELS = {
    "qwen3-0.6b": _qwen3(1024, 28, 16, 3072, True),
    "qwen3-1.7b": _qwen3(2048, 28, 16, 6144, True),
    "qwen3-8b": _qwen3(4096, 36, 32, 12288, False),
    "sinulix-2b": _sinulix(),
    "gulisun-2b": _gulisun(),
}


def _is_qwen3(case):
    return case["model"].startswith("qwen3")


def _vocab(case):
    m = MODELS[case["model"]]
    return m["vocab_size"] if _is_qwen3(case) else m["vocab"]


def _named(case, seed, name, shape):
    """The checkpoint tensor ``name``. Matrices N(0, 0.02) in the compute type, in the Qwen3 models with the embedding
    N(0, 1) and the projections back into the residual divided by the root of their number, so that the residual is larger
    than what a layer adds to it, as in a trained model; norm weights 1 + N(0, 0.1); routers that prefer some experts
    clearly, as trained ones do; decays that remember some tens to hundreds of tokens."""
    gen = torch.Generator(device=DEVICE).manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) % (1 << 62))

    def noise(kind):
        return torch.empty(tuple(shape), dtype=kind, device=DEVICE).normal_(0.0, 1.0, generator=gen)

    last = name.rsplit(".", 1)[-1]
    if "norm" in name:
        added_to_one = case["model"].startswith("sinulix") and (last in ("norm1", "norm2") or name == "final.norm")
        return (0.0 if added_to_one else 1.0) + 0.1 * noise(torch.float32)
    for ending, centre, spread in (("conv", 0.0, 0.5), ("lam", -5.0, 0.5), ("dt_bias", -4.0, 0.5), ("A_log", 0.0, 0.5),
                                   ("sink", 0.0, 0.5), ("correction", 0.0, 0.02)):
        if last == ending:
            return centre + spread * noise(torch.float32)
    if last == "b" and not name.endswith("mix.b"):       # a bias; mix.b is a projection
        return 0.02 * noise(torch.float32)
    std = 0.06 if last == "router" else 0.02
    if name == "model.embed_tokens.weight":
        std = 1.0
    elif name.endswith(("o_proj.weight", "down_proj.weight")):
        std /= math.sqrt(2 * MODELS[case["model"]]["num_hidden_layers"])
    return noise(DTYPES[case["dtype"]]) * std


class _Weights:
    """What ``DecoderModel.load_tensors`` asks: every tensor drawn when it is wanted."""

    def __init__(self, case, seed, shapes):
        self.case, self.seed, self.shapes = case, seed, shapes

    def __getitem__(self, name):
        return _named(self.case, self.seed, name, self.shapes[name])


# ------------------------------------------------------------------------------------------------ the steps of a case
def _lengths(case, top):
    n = case["batch"]
    return [top - (i * top) // (2 * n) if case["ragged"] else top for i in range(n)]


def _tokens(case, seed, stream, count):
    gen = torch.Generator().manual_seed((int(seed) * 7919 + 13 * stream + 5) % (1 << 62))
    return torch.randint(0, _vocab(case), (count,), generator=gen).tolist()


def _stored(case, seed, layer, blocks):
    """The keys and values that a layer's cache holds before the first pass: [2, pages, kv heads, page, head size]."""
    gen = torch.Generator(device=DEVICE).manual_seed((int(seed) * 31337 + 17 * layer + 3) % (1 << 62))
    m = MODELS[case["model"]]
    shape = (2, sum(blocks), m["num_key_value_heads"], PAGE, m["head_dim"])
    return torch.empty(shape, dtype=DTYPES[case["dtype"]], device=DEVICE).normal_(0.0, 1.0, generator=gen)


def _pages(tokens):
    return -(-tokens // PAGE)


class _State:
    def __init__(self, case, seed):
        self.case, self.seed = case, seed
        m = MODELS[case["model"]]
        arch = lookup_architecture(m["architectures"][0] if _is_qwen3(case) else m["architecture"])
        model = arch.model_factory(arch.config_class.from_dict(dict(m)), DTYPES[case["dtype"]], torch.device(DEVICE))
        model.load_tensors(_Weights(case, seed, {n: t.shape for n, t in model.expected_tensors().items()}))
        kind, batch = case["kind"], case["batch"]
        self.lengths = _lengths(case, case["context"]) if kind != "prompt" else []
        self.blocks = [_pages(n + HEADROOM) for n in self.lengths]
        pages = sum(self.blocks)
        longest = max(self.lengths, default=0) + HEADROOM
        step_tokens = batch
        if kind == "prompt":
            self.prompts = [_tokens(case, seed, i, n) for i, n in enumerate(_lengths(case, case["tokens"]))]
            pages, longest = sum(_pages(len(p)) for p in self.prompts), max(map(len, self.prompts))
            step_tokens = sum(map(len, self.prompts))
        elif kind == "mixed":
            self.prompts = [_tokens(case, seed, 1000, PORTIONS * case["tokens"])]
            pages += _pages(len(self.prompts[0]))
            longest, step_tokens = max(longest, len(self.prompts[0])), batch + case["tokens"]
        elif not _is_qwen3(case):
            step_tokens = max(batch, longest)
        self.feed = _tokens(case, seed, 2000, max(1, batch) * HEADROOM)
        self.runner = ModelRunner(model, page_size=PAGE, num_pages=pages, max_requests=batch + 1,
                                  max_tokens_per_step=max(4096, step_tokens), max_model_len=longest, cuda_graphs=True)
        self.taken = self.portion = 0
        if self.lengths:
            self.begin()

    def begin(self):
        """The decoding requests, each behind its context."""
        runner, case = self.runner, self.case
        for i, n in enumerate(self.lengths):
            if _is_qwen3(case):
                runner.admit(i)
                runner.manager.extend(i, n + HEADROOM)
                runner.manager.commit(i, n)
            else:
                runner.step([StepEntry(i, _tokens(case, self.seed, i, n), [])])
        if _is_qwen3(case):
            table = [p for i in range(len(self.lengths)) for p in runner.manager.get(i).tables[0]]
            at = torch.tensor(table, device=DEVICE)
            for layer, kv in enumerate(runner.storage.kv):
                kv[:, at] = _stored(case, self.seed, layer, self.blocks)
        self.taken = 0


def prepare(case, seed):
    return _State(case, seed)


def run(s):
    case, runner, batch = s.case, s.runner, s.case["batch"]
    if case["kind"] == "prompt":
        logits = runner.step([StepEntry(i, p, [len(p) - 1]) for i, p in enumerate(s.prompts)])
        for i in range(batch):
            runner.release(i)
    else:
        if s.taken == HEADROOM:                          # the requests are at their length limit: new ones
            for i in range(batch):
                runner.release(i)
            s.begin()
        entries = [StepEntry(i, [s.feed[s.taken * batch + i]], [0]) for i in range(batch)]
        if case["kind"] == "mixed":
            n = case["tokens"]
            last = s.portion == PORTIONS - 1
            entries.append(StepEntry("prompt", s.prompts[0][s.portion * n:(s.portion + 1) * n], [n - 1] if last else []))
        logits = runner.step(entries)
        s.taken += 1
        if case["kind"] == "mixed":
            s.portion = (s.portion + 1) % PORTIONS
            if s.portion == 0:
                runner.release("prompt")
    out = {"logits": logits}
    if _is_qwen3(case):
        if case["kind"] == "prompt":                     # what a prompt is run for: its keys and values
            out["cache"] = list(runner.storage.kv)
    else:
        out["states"] = [t[:-1] for t in runner.storage.state if t is not None]     # the last slot is no request's
    return out


# ------------------------------------------------------------------------------------------------ the cases
def _case(name, model, kind, batch, context=0, tokens=0, dtype="bfloat16", ragged=False):
    c = dict(model=model, kind=kind, dtype=dtype, batch=batch, context=context, tokens=tokens, ragged=ragged)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user of a small model: nothing but launches and latency
        _case("qwen3_0p6b_decode_1", "qwen3-0.6b", "decode", 1, context=300),
        # the headline of the benchmark: eight users of an 8B model at 4,096 tokens
        _case("qwen3_8b_decode_8", "qwen3-8b", "decode", 8, context=4096),
        # a full batch with contexts of every length
        _case("qwen3_8b_decode_64", "qwen3-8b", "decode", 64, context=2048, ragged=True),
        # a short question: the time to the first token is the launches
        _case("qwen3_0p6b_prompt_37", "qwen3-0.6b", "prompt", 1, tokens=37),
        # the headline's prompt
        _case("qwen3_8b_prompt_2048", "qwen3-8b", "prompt", 1, tokens=2048),
        # continuous batching: a portion of a prompt beside the decoded tokens of 27 others
        _case("qwen3_1p7b_mixed_512_27", "qwen3-1.7b", "mixed", 27, context=901, tokens=512, ragged=True),
        # the true 32-bit path, which the equality runs and numerical checks of a checkpoint use
        _case("qwen3_1p7b_float32_prompt_333", "qwen3-1.7b", "prompt", 1, tokens=333, dtype="float32"),
        _case("qwen3_1p7b_float32_decode_4", "qwen3-1.7b", "decode", 4, context=1024, dtype="float32"),
        # a hybrid of matrix states, softmax attention and experts
        _case("sinulix_2b_prompt_2000", "sinulix-2b", "prompt", 1, tokens=2000),
        _case("sinulix_2b_decode_8", "sinulix-2b", "decode", 8, context=2048),
        # latent attention, gated recurrences and experts
        _case("gulisun_2b_prompt_2048", "gulisun-2b", "prompt", 1, tokens=2048),
        _case("gulisun_2b_decode_8", "gulisun-2b", "decode", 8, context=2048),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "prompt", "prompt", "mixed"))
    if kind == "mixed":
        return _case(None, rng.choice(("qwen3-0.6b", "qwen3-1.7b")), kind, _log(rng, 1, 48), context=_log(rng, 64, 2048),
                     tokens=_log(rng, 64, 512), ragged=True)
    model = rng.choice(("qwen3-0.6b", "qwen3-1.7b", "qwen3-8b", "sinulix-2b", "gulisun-2b"))
    wide = model in ("qwen3-0.6b", "qwen3-1.7b") and rng.random() < 0.4
    if kind == "decode":
        if not model.startswith("qwen3"):
            return _case(None, model, kind, _log(rng, 1, 16), context=_log(rng, 64, 2048))
        batch = _log(rng, 1, 8 if wide else 64)
        return _case(None, model, kind, batch, context=min(_log(rng, 64, 4096), 65536 // batch),
                     dtype="float32" if wide else "bfloat16", ragged=rng.random() < 0.5)
    if wide:
        return _case(None, model, kind, 1, tokens=_log(rng, 16, 333), dtype="float32")
    if not model.startswith("qwen3"):
        return _case(None, model, kind, 1, tokens=_log(rng, 16, 2048))
    batch = rng.choice((1, 1, 2, 3))
    return _case(None, model, kind, batch, tokens=_log(rng, 16, 2048) // batch + 1, ragged=batch > 1)


# ------------------------------------------------------------------------------------------------ what a pass must do
def _layer_costs(case):
    """Per layer (weight elements that every step reads, multiply-adds a token, expert elements, experts, experts a token,
    elements read per stored token, multiply-adds per pair of a query and a key, state elements)."""
    m = MODELS[case["model"]]
    if _is_qwen3(case):
        h, d, q, kv = m["hidden_size"], m["head_dim"], m["num_attention_heads"], m["num_key_value_heads"]
        w = h * (q + 2 * kv) * d + q * d * h + 3 * h * m["intermediate_size"]
        return [(w, w, 0, 0, 0, 2 * kv * d, 2 * q * d, 0)] * m["num_hidden_layers"]
    out, width = [], m["width"]
    for layer in m["layers"]:
        x, f, kind = layer["mixer"], layer["mlp"], layer["type"]
        stored = pair = state = extra = 0
        if kind == "attention":
            kv = 0 if "kv_from" in x else 2 * x["kv_heads"] * x["dim"]
            w = width * (2 * x["heads"] * x["dim"] + kv + x["heads"])
            stored, pair = 2 * x["kv_heads"] * x["dim"], 2 * x["heads"] * x["dim"]
        elif kind in ("retention", "channel_delta"):
            inner = x["heads"] * x["dim"]
            w = width * inner * (5 if kind == "retention" else 4)
            if kind == "channel_delta":
                w += 2 * x["gate_rank"] * (width + inner) + width * x["heads"]
            state = inner * x["vdim"]
            extra = (2 if kind == "retention" else 3) * state
        elif kind == "rglru":
            w = 3 * width * x["width"] + 2 * x["width"] ** 2 // x["blocks"]
            state = 4 * x["width"]
        else:
            H, d, r, dv, qr, kr = (x[n] for n in ("heads", "dim", "rot_dim", "vdim", "q_rank", "kv_rank"))
            w = width * qr + qr * H * (d + r) + H * kr * (d + dv) + H * dv * width + (0 if "kv_from" in x else width * (kr + r))
            stored, pair = kr + r, H * (d + r + dv)
        flops, each, experts, top = w + extra, 0, 0, 0
        if f["kind"] == "dense":
            w, flops = w + 3 * width * f["ff"], flops + 3 * width * f["ff"]
        else:
            experts, top = f["router"]["experts"], f["router"]["top"]
            each = (3 if "limit" in f["expert"] else 2) * width * f["expert"]["ff"]
            shared = 2 * width * f["shared"]["ff"] if "shared" in f else 0
            w, flops = w + width * experts + shared, flops + width * experts + shared + top * each
        out.append((w, flops, each, experts, top, stored, pair, state))
    return out


def work(case):
    size = 4 if case["dtype"] == "float32" else 2
    if case["kind"] == "prompt":
        entries = [(0, n) for n in _lengths(case, case["tokens"])]
    else:
        entries = [(n, 1) for n in _lengths(case, case["context"])]
    wanted = len(entries)
    if case["kind"] == "mixed":
        entries.append(((PORTIONS - 1) * case["tokens"] // 2, case["tokens"]))      # a portion in the middle of the prompt
    tokens = sum(n for _s, n in entries)
    keys = sum(s + n for s, n in entries)
    pairs = sum(n * s + n * (n + 1) / 2 for s, n in entries)
    m = MODELS[case["model"]]
    width = m["hidden_size"] if _is_qwen3(case) else m["width"]
    head = width * _vocab(case)
    byts, flops = size * (head + tokens * width) + 4 * wanted * _vocab(case), 2.0 * head * wanted
    for w, per_token, each, experts, top, stored, pair, state in _layer_costs(case):
        met = experts * (1.0 - (1.0 - top / experts) ** tokens) if experts else 0.0
        byts += size * (w + met * each + stored * keys) + 8 * state * len(entries)
        flops += 2.0 * (per_token * tokens + pair * pairs)
    return {"bytes": byts, "flops": flops}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 8e-6}          # measured 1.3e-6 to 2e-6 against 64 bits
    return {"rel": 0.03}              # measured 0.009 to 0.02 against 64 bits


# ------------------------------------------------------------------------------------------------ in 64 bits
def _rms(x, eps, weight=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _rotate(x, positions, dims, base):
    """x [..., tokens, heads, size]: the first ``dims`` features turn in pairs (i, i + dims / 2)."""
    half = dims // 2
    i = torch.arange(half, dtype=torch.float64, device=x.device)
    angle = positions.double()[:, None, None] * base ** (-2.0 * i / dims)
    c, s = torch.cos(angle), torch.sin(angle)
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], dim=-1)


def _attend(q, k, v, scale, start, sink=None):
    """q [n, heads, size] at positions start .., k and v [keys, kv heads, size]; a sink is one more term per head in the
    softmax's denominator."""
    n, H, _d = q.shape
    L, G, dv = v.shape
    out = torch.empty(n, H, dv, dtype=q.dtype, device=q.device)
    seen = torch.arange(L, device=q.device)[None] <= torch.arange(start, start + n, device=q.device)[:, None]
    for g in range(G):
        heads = slice(g * (H // G), (g + 1) * (H // G))
        z = torch.einsum("nhd,ld->hnl", q[:, heads], k[:, g]) * scale
        z = z.masked_fill(~seen, -math.inf)
        if sink is not None:
            z = torch.cat([z, sink[heads, None, None].expand(-1, n, 1)], dim=-1)
        p = torch.softmax(z, dim=-1)[..., :L]
        out[:, heads] = torch.einsum("hnl,ld->nhd", p, v[:, g])
    return out


def _exact_qwen3(case, seed):
    m = MODELS[case["model"]]
    h, d, H, G = m["hidden_size"], m["head_dim"], m["num_attention_heads"], m["num_key_value_heads"]
    ff, eps, base = m["intermediate_size"], m["rms_norm_eps"], m["rope_theta"]

    def w(name, *shape):
        return _named(case, seed, name, shape).double()

    if case["kind"] == "prompt":
        entries = [(0, _tokens(case, seed, i, n)) for i, n in enumerate(_lengths(case, case["tokens"]))]
        blocks, past = [_pages(len(t)) for _s, t in entries], None
    else:
        lengths = _lengths(case, case["context"])
        feed = _tokens(case, seed, 2000, max(1, case["batch"]) * HEADROOM)
        entries = [(n, [feed[i]]) for i, n in enumerate(lengths)]
        blocks = [_pages(n + HEADROOM) for n in lengths]
        if case["kind"] == "mixed":
            entries.append((0, _tokens(case, seed, 1000, PORTIONS * case["tokens"])[:case["tokens"]]))
    ids = torch.tensor([t for _s, ts in entries for t in ts], device=DEVICE)
    pos = torch.tensor([s + j for s, ts in entries for j in range(len(ts))], device=DEVICE)
    embed = _named(case, seed, "model.embed_tokens.weight", (m["vocab_size"], h))
    x = embed[ids].double()
    T, cache = x.shape[0], []
    for layer in range(m["num_hidden_layers"]):
        p = f"model.layers.{layer}."
        y = _rms(x, eps, w(p + "input_layernorm.weight", h))
        q = (y @ w(p + "self_attn.q_proj.weight", H * d, h).T).view(T, H, d)
        k = (y @ w(p + "self_attn.k_proj.weight", G * d, h).T).view(T, G, d)
        v = (y @ w(p + "self_attn.v_proj.weight", G * d, h).T).view(T, G, d)
        q = _rotate(_rms(q, eps, w(p + "self_attn.q_norm.weight", d)), pos, d, base)
        k = _rotate(_rms(k, eps, w(p + "self_attn.k_norm.weight", d)), pos, d, base)
        past = _stored(case, seed, layer, blocks) if case["kind"] != "prompt" else None
        outs, row, page = [], 0, 0
        for i, (start, ts) in enumerate(entries):
            n = len(ts)
            kn, vn = k[row:row + n], v[row:row + n]
            if start:
                old = past[:, page:page + blocks[i]].permute(0, 1, 3, 2, 4).reshape(2, -1, G, d)[:, :start].double()
                page += blocks[i]
                kn, vn = torch.cat([old[0], kn]), torch.cat([old[1], vn])
            outs.append(_attend(q[row:row + n], kn, vn, d ** -0.5, start).reshape(n, H * d))
            row += n
        if case["kind"] == "prompt":
            kept, row, page = torch.zeros(2, sum(blocks) + 1, G, PAGE, d, dtype=torch.float64, device=DEVICE), 0, 0
            for (_s, ts), b in zip(entries, blocks):
                room = torch.zeros(2, b * PAGE, G, d, dtype=torch.float64, device=DEVICE)
                room[0, :len(ts)], room[1, :len(ts)] = k[row:row + len(ts)], v[row:row + len(ts)]
                kept[:, page:page + b] = room.view(2, b, PAGE, G, d).permute(0, 1, 3, 2, 4)
                row, page = row + len(ts), page + b
            cache.append(kept)
        x = x + torch.cat(outs) @ w(p + "self_attn.o_proj.weight", h, H * d).T
        y = _rms(x, eps, w(p + "post_attention_layernorm.weight", h))
        gate = y @ w(p + "mlp.gate_proj.weight", ff, h).T
        up = y @ w(p + "mlp.up_proj.weight", ff, h).T
        x = x + (torch.nn.functional.silu(gate) * up) @ w(p + "mlp.down_proj.weight", h, ff).T
    counts = [len(ts) for _s, ts in entries]
    rows = [sum(counts[:i + 1]) - 1 for i in range(case["batch"])]
    y = _rms(x[rows], eps, w("model.norm.weight", h))
    head = embed if m["tie_word_embeddings"] else _named(case, seed, "lm_head.weight", (m["vocab_size"], h))
    out = {"logits": y @ head.double().T}
    return dict(out, cache=cache) if cache else out


def _convolve(x, taps):
    """Causal per-channel convolution of x [batch, tokens, channels]; the last column of ``taps`` meets the current token."""
    n = taps.shape[1]
    padded = torch.nn.functional.pad(x, (0, 0, n - 1, 0))
    return sum(padded[:, j:j + x.shape[1]] * taps[:, j] for j in range(n))


def _experts(h, weight, chosen, run):
    """sum over a token's choices of weight x expert(h); ``run(e, rows)`` is expert e's output."""
    flat, out = h.reshape(-1, h.shape[-1]), torch.zeros(h.numel() // h.shape[-1], h.shape[-1], dtype=h.dtype, device=h.device)
    weight, chosen = weight.reshape(flat.shape[0], -1), chosen.reshape(flat.shape[0], -1)
    for e in chosen.unique().tolist():
        rows, slot = (chosen == e).nonzero(as_tuple=True)
        out[rows] += weight[rows, slot, None] * run(e, flat[rows])
    return out.view(h.shape)


def _exact_sinulix(case, w, tokens):
    m, silu = MODELS[case["model"]], torch.nn.functional.silu
    width, eps = m["width"], m["norm"]["eps"]
    B, T = tokens.shape
    pos = torch.arange(T, device=DEVICE)
    x = w("embed", m["vocab"], width)[tokens] * m["embedding"]["scale"]
    kept = {}
    for i, layer in enumerate(m["layers"]):
        a, f, p = layer["mixer"], layer["mlp"], f"l{i}."
        h = _rms(x, eps, 1.0 + w(p + "norm1", width))
        H, d, dv = a["heads"], a["dim"], a["vdim"]
        mat = lambda name, rows, cols=width: w(p + "mix." + name, rows, cols).T  # noqa: E731
        if layer["type"] == "attention":
            G, rot = a["kv_heads"], a["rot"]
            q = _rotate(_rms((h @ mat("q", H * d)).view(B, T, H, d), eps, w(p + "mix.q.norm", d)), pos, rot["dims"], rot["base"])
            if "kv_from" not in a:
                k = _rms((h @ mat("k", G * d)).view(B, T, G, d), eps, w(p + "mix.k.norm", d))
                kept[i] = _rotate(k, pos, rot["dims"], rot["base"]), (h @ mat("v", G * dv)).view(B, T, G, dv)
            k, v = kept[a.get("kv_from", i)]
            sink = w(p + "mix.sink", H)
            o = torch.stack([_attend(q[b], k[b], v[b], a["scale"], 0, sink) for b in range(B)])
            y = (o * torch.sigmoid(h @ mat("g", H))[..., None]).reshape(B, T, H * dv)
        elif layer["type"] == "retention":
            rot = a["rot"]
            q = _rotate((h @ mat("q", H * d)).view(B, T, H, d), pos, rot["dims"], rot["base"])
            k = _rotate((h @ mat("k", H * d)).view(B, T, H, d), pos, rot["dims"], rot["base"]) * d ** -0.5
            v = (h @ mat("v", H * dv)).view(B, T, H, dv)
            age = (pos[:, None] - pos[None]).double()
            o = torch.empty_like(v)
            for n, decay in enumerate(a["decay"]):
                fade = torch.where(age >= 0, decay ** age.clamp(min=0), 0.0)
                o[:, :, n] = (torch.einsum("btd,bsd->bts", q[:, :, n], k[:, :, n]) * fade) @ v[:, :, n]
            y = _rms(o, eps).reshape(B, T, H * dv) * silu(h @ mat("g", H * dv))
        else:
            G, r = a["kv_heads"], a["gate_rank"]
            q, k, v = (silu(_convolve(h @ mat(n, heads * size), w(p + f"mix.{n}.conv", heads * size, a["conv"])))
                       .view(B, T, heads, size) for n, heads, size in (("q", G, d), ("k", G, d), ("v", H, dv)))
            q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
            k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            beta = torch.sigmoid(h @ mat("b", H))
            dt = torch.nn.functional.softplus(h @ mat("a1", r) @ mat("a2", H * d, r) + w(p + "mix.dt_bias", H * d)).view(B, T, H, d)
            g = torch.exp(-torch.exp(w(p + "mix.A_log", H))[:, None] * dt)
            S, o = torch.zeros(B, H, d, dv, dtype=torch.float64, device=DEVICE), torch.empty_like(v)
            for t in range(T):
                S = S * g[:, t, :, :, None]
                u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhkv,bhk->bhv", S, k[:, t]))
                S = S + k[:, t, :, :, None] * u[:, :, None, :]
                o[:, t] = torch.einsum("bhkv,bhk->bhv", S, q[:, t])
            y = _rms(o, eps, w(p + "mix.norm", dv)).reshape(B, T, H * dv) * torch.sigmoid(h @ mat("g1", r) @ mat("g2", H * dv, r))
        x = x + y @ w(p + "mix.o", width, H * dv).T
        h = _rms(x, eps, 1.0 + w(p + "norm2", width))
        if f["kind"] == "dense":
            gate, up = h @ w(p + "mlp.gate", f["ff"], width).T, h @ w(p + "mlp.up", f["ff"], width).T
            x = x + (silu(gate) * up) @ w(p + "mlp.down", width, f["ff"]).T
            continue
        r, e = f["router"], f["expert"]
        every = r["experts"] + r["identity"]
        scores = torch.softmax(h @ w(p + "mlp.router", every, width).T, dim=-1)
        chosen = torch.topk(scores + w(p + "mlp.correction", every), r["top"]).indices

        def run_expert(n, rows):
            if n >= r["experts"]:
                return rows
            g = (rows @ w(p + f"mlp.e{n}.gate", e["ff"], width).T).clamp(max=e["limit"])
            u = (rows @ w(p + f"mlp.e{n}.up", e["ff"], width).T).clamp(-e["limit"], e["limit"])
            return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(p + f"mlp.e{n}.down", width, e["ff"]).T

        x = x + _experts(h, scores.gather(-1, chosen), chosen, run_expert)
    z = _rms(x[:, -1], eps, 1.0 + w("final.norm", width)) @ w("head", m["vocab"], width).T
    return m["logit_softcap"] * torch.tanh(z / m["logit_softcap"])


def _exact_gulisun(case, w, tokens):
    m = MODELS[case["model"]]
    width, eps = m["width"], m["norm"]["eps"]
    B, T = tokens.shape
    pos = torch.arange(T, device=DEVICE)
    embed = w("embed", m["vocab"], width)
    x = embed[tokens] * m["embedding"]["scale"]
    kept = {}
    for i, layer in enumerate(m["layers"]):
        a, f, p = layer["mixer"], layer["mlp"], f"l{i}."
        if layer["type"] == "rglru":
            n, blocks = a["width"], a["blocks"]
            part = n // blocks
            y = torch.nn.functional.gelu(x @ w(p + "mix.y", n, width).T + w(p + "mix.y.b", n), approximate="tanh")
            u = _convolve(x @ w(p + "mix.x", n, width).T + w(p + "mix.x.b", n), w(p + "mix.conv", n, a["conv"])) + w(p + "mix.conv.b", n)
            gates = [torch.sigmoid(torch.einsum("btki,koi->btko", u.view(B, T, blocks, part), w(p + "mix." + g, blocks, part, part))
                                   + w(p + f"mix.{g}.b", blocks, part)).reshape(B, T, n) for g in ("ra", "ri")]
            decay = torch.exp(-8.0 * gates[0] * torch.nn.functional.softplus(w(p + "mix.lam", n)))
            drive = torch.sqrt(1.0 - decay * decay) * gates[1] * u
            S, o = torch.zeros(B, n, dtype=torch.float64, device=DEVICE), torch.empty_like(u)
            for t in range(T):
                S = decay[:, t] * S + drive[:, t]
                o[:, t] = S
            mixed = (o * y) @ w(p + "mix.o", width, n).T
        else:
            H, d, r, dv, rank, rot = a["heads"], a["dim"], a["rot_dim"], a["vdim"], a["kv_rank"], a["rot"]
            if "kv_from" not in a:
                down = x @ w(p + "mix.dkv", rank + r, width).T
                kept[i] = (_rms(down[..., :rank], eps, w(p + "mix.dkv.norm", rank)),
                           _rotate(down[..., None, rank:], pos, rot["dims"], rot["base"]))
            c, turned = kept[a.get("kv_from", i)]
            q = _rms(x @ w(p + "mix.dq", a["q_rank"], width).T, eps, w(p + "mix.dq.norm", a["q_rank"]))
            q = (q @ w(p + "mix.uq", H * (d + r), a["q_rank"]).T).view(B, T, H, d + r)
            q = torch.cat([q[..., :d], _rotate(q[..., d:], pos, rot["dims"], rot["base"])], dim=-1)
            k = torch.cat([(c @ w(p + "mix.uk", H * d, rank).T).view(B, T, H, d), turned.expand(B, T, H, r)], dim=-1)
            v = (c @ w(p + "mix.uv", H * dv, rank).T).view(B, T, H, dv)
            sink = w(p + "mix.sink", H) if layer["type"] == "latent_attention" else None
            o = torch.stack([_attend(q[b], k[b], v[b], a["scale"], 0, sink) for b in range(B)])
            mixed = o.reshape(B, T, H * dv) @ w(p + "mix.o", width, H * dv).T
        x = x + _rms(mixed, eps, w(p + "norm1", width))
        r, ff = f["router"], f["expert"]["ff"]
        scores = torch.softmax(x @ w(p + "mlp.router", r["experts"], width).T, dim=-1)
        best, chosen = torch.topk(scores, r["top"])

        def relu_squared(rows, up, down):
            return torch.relu(rows @ up.T) ** 2 @ down.T

        out = _experts(x, best / (best.sum(-1, keepdim=True) + 1e-20), chosen, lambda n, rows: relu_squared(
            rows, w(p + f"mlp.e{n}.up", ff, width), w(p + f"mlp.e{n}.down", width, ff)))
        sf = f["shared"]["ff"]
        out = out + relu_squared(x, w(p + "mlp.shared.up", sf, width), w(p + "mlp.shared.down", width, sf))
        x = x + _rms(out, eps, w(p + "norm2", width))
    return _rms(x[:, -1], eps, w("final.norm", width)) @ embed.T


def exact(case, seed):
    """What the first pass on a new state returns, in 64 bits."""
    if _is_qwen3(case):
        return _exact_qwen3(case, seed)

    def w(name, *shape):
        return _named(case, seed, name, shape).double()

    batch = case["batch"]
    if case["kind"] == "prompt":
        rows = [_tokens(case, seed, i, case["tokens"]) for i in range(batch)]
    else:
        feed = _tokens(case, seed, 2000, batch * HEADROOM)
        rows = [_tokens(case, seed, i, case["context"]) + [feed[i]] for i in range(batch)]
    forward = _exact_sinulix if case["model"].startswith("sinulix") else _exact_gulisun
    return {"logits": forward(case, w, torch.tensor(rows, device=DEVICE)), "states": None}
