"""What the engine's speed is measured on: whole decode steps of a Qwen3 model through the step function, and the layers of the seven
architectures one by one through the parts' ``forward``, over the sizes that `bench.py` and `cppvllm_b200/design_bench.py` use.

A case is a dict of plain values.  ``kind`` names the entry point, ``size`` the layer sizes, ``tokens`` and ``past`` hold one number per
request of the step (this step's tokens, and how many the cache already holds)."""
import json
import math
import os
import shutil
import tempfile

import torch

from cppvllm_b200 import models as _models, parts as _parts  # noqa: F401  (architectures and parts register themselves)
from cppvllm_b200.engine.runner import ModelRunner, StepEntry
from cppvllm_b200.parts.base import Runtime, Workspace, part_class
from cppvllm_b200.parts.context import CacheUnitView, GroupStepView, StepContext
from cppvllm_b200.weights.safetensors_io import save_safetensors

F64 = torch.float64
PAGE = 32                                   # the engine's page size
SIZES = {"small": dict(width=1024, heads=16, kv_heads=8, dim=128, ff=3072), "large": dict(width=4096, heads=32, kv_heads=8, dim=128, ff=12288)}
DECODE_LAYERS, DECODE_VOCAB, DECODE_RUN = 8, 32000, 32
WINDOW, KEEP, CHUNK, POOL, CAP = 1024, 4, 1024, 64, 30.0
BIAS_ROWS, BIAS_FAR, TEMP_COEF, TEMP_EVERY = 32, 1024, 0.25, 128
KV_RANK, ROT_DIM, EXPERTS, TOP, TAPS = 96, 32, 8, 2, 4
SSD_STATE, SSD_VDIM, SSD_GROUPS, SSD_PARTS = 128, 64, 8, 8


def listed():
    def case(name, kind, size, tokens, past="0", variant="", dtype="bfloat16"):
        return dict(name=name, kind=kind, size=size, tokens=tokens, past=past, variant=variant, dtype=dtype)
    return [
        # one user's chat: a single decoded token, as small as a step gets
        case("decode_one", "decode", "small", "1", "511"),
        # a busy server between admissions: eight requests with long contexts
        case("decode_batch", "decode", "small", ",".join(["1"] * 8), ",".join(["4095"] * 8)),
        # attention layer of a prompt that arrives whole (Qwen3-0.6B layer sizes)
        case("attention_prompt", "attention", "small", "2048"),
        # attention layer of a portion of a long prompt behind what is cached already (Qwen3-8B layer sizes)
        case("attention_portion", "attention", "large", "512", "7680"),
        # the 32-bit path: three short prompts in one step
        case("attention_float32", "attention", "small", "255,130,64", "0,33,0", dtype="float32"),
        # attention inside chunks with a gate per element, a whole prompt (Sumevik)
        case("chunked_attention", "masked", "small", "2048", variant="chunk"),
        # attention over a latent, a whole prompt (Dugulorn)
        case("latent_attention", "latent", "small", "2048", variant="head"),
        # attention over keys that are the values, behind a window with kept first tokens: prompts of several users (Givirax)
        case("window_attention", "keys", "large", "1100,517,300", "0,900,2000"),
        # attention with a bias per distance (Lorulix)
        case("biased_attention", "biased", "small", "1500,548", "0,700"),
        # delta rule with one decay per head, two prompts (Lorulix)
        case("delta_rule", "delta", "small", "1511,537"),
        # state-space recurrence over a prompt (Legalix)
        case("state_space", "ssd", "small", "2048"),
        # mixture of experts over a step's tokens (Givirax)
        case("experts", "experts", "large", "2048"),
    ]


VARIANTS = {"masked": ("chunk", "chunk_capped", "window_pooled", "window_kept"), "latent": ("head", "element", "sink")}


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(("decode", "decode", "attention", "attention", "masked", "masked", "latent", "keys", "biased", "delta", "ssd", "experts"))
    size, dtype = rng.choice(("small", "small", "large")), "bfloat16"
    if kind == "decode":
        n = log(1, 48)
        ctx = log(64, 4000 if n <= 16 else 1500)
        tokens, past, size = [1] * n, [max(1, ctx - rng.randrange(0, 33)) for _ in range(n)], "small"
    else:
        if kind == "attention" and rng.random() < 0.3:
            dtype, size = "float32", "small"
        total = log(64, 600 if dtype == "float32" else 2048)
        n = rng.choice((1, 1, 2, 3)) if total >= 96 else 1
        cuts = sorted(rng.randrange(1, total) for _ in range(n - 1))
        tokens = [b - a for a, b in zip([0] + cuts, cuts + [total]) if b > a]
        cached = kind in ("attention", "masked", "latent", "keys", "biased") and rng.random() < 0.5
        past = [log(1, 400 if dtype == "float32" else 4000) if cached else 0 for _ in tokens]
    return dict(kind=kind, size=size, tokens=",".join(map(str, tokens)), past=",".join(map(str, past)),
                variant=rng.choice(VARIANTS[kind]) if kind in VARIANTS else "", dtype=dtype)


# ---- what a case is made of --------------------------------------------------------------------------------------------------

def _shape(case):
    s = SIZES[case["size"]]
    tokens = [int(t) for t in case["tokens"].split(",")]
    past = [int(t) for t in case["past"].split(",")]
    if len(past) == 1:
        past = past * len(tokens)
    return s, tokens, past


def _params(case):
    """(part category, registered kind, parameters but for the position encoding, its parameters or None, cache entry shape, token axis)."""
    s, _, _ = _shape(case)
    D, H, G, d = s["width"], s["heads"], s["kv_heads"], s["dim"]
    rot = dict(rotary_dim=d, theta=1e6)
    heads = dict(hidden_size=D, num_heads=H, num_kv_heads=G)
    kind, v = case["kind"], case["variant"]
    if kind == "attention":
        return "mixer", "paged_attention", dict(heads, head_dim=d), dict(rot, pairing="half"), (2, G, d), 2
    if kind == "masked":
        p = dict(heads, dim=d, vdim=d, scale=1 / math.sqrt(d), eps=1e-5)
        if v == "chunk":
            p.update(chunk=CHUNK, qkv_bias=True, element_gate=True)
        elif v == "chunk_capped":
            return "mixer", "masked_attention", dict(p, chunk=CHUNK, softcap=CAP, distance_bias=True, sink=True, head_gate=True), None, (G, 2 * d), 1
        elif v == "window_pooled":
            return "mixer", "masked_attention", dict(p, window=WINDOW, pool=POOL), dict(rot, pairing="interleaved"), (2, G, 2 * d), 2
        else:
            p.update(window=WINDOW, keep_first=KEEP, softcap=CAP, qk_norm=False)
        return "mixer", "masked_attention", p, dict(rot, pairing="half" if v == "window_kept" else "interleaved"), (G, 2 * d), 1
    if kind == "latent":
        p = dict(hidden_size=D, num_heads=H, nope_dim=d, rot_dim=ROT_DIM, value_dim=d, q_rank=0 if v == "element" else 3 * D // 8, kv_rank=KV_RANK,
                 scale=1 / math.sqrt(d + ROT_DIM), eps=1e-5, gate={"head": "head", "element": "element", "sink": "none"}[v], sink=v == "sink")
        return "mixer", "latent_attention", p, dict(rotary_dim=ROT_DIM, theta=1e6, pairing="interleaved"), (KV_RANK + ROT_DIM,), 0
    if kind == "keys":
        return "mixer", "keys_attention", dict(heads, head_dim=d, window=WINDOW, keep_first=KEEP), None, (G, d), 1
    if kind == "biased":
        return "mixer", "biased_attention", dict(heads, dim=d, vdim=d, scale=1 / math.sqrt(d), eps=1e-5, bias_max=BIAS_FAR, bias_rows=BIAS_ROWS,
                                                 temp_coef=TEMP_COEF, temp_every=TEMP_EVERY), None, (G, 2 * d), 1
    if kind == "delta":
        return "mixer", "head_delta", dict(heads, dim=d, vdim=d, taps=TAPS, eps=1e-5), None, None, 0
    if kind == "ssd":
        return "mixer", "ssd", dict(hidden_size=D, num_heads=2 * D // SSD_VDIM, groups=SSD_GROUPS, state=SSD_STATE, vdim=SSD_VDIM, taps=TAPS,
                                    norm_parts=SSD_PARTS, eps=1e-5), None, None, 0
    return "ffn", "routed_glu", dict(hidden_size=D, intermediate_size=s["ff"] // 2, num_experts=EXPERTS, top=TOP), None, None, 0


def _weight_shapes(case):
    """name -> (shape, how its values are distributed); "m" matrices in the case's element type, the others are 32-bit vectors."""
    _, kind, p, _, _, _ = _params(case)
    D, H, G = p.get("hidden_size"), p.get("num_heads"), p.get("num_kv_heads")
    if kind == "paged_attention":
        d = p["head_dim"]
        return {"q_proj.weight": ((H * d, D), "m"), "k_proj.weight": ((G * d, D), "m"), "v_proj.weight": ((G * d, D), "m"), "o_proj.weight": ((D, H * d), "m"),
                "q_norm.weight": ((d,), "one"), "k_norm.weight": ((d,), "one")}
    if kind == "masked_attention":
        d = p["dim"]
        w = {"q": ((H * d, D), "m"), "k": ((G * d, D), "m"), "v": ((G * d, D), "m"), "o": ((D, H * d), "m")}
        if p.get("qk_norm", True):
            w.update({"q.norm": ((d,), "one"), "k.norm": ((d,), "one")})
        if p.get("distance_bias"):
            w.update({"r1": ((H,), "one"), "r2": ((H,), "one")})
        if p.get("sink"):
            w["sink"] = ((H,), "normal")
        if p.get("head_gate") or p.get("element_gate"):
            w["g"] = ((H if p.get("head_gate") else H * d, D), "m")
        if p.get("qkv_bias"):
            w.update({"q.b": ((H * d,), "small"), "k.b": ((G * d,), "small"), "v.b": ((G * d,), "small")})
        return w
    if kind == "latent_attention":
        dn, dr, dv, Q, R = p["nope_dim"], p["rot_dim"], p["value_dim"], p["q_rank"], p["kv_rank"]
        w = {"uk": ((H * dn, R), "m5"), "uv": ((H * dv, R), "m5"), "o": ((D, H * dv), "m"), "dkv": ((R + dr, D), "m"), "dkv.norm": ((R,), "one")}
        w.update({"dq": ((Q, D), "m"), "dq.norm": ((Q,), "one"), "uq": ((H * (dn + dr), Q), "m5")} if Q else {"q": ((H * (dn + dr), D), "m")})
        if p["gate"] != "none":
            w["g"] = ((H if p["gate"] == "head" else H * dv, D), "m")
        if p["sink"]:
            w["sink"] = ((H,), "normal")
        return w
    if kind == "keys_attention":
        d = p["head_dim"]
        return {"q": ((H * d, D), "m"), "k": ((G * d, D), "m"), "o": ((D, H * d), "m")}
    if kind == "biased_attention":
        d = p["dim"]
        return {"q": ((H * d, D), "m"), "k": ((G * d, D), "m"), "v": ((G * d, D), "m"), "o": ((D, H * d), "m"), "q.norm": ((H * d,), "one"),
                "k.norm": ((G * d,), "one"), "rel": ((BIAS_ROWS, H), "half")}
    if kind == "head_delta":
        d = p["dim"]
        return {"q": ((G * d, D), "m"), "q.conv": ((G * d, TAPS), "taps"), "k": ((G * d, D), "m"), "k.conv": ((G * d, TAPS), "taps"), "v": ((H * d, D), "m"),
                "v.conv": ((H * d, TAPS), "taps"), "b": ((H, D), "m"), "a": ((H, D), "m"), "A_log": ((H,), "rate"), "dt_bias": ((H,), "step"),
                "norm": ((d,), "one"), "g": ((H * d, D), "m"), "o": ((D, H * d), "m")}
    if kind == "ssd":
        inner, C = H * SSD_VDIM, H * SSD_VDIM + 2 * SSD_GROUPS * SSD_STATE
        return {"in": ((inner + C + H, D), "m"), "conv": ((C, TAPS), "taps"), "conv.b": ((C,), "small"), "dt_bias": ((H,), "step"), "A_log": ((H,), "rate"),
                "D": ((H,), "one"), "norm": ((inner,), "one"), "o": ((D, inner), "m")}
    I = p["intermediate_size"]
    w = {"router": ((EXPERTS, D), "router"), "router.b": ((EXPERTS,), "small")}
    for e in range(EXPERTS):
        w.update({f"e{e}.gate": ((I, D), "m"), f"e{e}.up": ((I, D), "m"), f"e{e}.down": ((D, I), "m")})
    return w


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, shape, std=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=g, device="cuda") * std).to(dtype)


def _value(g, shape, how, dtype):
    if how == "m":
        return _normal(g, shape, 0.02, dtype)
    if how == "m5":                         # low-rank factors: the inner size is small
        return _normal(g, shape, 0.05, dtype)
    u = torch.rand(shape, generator=g, device="cuda")
    n = torch.randn(shape, generator=g, device="cuda")
    return {"one": 0.9 + 0.2 * u, "normal": n, "half": 0.5 * n, "small": 0.02 * n, "router": 0.02 * n, "taps": u - 0.5, "rate": torch.log(1 + 7 * u),
            "step": torch.log(torch.expm1(torch.exp(math.log(1e-3) + math.log(100.0) * u)))}[how].contiguous()


def _layout(case, g):
    """Pages of the step's requests in a random order: (pages a request, block tables [S, W], entries [S][past, *entry])."""
    _, tokens, past = _shape(case)
    per = [-(-(a + n) // PAGE) for a, n in zip(past, tokens)]
    order = torch.randperm(sum(per), generator=g, device="cuda")
    tables = torch.full((len(per), max(per)), -1, dtype=torch.int32, device="cuda")
    at = 0
    for s, n in enumerate(per):
        tables[s, :n] = order[at:at + n].to(torch.int32)
        at += n
    return sum(per), tables


def _inputs(case, seed):
    """Everything that is drawn from the seed, in one order: weights, activations, pages with what earlier steps left in them."""
    s, tokens, past = _shape(case)
    dtype = getattr(torch, case["dtype"])
    g = _gen(seed)
    w = {n: _value(g, shape, how, dtype) for n, (shape, how) in _weight_shapes(case).items()}
    x = _normal(g, (sum(tokens), s["width"]), 1.0, dtype)
    _, _, _, _, entry, axis = _params(case)
    pages = tables = None
    if entry is not None:
        n, tables = _layout(case, g)
        pages = _normal(g, (n + 1,) + entry[:axis] + (PAGE,) + entry[axis:], 1.0, dtype)
    return w, x, pages, tables


def prepare(case, seed):
    if case["kind"] == "decode":
        return _prepare_decode(case, seed)
    s, tokens, past = _shape(case)
    w, x, pages, tables = _inputs(case, seed)
    dev, T, S = torch.device("cuda:0"), sum(tokens), len(tokens)
    category, kind, params, pos, entry, _ = _params(case)
    longest = max(a + n for a, n in zip(past, tokens))
    rt = Runtime(dev, x.dtype, Workspace(dev, max(T, 64), max(8, S)), max_positions=longest + 1)
    if pos is not None:
        params = dict(params, position=part_class("position", "rotary")(rt, max_positions=longest + 1, **pos))
    part = part_class(category, kind)(rt, **params)
    part.bind(w)

    def ints(v):
        return torch.tensor(v, dtype=torch.int32, device=dev)
    cu = [0]
    for n in tokens:
        cu.append(cu[-1] + n)
    positions = [p for a, n in zip(past, tokens) for p in range(a, a + n)]
    seq_of = [i for i, n in enumerate(tokens) for _ in range(n)]
    groups, view, state = [], None, None
    if entry is not None:
        pt, st = ints(positions).long(), ints(seq_of).long()
        slots = tables[st, pt // PAGE] * PAGE + (pt % PAGE).to(torch.int32)
        groups = [GroupStepView(tables, slots.to(torch.int32).contiguous(), PAGE, pages.shape[0])]
        view = CacheUnitView(pages, 0, part.cache_spec())
    elif category == "mixer":
        spec = part.state_spec()
        state = torch.zeros((S + 1,) + tuple(spec.shape), dtype=spec.dtype, device=dev)
    ctx = StepContext(num_tokens=T, num_seqs=S, tokens=ints([0] * T), positions=ints(positions), seq_of_token=ints(seq_of), cu_seqlens=ints(cu),
                      kv_lens=ints([a + n for a, n in zip(past, tokens)]), state_slots=ints(list(range(S))), groups=groups, logit_rows=ints([T - 1]),
                      num_logit_rows=1, q_lens=list(tokens), max_q_len=max(tokens), max_kv_len=longest, all_decode=all(n == 1 for n in tokens))
    return dict(part=part, x=x, ctx=ctx, view=view, pages=pages, state=state, category=category, fresh=torch.arange(S, device=dev),
                matrix=_matrix_floats(case), slots=S)


def _matrix_floats(case):
    """Floats of a request's state that hold the recurrence's matrices; the convolution's inputs lie behind them."""
    s, _, _ = _shape(case)
    if case["kind"] == "delta":
        return s["heads"] * s["dim"] * s["dim"]
    return 2 * s["width"] * SSD_STATE if case["kind"] == "ssd" else 0


def run(st):
    if "runner" in st:
        return _run_decode(st)
    if st["category"] == "ffn":
        return [st["part"].forward(st["x"], st["ctx"])]
    if st["state"] is not None:
        st["state"].index_fill_(0, st["fresh"], 0)                  # a prompt begins: the step function clears the slots of new requests
        y = st["part"].forward(st["x"], st["ctx"], None, st["state"])
        return [y, st["state"][:st["slots"], :st["matrix"]]]
    y = st["part"].forward(st["x"], st["ctx"], st["view"], None)
    return [y, st["pages"]]


# ---- decode steps of a whole model -------------------------------------------------------------------------------------------

def _decode_config(case):
    s, tokens, past = _shape(case)
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", hidden_size=s["width"], num_hidden_layers=DECODE_LAYERS,
                num_attention_heads=s["heads"], num_key_value_heads=s["kv_heads"], head_dim=s["dim"], intermediate_size=s["ff"],
                vocab_size=DECODE_VOCAB, rope_theta=1e6, rms_norm_eps=1e-6, tie_word_embeddings=True, max_position_embeddings=8192)


def _decode_inputs(case, seed):
    """Weights by name, the tokens of every step, and the cached keys and values by request: [past, layers, 2, kv heads, dim]."""
    s, tokens, past = _shape(case)
    D, H, G, d, I = s["width"], s["heads"], s["kv_heads"], s["dim"], s["ff"]
    g, bf = _gen(seed), torch.bfloat16
    w = {"model.embed_tokens.weight": _normal(g, (DECODE_VOCAB, D), 0.02, bf), "model.norm.weight": _value(g, (D,), "one", bf).to(bf)}
    for i in range(DECODE_LAYERS):
        p = f"model.layers.{i}."
        for n, rows, cols in (("self_attn.q_proj", H * d, D), ("self_attn.k_proj", G * d, D), ("self_attn.v_proj", G * d, D), ("self_attn.o_proj", D, H * d),
                              ("mlp.gate_proj", I, D), ("mlp.up_proj", I, D), ("mlp.down_proj", D, I)):
            w[p + n + ".weight"] = _normal(g, (rows, cols), 0.02, bf)
        for n, size in (("input_layernorm", D), ("post_attention_layernorm", D), ("self_attn.q_norm", d), ("self_attn.k_norm", d)):
            w[p + n + ".weight"] = _value(g, (size,), "one", bf).to(bf)
    ids = torch.randint(0, DECODE_VOCAB, (DECODE_RUN, len(tokens)), generator=g, device="cuda").tolist()
    cached = (_normal(g, (n, DECODE_LAYERS, 2, G, d), 1.0, bf) for n in past)      # one request at a time
    return w, ids, cached


def _prepare_decode(case, seed):
    s, tokens, past = _shape(case)
    w, ids, cached = _decode_inputs(case, seed)
    B, longest = len(tokens), max(past) + DECODE_RUN
    folder = tempfile.mkdtemp(prefix="perf_model_")
    try:
        with open(os.path.join(folder, "config.json"), "w") as f:
            json.dump(_decode_config(case), f)
        save_safetensors(os.path.join(folder, "model.safetensors"), {n: t.cpu() for n, t in w.items()})
        del w
        runner = ModelRunner(folder, dtype=torch.bfloat16, page_size=PAGE, num_pages=sum(-(-(n + DECODE_RUN) // PAGE) for n in past) + 1,
                             max_step_tokens=max(64, B), max_seqs=B, max_model_len=longest)
    finally:
        shutil.rmtree(folder, ignore_errors=True)
    st = dict(runner=runner, ids=ids, past=past, at=0, names=list(range(B)))
    for r, kv in zip(st["names"], cached):                # what earlier steps left in the cache
        _admit(st, r)
        table = torch.tensor(list(runner.cache.block_table(r, 0)), dtype=torch.long, device="cuda")
        pos = torch.arange(past[r], device="cuda")
        pool = runner.storage[0]                          # [layers, pages, 2, kv heads, slot, dim]
        pool[:, table[pos // PAGE], :, :, pos % PAGE] = kv
    return st


def _admit(st, r):
    cache, n = st["runner"].cache, st["past"][r]
    cache.admit(r)
    cache.reserve(r, n + DECODE_RUN)
    cache.advance(r, n)


def _run_decode(st):
    runner, at = st["runner"], st["at"]
    if at == DECODE_RUN:                                  # the requests end and others take their places
        for r in st["names"]:
            runner.cache.release(r)
        for r in st["names"]:
            _admit(st, r)
        at = 0
    st["at"] = at + 1
    logits = runner.step([StepEntry(r, [st["ids"][at][r]], st["past"][r] + at, [0]) for r in st["names"]])
    return [logits, runner.storage[0]]                    # the cache holds the step's keys and values now


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------------

def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _turn(x, positions, pos):
    """x [T, heads, d]; the first rotary_dim elements turned in pairs by the position."""
    r = pos["rotary_dim"]
    ang = positions.to(F64)[:, None] * torch.pow(torch.tensor(pos["theta"], dtype=F64), -torch.arange(0, r, 2, dtype=F64, device="cpu") / r).to(x.device)
    c, s = ang.cos()[:, None, :], ang.sin()[:, None, :]
    y = x.clone()
    a, b = (x[..., 0:r:2], x[..., 1:r:2]) if pos["pairing"] == "interleaved" else (x[..., :r // 2], x[..., r // 2:r])
    u, v = a * c - b * s, b * c + a * s
    if pos["pairing"] == "interleaved":
        y[..., 0:r:2], y[..., 1:r:2] = u, v
    else:
        y[..., :r // 2], y[..., r // 2:r] = u, v
    return y


def _softmax_sum(s, v, sink=None):
    m = s.amax(-1, keepdim=True)
    if sink is not None:
        m = torch.maximum(m, sink.expand_as(m))
    e = torch.exp(s - m)
    den = e.sum(-1, keepdim=True)
    if sink is not None:
        den = den + torch.exp(sink - m)
    return (e / den) @ v


def _entries(pages, tables, s, n, axis):
    """The first n entries of request s as its pages hold them: [n, *entry]."""
    p = pages.movedim(axis + 1, 1)                        # [page, slot, *entry]
    pos = torch.arange(n, device=pages.device)
    return p[tables[s].long()[pos // PAGE], pos % PAGE]


def _put(pages, tables, s, first, new, axis):
    p = pages.movedim(axis + 1, 1)
    pos = torch.arange(first, first + new.shape[0], device=pages.device)
    p[tables[s].long()[pos // PAGE], pos % PAGE] = new


def exact(case, seed):
    if case["kind"] == "decode":
        return _exact_decode(case, seed)
    _, tokens, past = _shape(case)
    w, x, pages, tables = _inputs(case, seed)
    w, x = {n: t.to(F64) for n, t in w.items()}, x.to(F64)
    if pages is not None:
        pages = pages.to(F64)
    if case["kind"] == "experts":
        return [_exact_experts(w, x)]
    _, kind, p, pos, _, axis = _params(case)
    ys, states, at = [], [], 0
    for s, (n, a) in enumerate(zip(tokens, past)):
        rows, at = x[at:at + n], at + n
        if kind in ("head_delta", "ssd"):
            y, state = (_exact_delta if kind == "head_delta" else _exact_ssd)(w, rows, p)
            states.append(state.reshape(-1))
        else:
            y = _exact_attention(kind, w, rows, p, pos, pages, tables, s, a, axis)
        ys.append(y)
    y = torch.cat(ys)
    if states:
        return [y, torch.stack(states)]
    return [y, None if case["variant"] == "window_pooled" else pages]


def _exact_attention(kind, w, x, p, pos, pages, tables, s, a, axis):
    T, H = x.shape[0], p["num_heads"]
    i = torch.arange(a, a + T, device=x.device)
    if kind == "latent_attention":
        return _exact_latent(w, x, p, pos, pages, tables, s, a, i, axis)
    G = p["num_kv_heads"]
    d = p.get("head_dim", p.get("dim"))
    scale = p.get("scale", 1 / math.sqrt(d))
    names = {"paged_attention": ("q_proj.weight", "k_proj.weight", "v_proj.weight", "o_proj.weight")}.get(kind, ("q", "k", "v", "o"))
    q, k = x @ w[names[0]].T, x @ w[names[1]].T
    v = k if kind == "keys_attention" else x @ w[names[2]].T
    if p.get("qkv_bias"):
        q, k, v = q + w["q.b"], k + w["k.b"], v + w["v.b"]
    if kind == "biased_attention":
        temp = torch.tensor([1.0 + TEMP_COEF * math.log((t + 1) // TEMP_EVERY + 1) for t in range(a, a + T)], dtype=F64, device=x.device)
        q, k = _rms(q, w["q.norm"], p["eps"]) * temp[:, None], _rms(k, w["k.norm"], p["eps"])
    q, k, v = q.view(T, H, d), k.view(T, G, d), v.view(T, G, d)
    if kind == "paged_attention":
        q, k = _rms(q, w["q_norm.weight"], 1e-6), _rms(k, w["k_norm.weight"], 1e-6)
    elif kind == "masked_attention" and p.get("qk_norm", True):
        q, k = _rms(q, w["q.norm"], p["eps"]), _rms(k, w["k.norm"], p["eps"])
    if pos is not None:
        q, k = _turn(q, i, pos), _turn(k, i, pos)
    pooled = p.get("pool", 0)
    if kind == "paged_attention":
        _put(pages, tables, s, a, torch.stack([k, v], 1), axis)
        e = _entries(pages, tables, s, a + T, axis)
        K, V = e[:, 0], e[:, 1]
    elif kind == "keys_attention":
        _put(pages, tables, s, a, k, axis)
        K = V = _entries(pages, tables, s, a + T, axis)
    elif pooled:
        new = _entries(pages, tables, s, a + T, axis).clone()        # [n, plane, G, 2 d]
        new[a:, 0] = torch.cat([k, v], -1)
        K, V = new[:, 0, :, :d], new[:, 0, :, d:]
        blocks = (a + T) // pooled
        mean = new[:blocks * pooled, 0].view(blocks, pooled, G, 2 * d).mean(1)
        done = a // pooled                                           # blocks that earlier steps closed: their means lie in the second plane
        mean[:done] = new[:done, 1]
    else:
        _put(pages, tables, s, a, torch.cat([k, v], -1), axis)
        e = _entries(pages, tables, s, a + T, axis)
        K, V = e[..., :d], e[..., d:]
    j = torch.arange(a + T, device=x.device)
    seen = j[None, :] <= i[:, None]
    if p.get("chunk"):
        seen = seen & (j[None, :] // p["chunk"] == i[:, None] // p["chunk"])
    if p.get("window"):
        seen = seen & ((i[:, None] - j[None, :] < p["window"]) | (j[None, :] < p.get("keep_first", 0)))
    dist = (i[:, None] - j[None, :]).clamp(min=0)
    if kind == "biased_attention":
        half = BIAS_ROWS // 2
        table = torch.tensor([n if n < half else min(BIAS_ROWS - 1, half + int(math.floor(math.log(n / half) / math.log(BIAS_FAR / half) * (BIAS_ROWS - half))))
                              for n in range(BIAS_FAR + 1)], device=x.device)
        bucket = table[dist.clamp(max=BIAS_FAR)]
    out = torch.empty(T, H, d, dtype=F64, device=x.device)
    for h in range(H):
        g = h // (H // G)
        sc = q[:, h] @ K[:, g].T * scale
        if p.get("softcap"):
            sc = p["softcap"] * torch.tanh(sc / p["softcap"])
        if p.get("distance_bias"):
            sc = sc - w["r1"][h] * torch.log1p(w["r2"][h] * dist)
        if kind == "biased_attention":
            sc = sc + w["rel"][:, h][bucket]
        sc = sc.masked_fill(~seen, -math.inf)
        vals = V[:, g]
        if pooled and blocks:
            sb = q[:, h] @ mean[:, g, :d].T * scale
            last = torch.arange(blocks, device=x.device) * pooled + pooled - 1
            sc = torch.cat([sc, sb.masked_fill(last[None, :] > i[:, None] - p["window"], -math.inf)], 1)
            vals = torch.cat([vals, mean[:, g, d:]])
        out[:, h] = _softmax_sum(sc, vals, w["sink"][h] if p.get("sink") else None)
    if p.get("head_gate"):
        out = out * torch.sigmoid(x @ w["g"].T)[:, :, None]
    out = out.reshape(T, H * d)
    if p.get("element_gate"):
        out = out * torch.sigmoid(x @ w["g"].T)
    return out @ w[names[3]].T


def _exact_latent(w, x, p, pos, pages, tables, s, a, i, axis):
    T, H, dn, dr, dv, R = x.shape[0], p["num_heads"], p["nope_dim"], p["rot_dim"], p["value_dim"], p["kv_rank"]
    q = (_rms(x @ w["dq"].T, w["dq.norm"], p["eps"]) @ w["uq"].T if p["q_rank"] else x @ w["q"].T).view(T, H, dn + dr)
    c = x @ w["dkv"].T
    lat, kr = _rms(c[:, :R], w["dkv.norm"], p["eps"]), _turn(c[:, None, R:], i, pos)[:, 0]
    _put(pages, tables, s, a, torch.cat([lat, kr], -1), axis)
    e = _entries(pages, tables, s, a + T, axis)
    qr = _turn(q[..., dn:], i, pos)
    hidden = torch.arange(a + T, device=x.device)[None, :] > i[:, None]
    out = torch.empty(T, H, dv, dtype=F64, device=x.device)
    for h in range(H):
        keys, vals = e[:, :R] @ w["uk"][h * dn:(h + 1) * dn].T, e[:, :R] @ w["uv"][h * dv:(h + 1) * dv].T
        sc = (q[:, h, :dn] @ keys.T + qr[:, h] @ e[:, R:].T) * p["scale"]
        out[:, h] = _softmax_sum(sc.masked_fill(hidden, -math.inf), vals, w["sink"][h] if p["sink"] else None)
    if p["gate"] == "head":
        out = out * torch.sigmoid(x @ w["g"].T)[:, :, None]
    out = out.reshape(T, H * dv)
    if p["gate"] == "element":
        out = out * torch.sigmoid(x @ w["g"].T)
    return out @ w["o"].T


def _silu(x):
    return x * torch.sigmoid(x)


def _conv(u, taps, bias=0.0):
    K = taps.shape[1]
    padded = torch.cat([torch.zeros(K - 1, u.shape[1], dtype=u.dtype, device=u.device), u])
    return _silu(sum(padded[j:j + u.shape[0]] * taps[:, j] for j in range(K)) + bias)


def _exact_delta(w, x, p):
    T, H, G, d = x.shape[0], p["num_heads"], p["num_kv_heads"], p["dim"]
    q, k, v = (_conv(x @ w[n].T, w[n + ".conv"]).view(T, -1, d) for n in ("q", "k", "v"))
    q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = (t.repeat_interleave(H // G, 1) for t in (q * d ** -0.5, k))
    beta = torch.sigmoid(x @ w["b"].T)[..., None]
    g = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a"].T + w["dt_bias"], threshold=60.0))[..., None, None]
    S, o = torch.zeros(H, d, d, dtype=F64, device=x.device), torch.empty(T, H, d, dtype=F64, device=x.device)
    for t in range(T):
        S *= g[t]
        u = beta[t] * (v[t] - torch.bmm(k[t][:, None, :], S)[:, 0])
        S.baddbmm_(k[t][:, :, None], u[:, None, :])
        o[t] = torch.bmm(q[t][:, None, :], S)[:, 0]
    y = _rms(o, w["norm"], p["eps"]) * _silu(x @ w["g"].T).view(T, H, d)
    return y.reshape(T, H * d) @ w["o"].T, S


def _exact_ssd(w, x, p):
    T, H, G, N, P = x.shape[0], p["num_heads"], p["groups"], p["state"], p["vdim"]
    inner, gn = H * P, G * N
    z, u, dt = (x @ w["in"].T).split([inner, inner + 2 * gn, H], 1)
    u = _conv(u, w["conv"], w["conv.b"])
    xs = u[:, :inner].view(T, H, P)
    B, C = (t.reshape(T, G, N).repeat_interleave(H // G, 1) for t in u[:, inner:].split(gn, 1))
    dt = torch.nn.functional.softplus(dt + w["dt_bias"], threshold=60.0)
    decay, dx = torch.exp(-torch.exp(w["A_log"]) * dt)[..., None, None], dt[..., None] * xs
    S, y = torch.zeros(H, N, P, dtype=F64, device=x.device), torch.empty(T, H, P, dtype=F64, device=x.device)
    for t in range(T):
        S *= decay[t]
        S.baddbmm_(B[t][:, :, None], dx[t][:, None, :])
        y[t] = torch.bmm(C[t][:, None, :], S)[:, 0]
    y = (y + w["D"][:, None] * xs).reshape(T, inner) * _silu(z)
    y = _rms(y.view(T, p["norm_parts"], -1), 1.0, p["eps"]).reshape(T, inner) * w["norm"]
    return y @ w["o"].T, S


def _exact_experts(w, x):
    z = x @ w["router"].T + w["router.b"]
    top, ids = z.topk(TOP, -1)
    share = torch.softmax(top, -1)
    y = torch.zeros_like(x)
    for e in range(EXPERTS):
        t, k = (ids == e).nonzero(as_tuple=True)
        h = _silu(x[t] @ w[f"e{e}.gate"].T) * (x[t] @ w[f"e{e}.up"].T)
        y.index_add_(0, t, share[t, k][:, None] * (h @ w[f"e{e}.down"].T))
    return y


def _exact_decode(case, seed):
    s, tokens, past = _shape(case)
    w, ids, cached = _decode_inputs(case, seed)
    w = {n: t.to(F64) for n, t in w.items()}
    H, G, d, pos = s["heads"], s["kv_heads"], s["dim"], dict(rotary_dim=s["dim"], theta=1e6, pairing="half")
    rows = []
    for r, kv in enumerate(cached):
        kv, at = kv.to(F64), torch.tensor([past[r]], device="cuda")
        h = w["model.embed_tokens.weight"][ids[0][r]][None]
        for i in range(DECODE_LAYERS):
            p = f"model.layers.{i}."
            x = _rms(h, w[p + "input_layernorm.weight"], 1e-6)
            q, k, v = ((x @ w[p + f"self_attn.{n}_proj.weight"].T).view(1, -1, d) for n in "qkv")
            q, k = (_turn(_rms(t, w[p + f"self_attn.{n}_norm.weight"], 1e-6), at, pos) for n, t in (("q", q), ("k", k)))
            K, V = torch.cat([kv[:, i, 0], k]).transpose(0, 1), torch.cat([kv[:, i, 1], v]).transpose(0, 1)
            sc = q.view(G, H // G, d) @ K.transpose(1, 2) / math.sqrt(d)
            h = h + _softmax_sum(sc, V).reshape(1, H * d) @ w[p + "self_attn.o_proj.weight"].T
            x = _rms(h, w[p + "post_attention_layernorm.weight"], 1e-6)
            h = h + (_silu(x @ w[p + "mlp.gate_proj.weight"].T) * (x @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
        rows.append(_rms(h, w["model.norm.weight"], 1e-6) @ w["model.embed_tokens.weight"].T)
    return [torch.cat(rows), None]


# ---- what a pass cannot do without -------------------------------------------------------------------------------------------

def _seen(case, a, n):
    """(query, key) pairs that the mask lets through, for a request's n tokens behind a cached ones."""
    _, _, p, _, _, _ = _params(case)
    total = 0
    for i in range(a, a + n):
        k = i + 1
        if p.get("chunk"):
            k = i % p["chunk"] + 1
        if p.get("window"):
            k = min(i + 1, p["window"]) + min(p.get("keep_first", 0), max(0, i + 1 - p["window"]))
            if p.get("pool"):
                k += max(0, i - p["window"] + 1) // p["pool"]
        total += k
    return total


def work(case):
    s, tokens, past = _shape(case)
    D, H, G, d, I, T = s["width"], s["heads"], s["kv_heads"], s["dim"], s["ff"], sum(tokens)
    size = 4 if case["dtype"] == "float32" else 2
    if case["kind"] == "decode":
        layer = D * (H + 2 * G) * d + H * d * D + 3 * D * I
        weights = DECODE_LAYERS * layer + DECODE_VOCAB * D
        kv = DECODE_LAYERS * 2 * G * d * sum(a + 1 for a in past)
        return {"bytes": 2 * (weights + kv) + 4 * T * DECODE_VOCAB, "flops": 2 * T * weights + 4 * DECODE_LAYERS * H * d * sum(a + 1 for a in past)}
    weights = sum(math.prod(shape) * (size if how.startswith("m") else 4) for shape, how in _weight_shapes(case).values())
    dense = sum(math.prod(shape) for shape, how in _weight_shapes(case).values() if how.startswith("m"))
    if case["kind"] == "experts":
        dense = TOP * 3 * D * (I // 2)
        weights = min(1.0, T * TOP / EXPERTS) * weights
    moved, flops = weights + 2 * T * D * size, 2.0 * T * dense
    entry = _params(case)[4]
    if entry is not None:
        moved += sum(a + 2 * n for a, n in zip(past, tokens)) * math.prod(entry) * size
        pairs = sum(_seen(case, a, n) for a, n in zip(past, tokens))
        if case["kind"] == "latent":       # over the latent itself, the up-projections on the queries' and the outputs' side
            flops += 2.0 * H * pairs * (2 * KV_RANK + ROT_DIM)
        else:
            flops += 4.0 * H * d * pairs
    elif case["kind"] in ("delta", "ssd"):
        floats = _matrix_floats(case)
        moved += 4 * floats * len(tokens)
        flops += T * floats * (7.0 if case["kind"] == "delta" else 5.0)
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    # measured against `exact`: a layer in 16 bits is 4e-3 to 6e-3 off (its largest value 0.12), eight whole layers 2.2e-2 to 2.8e-2 (0.12),
    # a layer in 32 bits 1.2e-6
    if case["dtype"] == "float32":
        return {"rel": 5e-6, "max": 5e-5}
    return {"rel": 0.03 if case["kind"] == "decode" else 0.015, "max": 0.5}
