"""Whole layers at sizes where prompt portions take the kernels of their own (csrc/attention_entries_tcgen05.cu, delta_chunks.cu, attention_f32.cu):
prompts cut into portions, mixed with decoded tokens of other requests, against the same layer on the plain kernels (the general attention kernel,
the token-by-token scan).  Pages hold NaN where nothing has been written."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
PAGE, WIDTH = 32, 256


def layer(kind, seed=0, dtype=torch.bfloat16, plain=False, max_tokens=512, max_seqs=8, **over):
    """A mixer of `kind` with random weights; the same seed gives the same weights."""
    import cppvllm_b200.models  # noqa: F401
    import cppvllm_b200.parts  # noqa: F401
    from cppvllm_b200.parts.base import Runtime, Workspace, part_class
    dev = torch.device("cuda:0")
    H, G, d = over.pop("heads", 4), over.pop("kv_heads", 2), over.pop("dim", 128)
    rt = Runtime(dev, dtype, Workspace(dev, max_tokens, max_seqs), plain_kernels=plain, max_positions=4096)
    rotary = lambda n, pairing: part_class("position", "rotary")(rt, max_positions=4096, rotary_dim=n, theta=1e4, pairing=pairing)  # noqa: E731
    heads = dict(hidden_size=WIDTH, num_heads=H, num_kv_heads=G)
    if kind == "paged_attention":
        p = dict(heads, head_dim=d, position=rotary(d, "half"))
    elif kind == "masked_attention":
        p = dict(heads, dim=d, vdim=d, scale=1 / math.sqrt(d), eps=1e-5)
    elif kind == "keys_attention":
        p = dict(heads, head_dim=d)
    elif kind == "biased_attention":
        p = dict(heads, dim=d, vdim=d, scale=1 / math.sqrt(d), eps=1e-5, bias_max=100, bias_rows=16, temp_coef=0.2, temp_every=16)
    elif kind == "latent_attention":
        p = dict(hidden_size=WIDTH, num_heads=H, nope_dim=64, rot_dim=32, value_dim=64, kv_rank=96, scale=0.1, eps=1e-5, position=rotary(32, "interleaved"))
    else:
        p = dict(heads, dim=128, vdim=d, taps=4, eps=1e-5)
    part = part_class("mixer", kind)(rt, **dict(p, **over))
    gen = torch.Generator().manual_seed(seed)
    if kind == "paged_attention":
        shapes = {"q_proj.weight": (H * d, WIDTH), "k_proj.weight": (G * d, WIDTH), "v_proj.weight": (G * d, WIDTH), "o_proj.weight": (WIDTH, H * d),
                  "q_norm.weight": (d,), "k_norm.weight": (d,)}
    else:
        shapes = {n: s.shape for n, s in part.weight_specs().items()}
    w = {}
    for n, shape in shapes.items():
        t = torch.randn(*shape, generator=gen)
        if "norm" in n or n in ("r1", "r2"):
            t = 1 + 0.1 * t
        elif len(shape) == 2 and ".conv" not in n and n != "rel":
            t = (t * 1.5 / math.sqrt(shape[1])).to(dtype)
        elif n == "A_log":
            t = t - 3
        w[n] = t.to(dev)
    part.bind(w)
    return part


class Steps:
    """One layer with its cache or state over the steps of several requests."""

    def __init__(self, part, requests, longest, seed=0):
        from cppvllm_b200.parts.context import CacheUnitView
        self.part, self.rt, self.dev = part, part.rt, part.rt.device
        self.have, self.longest = {r: 0 for r in requests}, longest
        self.rows = {r: i for i, r in enumerate(requests)}
        spec = part.cache_spec()
        self.view = self.state = None
        if spec is not None:
            per = -(-longest // PAGE)
            n = per * len(requests)
            order = torch.randperm(n, generator=torch.Generator().manual_seed(seed)).view(len(requests), per)
            self.tables = order.to(torch.int32)
            self.pages = torch.full((n,) + spec.page_shape(PAGE), math.nan, dtype=self.rt.dtype, device=self.dev)
            self.view = CacheUnitView(self.pages, 0, spec)
        else:
            ss = part.state_spec()
            self.state = torch.zeros((len(requests) + 1,) + tuple(ss.shape), dtype=ss.dtype, device=self.dev)

    def __call__(self, x, step):
        """x [tokens, width]; step: (request, tokens) in order.  Entries of the block tables behind a request's last token stay -1."""
        from cppvllm_b200.parts.context import GroupStepView, StepContext
        i32 = lambda v: torch.as_tensor(v, dtype=torch.int32).to(self.dev)                       # noqa: E731
        cu, pos, seq_of, kv = [0], [], [], []
        for s, (r, n) in enumerate(step):
            a = self.have[r]
            cu.append(cu[-1] + n)
            pos += range(a, a + n)
            seq_of += [s] * n
            kv.append(a + n)
            self.have[r] = a + n
        groups = []
        if self.view is not None:
            tab = torch.stack([self.tables[self.rows[r]] for r, _ in step]).clone()
            slots = [int(tab[s, p // PAGE]) * PAGE + p % PAGE for s, p in zip(seq_of, pos)]
            for s, k in enumerate(kv):
                tab[s, -(-k // PAGE):] = -1
            groups = [GroupStepView(i32(tab), i32(slots), PAGE, self.pages.shape[0])]
        T = cu[-1]
        ctx = StepContext(num_tokens=T, num_seqs=len(step), tokens=i32([0] * T), positions=i32(pos), seq_of_token=i32(seq_of), cu_seqlens=i32(cu),
                          kv_lens=i32(kv), state_slots=i32([self.rows[r] for r, _ in step]), groups=groups, logit_rows=i32([T - 1]), num_logit_rows=1,
                          q_lens=[n for _, n in step], max_q_len=max(n for _, n in step), max_kv_len=max(kv), all_decode=all(n == 1 for _, n in step))
        y = self.part.forward(x, ctx, self.view, self.state).clone()
        from cppvllm_b200.csrc import ops
        torch.cuda.synchronize()
        ops.check_device_errors(self.dev)
        return y


MIXED = [[("a", 130)], [("b", 40)], [("a", 170), ("b", 1)], [("b", 1), ("c", 1), ("a", 1)], [("c", 210), ("a", 1), ("b", 1)], [("c", 1), ("a", 1), ("b", 1)]]


def both(monkeypatch, entry, kind, steps=MIXED, dtype=torch.bfloat16, longest=600, min_calls=1, **over):
    """The steps through the layer as it is and on the plain kernels: relative differences of every step's output, and how often `entry` ran."""
    from cppvllm_b200.csrc import ops
    calls, real = [], getattr(ops, entry)

    def counted(*a, **k):
        r = real(*a, **k)
        if r is not None:                # an answer of None: left to the other kernels
            calls.append(1)
        return r
    monkeypatch.setattr(ops, entry, counted)
    names = sorted({r for s in steps for r, _ in s})
    fast, plain = (Steps(layer(kind, dtype=dtype, plain=p, **over), names, longest) for p in (False, True))
    gen = torch.Generator().manual_seed(9)
    diffs = []
    for step in steps:
        x = torch.randn(sum(n for _, n in step), WIDTH, generator=gen).to(dtype).to("cuda:0")
        y, want = fast(x, step).double(), plain(x, step).double()
        assert bool(torch.isfinite(want).all())
        diffs.append(float((y - want).norm() / want.norm()))
    assert len(calls) >= min_calls, "the kernels under test were not reached"
    return diffs


# A layer in bf16 rounds its projections, the probabilities and its output, each to 2^-9 on average: two right ones are 2e-3 to 8e-3 apart.
BF16 = 2e-2


ROUTES = [("attn_entries_tcgen05", "masked_attention", dict(chunk=150, element_gate=True, qkv_bias=True)),
          ("attn_entries_tcgen05", "masked_attention", dict(chunk=200, softcap=5.0, distance_bias=True, sink=True, head_gate=True)),
          ("attn_entries_tcgen05", "masked_attention", dict(window=140, distance_bias=True, dim=64)),
          ("attn_entries_tcgen05", "masked_attention", dict(window=140, pool=16, heads=8)),
          ("attn_entries_tcgen05", "masked_attention", dict(window=140, keep_first=5, softcap=3.0, qk_norm=False)),
          ("attn_entries_tcgen05", "keys_attention", {}), ("attn_entries_tcgen05", "keys_attention", dict(window=140, keep_first=200, heads=6)),
          ("attn_entries_tcgen05", "latent_attention", dict(gate="element", q_rank=48)),
          ("attn_entries_tcgen05", "latent_attention", dict(gate="none", sink=True, heads=20)),
          ("attn_entries_tcgen05", "biased_attention", {}), ("attn_entries_tcgen05", "biased_attention", dict(dim=64, kv_heads=1)),
          ("delta_chunks", "head_delta", {}), ("delta_chunks", "head_delta", dict(dim=64, heads=3, kv_heads=1)),
          ("attn_prefill_f32", "paged_attention", {}), ("attn_prefill_f32", "paged_attention", dict(window=50, dim=64))]


@pytest.mark.parametrize("entry,kind,over", ROUTES)
def test_prompts_in_portions_beside_decoded_tokens(monkeypatch, entry, kind, over):
    exact = entry == "attn_prefill_f32"
    diffs = both(monkeypatch, entry, kind, dtype=torch.float32 if exact else torch.bfloat16, **over)
    assert max(diffs) < (1e-5 if exact else BF16), diffs


@pytest.mark.parametrize("scale", [0.0, -0.08])
@pytest.mark.parametrize("kind,over", [("keys_attention", {}), ("keys_attention", dict(window=100)), ("latent_attention", dict(sink=True)),
                                       ("masked_attention", dict(chunk=256)), ("masked_attention", dict(chunk=256, softcap=5.0)), ("biased_attention", {})])
def test_a_scale_that_is_not_positive(monkeypatch, kind, over, scale):
    """The tcgen05 kernel takes scores with a cap or a distance term at any scale and leaves the others at a scale of 0 or below to the mma.sync kernels."""
    terms = kind == "biased_attention" or "softcap" in over
    diffs = both(monkeypatch, "attn_entries_tcgen05", kind, min_calls=1 if terms else 0, scale=scale, **over)
    assert max(diffs) < BF16, diffs


def test_the_kernel_refuses_a_scale_it_would_apply_behind_the_mask():
    from cppvllm_b200.csrc import ops
    from cppvllm_b200.parts.base import Workspace
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    q, out, pages = (torch.zeros(*s, dtype=bf, device=dev) for s in ((8, 512), (8, 512), (2, 1, 2, PAGE, 256)))
    i32 = lambda v: torch.as_tensor(v, dtype=torch.int32).to(dev)                                # noqa: E731
    for scale in (0.0, -0.1, math.nan):
        assert not ops.attn_entries_supported(q, out, None, 4, 2, 128, 128, PAGE, 1000, scale=scale)
        assert ops.attn_entries_supported(q, out, None, 4, 2, 128, 128, PAGE, 1000, scale=scale, softcap=1.0)
        with pytest.raises(ops.KernelError):
            ops.attn_entries_tcgen05(out, q, pages, i32([[0, 1]]), i32([0, 8]), i32(range(8)), [8], 4, 2, 128, 128, PAGE, scale, 8, Workspace(dev, 64, 4))


def test_kept_first_tokens_with_a_distance_term(monkeypatch):
    """They are seen from beyond the chunk and the window: no table of distances is long enough, and the step stays with the other kernels."""
    diffs = both(monkeypatch, "attn_masked_bf16", "masked_attention", chunk=150, window=140, keep_first=100, distance_bias=True)
    assert max(diffs) < BF16, diffs


def test_an_optional_call_leaves_what_the_rule_refuses():
    from cppvllm_b200.csrc import ops
    from cppvllm_b200.parts.base import Workspace
    dev, bf = torch.device("cuda:0"), torch.bfloat16
    i32 = lambda v: torch.as_tensor(v, dtype=torch.int32).to(dev)                                # noqa: E731

    def ask(q=None, out=None, dim=128, q_lens=(8,), visible=500, heads=4, kv_heads=2, ws=None, **kw):
        q = torch.zeros(8, heads * dim, dtype=bf, device=dev) if q is None else q
        out = torch.zeros(8, heads * dim, dtype=bf, device=dev) if out is None else out
        pages = torch.zeros(2, 1, kv_heads, PAGE, 2 * dim, dtype=bf, device=dev)
        return ops.attn_entries_tcgen05(out, q, pages, i32([[0, 1]]), i32([0, 8]), i32(range(8)), list(q_lens), heads, kv_heads, dim, dim, PAGE, 0.1, visible,
                                        ws, optional=True, **kw)
    wide = torch.zeros(8, 4 * 128 + 4, dtype=bf, device=dev)
    assert ask() is not None
    for refused in (dict(visible=100), dict(dim=80), dict(q=wide[:, 4:]), dict(out=wide[:, 4:]), dict(gate=wide[:, 4:]), dict(q_lens=[131074], heads=128, kv_heads=1),
                    dict(table_len=20000, r1=torch.ones(4, device=dev), r2=torch.ones(4, device=dev))):
        before = ops.launches()
        assert ask(**refused) is None and ops.launches() == before
    ws = Workspace(dev, 64, 4)
    assert ask(visible=100, ws=ws) is None and 128 in ws.entry_pieces       # a graph captured later, for the longest context, finds its scratch
    torch.cuda.synchronize()
    ops.check_device_errors(dev)


def test_scratch_of_the_delta_rule_follows_the_largest_step_and_is_left_free():
    """What a step takes is what the part names, chunks for the largest step and no more; the pages' budget leaves it out."""
    from types import SimpleNamespace
    from cppvllm_b200.csrc import ops
    from cppvllm_b200.engine.runner import ModelRunner
    part = layer("head_delta", max_tokens=128, max_seqs=4)
    (name, size), = part.scratch_bytes().items()
    assert ops.delta_chunks_held(part.rt.workspace) == 128 // 32 + 4 and size == ops._delta_lib().cvb_delta_chunks_scratch(8, 4, 2, 128)
    run = Steps(part, ["a"], 128)
    run(torch.zeros(128, WIDTH, dtype=torch.bfloat16, device="cuda:0"), [("a", 128)])
    assert part.rt.workspace.flat(name, size, torch.uint8).numel() == size
    big = layer("head_delta", max_tokens=8192, max_seqs=64)
    assert ops.delta_chunks_held(big.rt.workspace) == ops.DELTA_CHUNKS_HELD
    assert layer("head_delta", plain=True).scratch_bytes() == {} and layer("head_delta", dtype=torch.float32).scratch_bytes() == {}

    def pages(*mixers):
        model = SimpleNamespace(hidden_size=64, vocab_size=100, blocks=[SimpleNamespace(mixer=m) for m in mixers])
        fake = SimpleNamespace(device=torch.device("cuda:0"), model=model, max_step_tokens=128, max_seqs=1 << 20, page_bytes=[1 << 16], table_width=1 << 20)
        return ModelRunner._pages_from_free_memory(fake, 0.9)
    other = layer("keys_attention")
    per = sum(big.scratch_bytes().values()) / 65536
    assert abs(pages(other) - pages(other, big, big) - per) < 0.02 * per + 64          # layers of one shape share it; other users' memory may move
