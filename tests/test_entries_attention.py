"""The tcgen05 attention of prompt portions over cache entries (csrc/attention_entries_tcgen05.cu) against plain arithmetic in float64, over
the masks, terms, gates, head counts, page sizes and cuttings it takes; what its rule refuses; and its row arithmetic."""
import math

import pytest
import torch

F = torch.float64


def test_rows_are_dealt_to_tokens_without_a_division():
    for g in range(1, 129):
        mul = ((1 << 20) + g - 1) // g
        assert all((r * mul) >> 20 == r // g for r in range(256))


def dev():
    return torch.device("cuda:0")


def plain(q, ent, blocks, pos, H, G, dk, dv, scale, shared, m):
    """q [T, H * dk], ent [n, G, E] the request's entries, blocks [nb, G, E] its pooled ones, pos [T]; returns o and sum p |v|, [T, H, dv]."""
    T, n = len(pos), ent.shape[0]
    i, j = pos[:, None], torch.arange(n)[None, :]
    seen = j <= i
    if m.get("chunk"):
        seen &= j // m["chunk"] == i // m["chunk"]
    if m.get("window"):
        seen &= (i - j < m["window"]) | (j < m.get("keep", 0))
    dist = (i - j).clamp(min=0)
    o, a = torch.zeros(T, H, dv, dtype=F), torch.zeros(T, H, dv, dtype=F)
    for h in range(H):
        g = h // (H // G)
        qh = q.view(T, -1)[:, h * dk:(h + 1) * dk]
        vals = ent[:, g, :dv] if shared else ent[:, g, dk:dk + dv]

        def capped(s):
            return m["cap"] * torch.tanh(s / m["cap"]) if m.get("cap") else s
        s = capped(qh @ ent[:, g, :dk].T * scale)
        if m.get("r1") is not None:
            s = s - m["r1"][h] * torch.log1p(m["r2"][h] * dist)
        if m.get("bias") is not None:
            s = s + m["bias"][h][dist.clamp(max=m["bias"].shape[1] - 1)]
        s = s.masked_fill(~seen, -math.inf)
        if blocks is not None and blocks.shape[0]:
            sb = capped(qh @ blocks[:, g, :dk].T * scale)
            last = torch.arange(blocks.shape[0])[None, :] * m["pool"] + m["pool"] - 1
            s = torch.cat([s, sb.masked_fill(last > i - m["window"], -math.inf)], 1)
            vals = torch.cat([vals, blocks[:, g, dk:dk + dv]])
        if m.get("sink") is not None:
            s = torch.cat([s, m["sink"][h].expand(T, 1)], 1)
        p = torch.softmax(s, -1)[:, :vals.shape[0]]
        o[:, h], a[:, h] = p @ vals, p @ vals.abs()
    return o, a


CASES = [
    # H, G, dk, dv, shared, page, mask and terms, gate, (tokens, cached) of every request, pieces (0: the rule's choice)
    (4, 2, 128, 128, False, 32, {}, None, [(130, 0)], 0),
    (4, 2, 128, 128, False, 16, {"chunk": 96}, "element", [(300, 50), (1, 40), (7, 0)], 0),
    (6, 2, 64, 64, False, 32, {"chunk": 200, "cap": 3.0, "dist": True, "sink": True}, "head", [(257, 0), (64, 333)], 0),
    (8, 2, 128, 128, False, 64, {"chunk": 1024, "cap": 30.0, "dist": True, "sink": True}, "head", [(500, 700)], 3),
    (4, 4, 128, 128, False, 32, {"window": 100, "pool": 16}, None, [(400, 0), (33, 1000)], 0),
    (4, 1, 64, 64, False, 16, {"window": 40, "pool": 8, "sink": True}, None, [(70, 2300)], 4),
    (8, 4, 128, 128, False, 32, {"window": 64, "keep": 5, "cap": 1.0}, None, [(300, 0), (20, 900), (2, 3)], 0),
    (4, 2, 128, 128, False, 128, {"window": 1, "keep": 130}, "element", [(260, 100)], 2),
    (32, 1, 128, 96, True, 32, {"sink": True}, None, [(50, 0), (9, 260)], 0),
    (12, 1, 128, 96, True, 32, {}, None, [(33, 2100)], 5),
    (8, 2, 128, 128, True, 32, {"window": 150, "keep": 4}, None, [(300, 0), (140, 400)], 0),
    (3, 3, 64, 64, True, 16, {"window": 300, "keep": 200}, None, [(260, 500)], 2),
    (4, 2, 128, 128, False, 32, {"bias": 33}, None, [(300, 0), (5, 77)], 0),
    (8, 2, 64, 64, False, 32, {"bias": 1025}, None, [(200, 2000)], 4),
    # requests shorter than what is kept: the block tables hold nothing behind them
    (4, 2, 128, 128, False, 32, {"window": 1024, "keep": 200}, None, [(130, 0)], 0),
    (8, 2, 128, 128, True, 16, {"window": 1024, "keep": 200}, None, [(5, 0), (300, 0)], 0),
    (4, 2, 64, 64, False, 64, {"window": 90, "keep": 500, "cap": 2.0}, "head", [(150, 0), (3, 190), (70, 400)], 0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(CASES)))
def test_portions_against_plain_arithmetic(case):
    from cppvllm_b200.csrc import ops
    from cppvllm_b200.parts.base import Workspace
    H, G, dk, dv, shared, page, mask, gate_kind, reqs, pieces = CASES[case]
    E, planes = (dk if shared else dk + dv), (2 if "pool" in mask else 1)
    gen = torch.Generator().manual_seed(case)
    bf = torch.bfloat16

    def rnd(*shape, scale=1.0):
        return torch.randn(*shape, generator=gen) * scale
    m = {k: mask[k] for k in ("chunk", "window", "pool", "keep", "cap") if k in mask}
    if mask.get("dist"):
        m["r1"], m["r2"] = 0.5 + torch.rand(H, generator=gen), 0.5 + torch.rand(H, generator=gen)
    if mask.get("sink"):
        m["sink"] = rnd(H)
    if mask.get("bias"):
        m["bias"] = rnd(H, mask["bias"])
    per = [-(-(n + c) // page) for n, c in reqs]
    n_pages, order = sum(per) + 2, torch.randperm(sum(per) + 2, generator=gen).tolist()
    pages = torch.full((n_pages, planes, G, page, E), math.nan)                 # what nobody may read: NaN
    tables = torch.full((len(reqs), max(per)), -1, dtype=torch.int32)
    qs, want, bound, positions, gates = [], [], [], [], []
    scale = 2.0 / math.sqrt(dk)
    for s, (n, c) in enumerate(reqs):
        ent = rnd(n + c, G, E).to(bf)
        first = 0                                                             # pages wholly behind the window may be gone
        if m.get("window") and not m.get("pool"):
            first = max(0, c - m["window"] + 1) // page
        for b in range(per[s]):
            pg = order.pop()
            if first > b and b * page >= m.get("keep", 0):
                continue
            tables[s, b] = pg
            rows = ent[b * page:(b + 1) * page]
            pages[pg, 0, :, :rows.shape[0]] = rows.movedim(0, 1).float()
        blocks = None
        if m.get("pool"):
            nb = (n + c) // m["pool"]
            blocks = rnd(nb, G, E).to(bf)
            for b in range(nb):
                pages[int(tables[s, b // page]), 1, :, b % page] = blocks[b].float()
        q = rnd(n, H * dk).to(bf)
        pos = torch.arange(c, c + n)
        o, a = plain(q.to(F), ent.to(F), blocks.to(F) if blocks is not None else None, pos, H, G, dk, dv, scale, shared,
                     {k: (v.to(F) if torch.is_tensor(v) else v) for k, v in m.items()})
        out_scale = 0.7
        gate = None
        if gate_kind:
            gate = rnd(n, H if gate_kind == "head" else H * dv).to(bf)
            f = torch.sigmoid(gate.to(F)).view(n, H, -1)
            o, a = o * f, a * f
        qs.append(q), want.append(o * out_scale), bound.append(a * out_scale), positions.append(pos), gates.append(gate)
    T = sum(n for n, _ in reqs)
    d = dev()
    lead = 16                                                                  # q, gate and out as columns of wider rows
    q_wide = torch.zeros(T, H * dk + lead, dtype=bf, device=d)
    q_wide[:, :H * dk] = torch.cat(qs).to(d)
    gate = None
    if gate_kind:
        g_all = torch.cat(gates)
        gate = torch.zeros(T, g_all.shape[1] + lead, dtype=bf, device=d)
        gate[:, lead:] = g_all.to(d)
        gate = gate[:, lead:]
    out = torch.full((T, H * dv + 2 * lead), 5.0, dtype=bf, device=d)
    cu = torch.tensor([0] + [sum(n for n, _ in reqs[:k + 1]) for k in range(len(reqs))], dtype=torch.int32, device=d)

    def on(t):
        return t.to(torch.float32).to(d) if t is not None else None
    reach = m.get("chunk", 0) if m.get("r1") is not None else mask.get("bias", 0)
    view = out[:, lead:lead + H * dv]
    assert ops.attn_entries_supported(q_wide, view, gate, H, G, dk, dv, page, 128, shared=shared, table_len=reach)
    ops.attn_entries_tcgen05(view, q_wide, pages.to(bf).to(d), tables.to(d), cu, torch.cat(positions).to(torch.int32).to(d), [n for n, _ in reqs], H, G,
                             dk, dv, page, scale, 1 << 20 if pieces else 1, workspace=Workspace(d, 1024, 8), shared=shared, planes=planes,
                             chunk=m.get("chunk", 0), window=m.get("window", 0), pool=m.get("pool", 0), keep_first=m.get("keep", 0),
                             softcap=m.get("cap", 0.0), bias=on(m.get("bias")), r1=on(m.get("r1")), r2=on(m.get("r2")), table_len=reach,
                             sink=on(m.get("sink")), gate=gate, out_scale=0.7, pieces=pieces, min_rounds=2 if pieces else 0)
    torch.cuda.synchronize()
    ops.check_device_errors(d)
    want, bound = torch.cat(want), torch.cat(bound)
    got = view.to(F).cpu().view(T, H, dv)
    # probabilities and outputs are rounded to bf16 (at most 2^-8 of their value each, 8 significant bits), the rest is float and far smaller
    assert bool(((got - want).abs() <= 2 ** -7 * bound + 1e-5).all()), float(((got - want).abs() / bound).max())
    assert bool((out[:, :lead] == 5).all()) and bool((out[:, lead + H * dv:] == 5).all())


@pytest.mark.gpu
def test_what_the_rule_leaves_to_the_other_kernels():
    from cppvllm_b200.csrc import ops
    d, bf = dev(), torch.bfloat16
    q, out = torch.zeros(8, 4 * 128, dtype=bf, device=d), torch.zeros(8, 4 * 128, dtype=bf, device=d)

    def takes(q, out, gate, dk, dv, page, visible=1000, **kw):
        return ops.attn_entries_supported(q, out, gate, 4, 2, dk, dv, page, visible, **kw)
    assert takes(q, out, None, 128, 128, 32)
    assert not takes(q, out, None, 128, 128, 32, visible=100)        # less than a tile to see
    assert not takes(q, out, None, 128, 64, 32)                      # values of another width
    assert not takes(q, out, None, 112, 112, 32)                     # other sizes
    assert not takes(q, out, None, 128, 128, 24)                     # pages that are no power of two
    assert not takes(q, out, None, 128, 128, 8)                      # or short
    assert not takes(q, out, None, 128, 128, 32, table_len=8192)     # a distance table that does not fit
    assert not takes(q.float(), out, None, 128, 128, 32)
    wide = torch.zeros(8, 4 * 128 + 4, dtype=bf, device=d)
    assert not takes(wide[:, 4:], out, None, 128, 128, 32)           # rows that start off 16 bytes
    assert not takes(q, wide[:, 4:], None, 128, 128, 32)
    assert not takes(q, out, wide[:, 4:], 128, 128, 32)
    assert not takes(q, out, None, 128, 96, 32)                      # 96 of 128 only where one entry is key and value


def one_request(H, G, dim, shared, n, cached, page=32, seed=3):
    """A request's queries and pages (in order, all in use), bf16 on the host."""
    gen = torch.Generator().manual_seed(seed)
    pages = torch.randn(-(-(n + cached) // page), 1, G, page, dim if shared else 2 * dim, generator=gen).to(torch.bfloat16)
    return torch.randn(n, H * dim, generator=gen).to(torch.bfloat16), pages


def run_one(q, pages, H, G, dim, shared, n, cached, pieces=1, scale=0.1, **kw):
    from cppvllm_b200.csrc import ops
    from cppvllm_b200.parts.base import Workspace
    d = dev()

    def i32(x):
        return torch.as_tensor(x, dtype=torch.int32).to(d)
    out = torch.zeros(n, H * dim, dtype=torch.bfloat16, device=d)
    ops.attn_entries_tcgen05(out, q.to(d), pages.to(d), i32([list(range(pages.shape[0]))]), i32([0, n]), i32(range(cached, cached + n)), [n], H, G, dim, dim,
                             pages.shape[3], scale, 1 << 20 if pieces > 1 else 1, workspace=Workspace(d, 1024, 8), shared=shared, pieces=pieces,
                             min_rounds=2, **kw)
    torch.cuda.synchronize()
    ops.check_device_errors(d)
    return out.cpu().view(n, H, dim)


@pytest.mark.gpu
@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("pieces", [1, 4])
def test_a_nan_is_answered_with_nan(shared, pieces):
    """A NaN in a key spoils the rows that see it, a NaN in a query its own row, and no other, whether the query block is cut or not."""
    H, G, dim, n, cached = 4, 2, 128, 40, 2100
    q, pages = one_request(H, G, dim, shared, n, cached)
    pages[700 // 32, 0, 1, 700 % 32, 3] = math.nan
    q[5, 7] = math.nan
    out = run_one(q, pages, H, G, dim, shared, n, cached, pieces)
    want = torch.zeros(n, H, dtype=torch.bool)
    want[:, 2:] = True
    want[5, 0] = True
    assert torch.equal(torch.isnan(out).all(-1), want) and not torch.isnan(out[~want]).any()


@pytest.mark.gpu
def test_a_cap_does_not_depend_on_what_unused_slots_hold():
    H, G, dim, n, cached = 4, 2, 128, 300, 77
    q, pages = one_request(H, G, dim, False, n, cached)
    outs = []
    for factor in (0.01, 3000.0):
        pages[-1, :, :, (n + cached) % 32:] *= factor
        outs.append(run_one(q, pages, H, G, dim, False, n, cached, softcap=30.0, chunk=200))
    assert torch.equal(*outs)


@pytest.mark.gpu
def test_the_largest_probability_of_a_row_is_not_rounded():
    """Two keys that count, one in the first tile and one in the last with 7 to 200 times its weight, and values of 1: the weighted sum over the sum of the
    weights is 1, where the larger weight is 1 and rounds to bf16 as 1 (the smaller one, at most 0.14, is off by 3e-4; outputs below 1 are 4e-3 apart)."""
    H, G, dim, n, cached, heavy = 2, 2, 128, 32, 480, 480
    for k in range(20, 56, 3):                               # times 0.1: the larger score; the smaller one is 0, the others -100
        q, pages = one_request(H, G, dim, False, n, cached)
        q[:], pages[..., :dim], pages[..., dim:] = 0, 0, 1
        q[:, 0], q[:, dim] = 1, 1
        pages[..., 0] = -1000
        pages[0, 0, :, 0, 0], pages[heavy // 32, 0, :, heavy % 32, 0] = 0, k
        out = run_one(q, pages, H, G, dim, False, n, cached)
        assert bool((out == 1).all()), (k, float(out.min()), float(out.max()))
