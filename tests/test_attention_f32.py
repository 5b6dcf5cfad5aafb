"""The tiled float32 attention of prompt portions (csrc/attention_f32.cu) against float64: portions around the tiles' edges, cached tokens, windows
whose older pages are gone, odd page sizes and groups."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
F = torch.float64


@pytest.mark.parametrize("H,KV,hd,page,window,reqs", [
    (4, 2, 128, 32, 0, [(65, 0), (1, 40), (31, 33)]), (3, 1, 64, 24, 0, [(50, 7)]), (2, 2, 64, 16, 20, [(90, 100), (8, 0)]),
    (16, 8, 128, 5, 100, [(33, 300)]), (64, 1, 64, 32, 0, [(33, 64)]), (5, 1, 128, 32, 1, [(40, 3)])])
def test_portions(H, KV, hd, page, window, reqs):
    from cppvllm_b200.csrc import ops
    gen, d = torch.Generator().manual_seed(H * hd + page), torch.device("cuda:0")
    per = [-(-(n + c) // page) for n, c in reqs]
    pages = torch.full((sum(per) + 1, 2, KV, page, hd), math.nan)
    order = torch.randperm(sum(per) + 1, generator=gen).tolist()
    tables = torch.full((len(reqs), max(per)), -1, dtype=torch.int32)
    qs, want, bound, pos, cu = [], [], [], [], [0]
    for s, (n, c) in enumerate(reqs):
        k, v, q = (torch.randn(m, x, hd, generator=gen) for m, x in ((n + c, KV), (n + c, KV), (n, H)))
        for b in range(per[s]):
            pg = order.pop()
            if window and (b + 1) * page <= c - window + 1:
                continue
            tables[s, b] = pg
            for i, t in enumerate((k, v)):
                rows = t[b * page:(b + 1) * page]
                pages[pg, i, :, :rows.shape[0]] = rows.movedim(0, 1)
        i, j = torch.arange(c, c + n)[:, None], torch.arange(n + c)[None, :]
        seen = (j <= i) & ((i - j < window) if window else True)
        kk, v2 = k.to(F).repeat_interleave(H // KV, 1), v.to(F).repeat_interleave(H // KV, 1)
        sc = torch.einsum("thd,jhd->htj", q.to(F), kk) / math.sqrt(hd)
        p = torch.softmax(sc.masked_fill(~seen, -math.inf), -1)
        want.append(torch.einsum("htj,jhd->thd", p, v2)), bound.append(torch.einsum("htj,jhd->thd", p, v2.abs()))
        qs.append(q.reshape(n, -1)), pos.append(i[:, 0]), cu.append(cu[-1] + n)
    T = cu[-1]
    out = torch.empty(T, H * hd, device=d)
    i32 = lambda x: torch.as_tensor(x, dtype=torch.int32).to(d)      # noqa: E731
    q_lens = [n for n, _ in reqs]
    assert ops.attn_prefill_f32_supported(torch.float32, H, KV, hd, q_lens)
    ops.attn_prefill_f32(out, torch.cat(qs).to(d), pages.to(d), i32(tables), i32(cu), i32(torch.cat(pos)), q_lens, H, KV, hd, page, 1 / math.sqrt(hd), window)
    torch.cuda.synchronize()
    ops.check_device_errors(d)
    err = (out.cpu().to(F).view(T, H, hd) - torch.cat(want)).abs()
    # a score's sum of hd products is off by at most hd 2^-24 of sum |q k| (here about 2 sqrt(hd)), which a probability feels as a factor; the
    # weighted sum adds (keys) 2^-24: 4e-5 of sum p |v| holds the sum of these with room
    assert bool((err <= 4e-5 * torch.cat(bound) + 1e-7).all())


def test_what_stays_with_the_general_kernel():
    from cppvllm_b200.csrc import ops
    ok = ops.attn_prefill_f32_supported
    assert ok(torch.float32, 4, 2, 128, [1, 32]) and not ok(torch.float32, 4, 2, 128, [1, 31]) and not ok(torch.float32, 4, 2, 32, [32])
    assert not ok(torch.bfloat16, 4, 2, 128, [32]) and not ok(torch.float32, 65, 1, 64, [32])


@pytest.mark.parametrize("window", [0, 20])
@pytest.mark.parametrize("plane", [0, 1])
@pytest.mark.parametrize("bad", [math.nan, math.inf])
def test_a_bad_token_reaches_no_token_that_does_not_see_it(window, plane, bad):
    from cppvllm_b200.csrc import ops
    gen, d = torch.Generator().manual_seed(5), torch.device("cuda:0")
    H, KV, hd, n, page, at = 4, 2, 128, 100, 32, 40
    pages, q = torch.randn(4, 2, KV, page, hd, generator=gen), torch.randn(n, H * hd, generator=gen)
    i32 = lambda x: torch.as_tensor(x, dtype=torch.int32).to(d)      # noqa: E731

    def run(p):
        out = torch.empty(n, H * hd, device=d)
        ops.attn_prefill_f32(out, q.to(d), p.to(d), i32([[0, 1, 2, 3]]), i32([0, n]), i32(range(n)), [n], H, KV, hd, page, 0.1, window)
        return out.cpu()
    clean = run(pages)
    pages[at // page, plane, :, at % page] = bad
    got = run(pages)
    sees = torch.zeros(n, dtype=torch.bool)
    sees[at:at + window if window else n] = True
    assert torch.equal(got[~sees], clean[~sees])
    if plane == 1:
        assert not torch.isfinite(got[sees]).any()


def test_steps_of_portions_and_single_tokens():
    from cppvllm_b200.csrc import ops
    ok = ops.attn_prefill_f32_supported
    assert ok(torch.float32, 16, 8, 128, [64] + [1] * 64) and not ok(torch.float32, 16, 8, 128, [64] + [1] * 65)
    assert ok(torch.float32, 16, 8, 128, [31] * 33 + [33]) and not ok(torch.float32, 16, 8, 128, [31] * 34 + [33])
    assert ok(torch.float32, 64, 1, 64, [65535]) and not ok(torch.float32, 64, 1, 64, [65536])            # a block holds one token of 64 heads
