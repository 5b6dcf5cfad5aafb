"""What stands around attention by 16 bytes per thread, against plain arithmetic, at sizes that leave remainders."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF = "cuda:0", torch.bfloat16


def rnd(gen, *shape, dtype=torch.float32, scale=1.0):
    return (torch.randn(*shape, generator=gen) * scale).to(dtype).to(DEV)


def i32(x):
    return torch.as_tensor(x, dtype=torch.int32).to(DEV)


@pytest.mark.parametrize("dtype", [torch.float32, BF])
@pytest.mark.parametrize("per_element", [False, True])
def test_head_gate_and_turned_queries(dtype, per_element):
    from cppvllm_b200.csrc import ops
    gen = torch.Generator().manual_seed(5)
    T, H, vd = (5003, 16, 128) if per_element and dtype == BF else (37, 6, 24)
    o, gate = rnd(gen, H, T, vd, dtype=dtype), rnd(gen, T, (H * vd if per_element else H) + 16, dtype=dtype)
    g = gate[:, 8:8 + (H * vd if per_element else H)]
    out = torch.zeros(T, H * vd, dtype=dtype, device=DEV)
    ops.head_gate(out, o, g, H, vd, per_element=per_element)
    f = torch.sigmoid(g.double()).view(T, H, -1)
    want = (o.double().transpose(0, 1) * f).reshape(T, -1)
    tol = 2 ** -8 if dtype == BF else 1e-6                        # one rounding to the output's type
    assert bool(((out.double() - want).abs() <= tol * want.abs() + 1e-30).all())
    nope, rank, width, rot = 24, 32, 16, 8
    q, q_out = rnd(gen, T, H * (nope + width), dtype=dtype), torch.zeros(T, H * (rank + width), dtype=dtype, device=DEV)
    ang = torch.rand(T, rot // 2, generator=gen) * 6
    cos, sin = ang.cos().to(DEV), ang.sin().to(DEV)
    ops.latent_q_turn(q_out, q, H, nope, rank, width, rot, cos, sin, i32(torch.arange(T)))
    r = q.double().view(T, H, nope + width)[..., nope:]
    c, s = cos.double()[:, None], sin.double()[:, None]
    x, y = r[..., 0:rot:2], r[..., 1:rot:2]
    want = r.clone()
    want[..., 0:rot:2], want[..., 1:rot:2] = x * c - y * s, y * c + x * s
    got = q_out.double().view(T, H, rank + width)
    assert bool((got[..., :rank] == 0).all())
    bound = r.abs().amax(-1, keepdim=True) * 1.5
    assert bool(((got[..., rank:] - want).abs() <= tol * bound + 1e-30).all())


@pytest.mark.parametrize("dtype", [torch.float32, BF])
@pytest.mark.parametrize("nq,G,dk,dv,write", [(512, 2, 64, 32, True), (2048, 8, 128, 128, True), (6144, 2, 128, 128, True), (8192, 8, 64, 64, False)])
def test_norm_over_whole_projections(dtype, nq, G, dk, dv, write):
    from cppvllm_b200.csrc import ops
    gen = torch.Generator().manual_seed(nq)
    T, page, eps = 9, 16, 1e-5
    packed = rnd(gen, T, nq + (G * (dk + dv) if write else 0) + 8, dtype=dtype)
    wq, wk = rnd(gen, nq) * 0.1 + 1, rnd(gen, G * dk) * 0.1 + 1
    q, pages = torch.zeros(T, nq, dtype=dtype, device=DEV), torch.zeros(2, G, page, dk + dv, dtype=dtype, device=DEV)
    slots, pos = torch.randperm(2 * page, generator=gen)[:T], torch.arange(T) * 50
    ops.wide_qk_prep(q, packed, wq, i32(pos), eps, 0.25, 128, G, dk, dv, **(dict(pages=pages, k_weight=wk, slots=i32(slots), page_size=page) if write else {}))
    ops.check_device_errors(torch.device(DEV))

    def norm(x, w):
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()
    temp = torch.tensor([1 + 0.25 * math.log((int(p) + 1) // 128 + 1) for p in pos], dtype=torch.float64, device=DEV)[:, None]
    tol = 2 ** -8 if dtype == BF else 2e-6
    want = norm(packed[:, :nq].double(), wq) * temp
    assert bool(((q.double() - want).abs() <= tol * want.abs() + 1e-30).all())
    if write:
        k = norm(packed[:, nq:nq + G * dk].double(), wk).view(T, G, dk)
        v = packed[:, nq + G * dk:nq + G * (dk + dv)].double().view(T, G, dv)
        got = pages.double().movedim(2, 1)[slots.to(DEV) // page, slots.to(DEV) % page]
        assert bool(((got[..., :dk] - k).abs() <= tol * k.abs() + 1e-30).all()) and torch.equal(got[..., dk:], v)


@pytest.mark.parametrize("T,D,top,weighted", [(5, 1032, 2, True), (3, 8, 6, True), (2, 2048, 1, False), (4, 20, 3, True)])
def test_sum_of_a_tokens_expert_rows(T, D, top, weighted):
    from ctypes import c_int
    from cppvllm_b200.csrc import ops
    gen = torch.Generator().manual_seed(D)
    rows, x, y = rnd(gen, T * top + 3, D, dtype=BF), rnd(gen, T, D, dtype=BF), torch.zeros(T, D, dtype=BF, device=DEV)
    slot = torch.randperm(T * top + 3, generator=gen)[:T * top].view(T, top)
    slot[-1, -1] = -1                                    # the input itself
    w = torch.rand(T, top, generator=gen)
    wd, sd = w.to(DEV), i32(slot)
    assert ops._moe_lib().cvb_combine_pairs_bf16(ops._ptr(y), ops._ptr(rows), ops._ptr(x), ops._ptr(sd), ops._ptr(wd if weighted else None), c_int(T),
                                                 c_int(D), c_int(top), ops._stream()) == 0
    src = torch.where((slot >= 0)[..., None], rows.cpu().double()[slot.clamp(min=0)], x.cpu().double()[:, None])
    terms = src * (w.double()[..., None] if weighted else 1.0)
    # one rounding to bf16 behind float sums of a few terms
    assert bool(((y.cpu().double() - terms.sum(1)).abs() <= 2 ** -8 * terms.sum(1).abs() + 1e-6 * terms.abs().sum(1)).all())
