"""The 16-byte forms of the cache writers beside what they take no part in: sizes and addresses that are no multiples of 16 bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,width,col0,extra,shift", [(8, 128, 0, 0, 0), (3, 8, 16, 8, 0), (2, 24, 4, 4, 0), (2, 20, 0, 0, 0), (1, 7, 3, 2, 0), (2, 16, 8, 0, 1)])
def test_rows_into_pages(dtype, heads, width, col0, extra, shift):
    from cppvllm_b200.csrc import ops
    dev, T, page = torch.device("cuda:0"), 37, 16
    src = torch.randn(T, col0 + heads * width + extra, device=dev).to(dtype)
    room = torch.zeros(6 * heads * page * width + shift, device=dev, dtype=dtype)[shift:].view(6, heads, page, width)
    slots = torch.randperm(6 * page, device=dev)[:T].to(torch.int32)
    slots[5] = -1
    ops.write_rows(room, src, slots, col0, heads, width, page)
    ops.check_device_errors(dev)
    want = torch.zeros_like(room)
    for t, s in enumerate(slots.tolist()):
        if s >= 0:
            want[s // page, :, s % page] = src[t, col0:col0 + heads * width].view(heads, width)
    assert torch.equal(room, want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("which", ["bias", "q", "k"])
def test_prep_with_vectors_off_16_bytes(dtype, which):
    """The same numbers at another address go another way and come out the same, up to the order of a sum of squares."""
    from cppvllm_b200.csrc import ops
    dev, T, H, G, d, page = torch.device("cuda:0"), 21, 6, 2, 64, 16
    g = torch.Generator().manual_seed(4)
    packed = torch.randn(T, (H + 2 * G) * d, generator=g).to(dev).to(dtype)
    vec = {"bias": torch.randn((H + 2 * G) * d, generator=g).to(dev), "q": torch.rand(d, generator=g).to(dev), "k": torch.rand(d, generator=g).to(dev)}
    outs = []
    for off in (False, True):
        v = dict(vec)
        if off:
            moved = torch.empty(v[which].numel() + 1, device=dev)[1:]
            v[which] = moved.copy_(v[which])
        q, pages = torch.zeros(T, H, d, device=dev, dtype=dtype), torch.zeros(4, 1, G, page, 2 * d, device=dev, dtype=dtype)
        ops.masked_qkv_prep(q, packed, H, G, d, d, 1e-5, q_weight=v["q"], k_weight=v["k"], bias=v["bias"], pages=pages,
                            slots=torch.arange(T, dtype=torch.int32, device=dev), page_size=page)
        outs.append((q.float(), pages.float()))
    ops.check_device_errors(dev)
    for a, b in zip(*outs):
        assert float(a.abs().max()) > 0
        torch.testing.assert_close(a, b, atol=0, rtol=2e-6 if dtype == torch.float32 else 2.0 ** -7)      # one unit in the last place


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,groups,G", [(1, 1, 4), (3, 5, 128), (2, 7, 132), (9, 3, 256), (5, 1, 260), (4, 2, 512)])
def test_gated_norm_by_rows_of_128(dtype, T, groups, G):
    from cppvllm_b200.csrc import ops
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(T * G)
    o, w = torch.randn(T, groups * G, generator=g).to(dev), torch.rand(G, generator=g).to(dev) + 0.5
    gate = torch.randn(T, groups * G + 8, generator=g).to(dev).to(dtype)[:, 4:-4]
    for act in ("sigmoid", "silu"):
        out = torch.full((T, groups * G + 4), 7.0, device=dev, dtype=dtype)
        ops.gated_norm(out[:, 4:], o, gate, w, groups, 1e-5, gate_act=act)
        x, z = o.double().view(T, groups, G), gate.double().view(T, groups, G)
        y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double() * torch.sigmoid(z) * (z if act == "silu" else 1)
        # a sum of G squares in float (half its error reaches the root), then five factors of one or two units in the last place each
        eps = G.bit_length() * 2.0 ** -24 + 12 * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
        err = (out[:, 4:].double().view_as(y) - y).abs()
        assert bool((err <= eps * y.abs() + 1e-30).all()), float((err / y.abs().clamp_min(1e-30)).max())
        assert bool((out[:, :4] == 7).all())
