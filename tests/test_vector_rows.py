"""The 16-byte forms of the cache writers beside what they take no part in: sizes and addresses that are no multiples of 16 bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


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
