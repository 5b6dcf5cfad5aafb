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
