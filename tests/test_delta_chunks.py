"""The delta rule with one decay per head in chunks on the tensor cores (csrc/delta_chunks.cu) against the rule in float64: lengths around
the chunk's edges, requests side by side and continued, decays at their ends, and steps that go through the scratch in several turns."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F = torch.float64


def rule(q, k, v, g, b, S):
    """q, k [T, H, dk], v [T, H, dv], g, b [T, H], S [H, dk, dv]."""
    o = torch.zeros_like(v)
    for t in range(q.shape[0]):
        S = S * g[t][:, None, None]
        u = b[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        o[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return o, S


@pytest.mark.parametrize("H,G,dv,lens,held,decay", [
    (2, 1, 128, [[33], [64], [1]], 96, "mixed"), (4, 2, 64, [[31, 65, 1], [40, 2, 97]], 96, "mixed"), (3, 3, 128, [[200, 70]], 2, "mixed"),
    (2, 2, 128, [[100]], 96, "one"), (2, 2, 128, [[100]], 96, "zero"), (6, 3, 128, [[50] * 8], 96, "mixed")])
def test_against_the_rule_token_by_token(H, G, dv, lens, held, decay):
    from cppvllm_b200.csrc import ops
    from cppvllm_b200.parts.base import Workspace
    dk, d = 128, torch.device("cuda:0")
    gen = torch.Generator().manual_seed(H * 1000 + dv)
    S, extra = len(lens[0]), 6
    slots = [(3 * s + 1) % (S + 1) for s in range(S)] if S % 3 != 2 else list(range(S - 1, -1, -1))
    state = torch.randn(S + 1, H * dk * dv + extra, generator=gen) * 0.1
    want_state = state.to(F).clone()
    on_gpu = state.to(d)
    ws = Workspace(d, 1024, 8)
    before, ops.DELTA_CHUNKS_HELD = ops.DELTA_CHUNKS_HELD, held
    try:
        for step in lens:                                            # portions, one after the other
            T = sum(step)
            unit = lambda x: x / x.norm(dim=-1, keepdim=True)        # noqa: E731
            q, k = unit(torch.randn(T, G, dk, generator=gen)) * dk ** -0.5, unit(torch.randn(T, G, dk, generator=gen))
            v, b = torch.randn(T, H, dv, generator=gen), torch.rand(T, H, generator=gen)
            g = {"mixed": torch.rand(T, H, generator=gen) ** 0.2, "one": torch.ones(T, H), "zero": torch.zeros(T, H)}[decay]
            cu, want = [0], []
            for s, n in enumerate(step):
                a, e = cu[-1], cu[-1] + n
                cu.append(e)
                share = H // G
                M = want_state[slots[s], :H * dk * dv].view(H, dk, dv)
                o, M = rule(q[a:e].to(F).repeat_interleave(share, 1), k[a:e].to(F).repeat_interleave(share, 1), v[a:e].to(F), g[a:e].to(F), b[a:e].to(F), M)
                want_state[slots[s], :H * dk * dv] = M.reshape(-1)
                want.append(o)
            out = torch.full((T, H * dv), 9.0, device=d)
            i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=d)     # noqa: E731
            ops.delta_chunks(out, *(t.reshape(T, -1).contiguous().to(d) for t in (q, k, v, g, b)), on_gpu, i32(cu), i32(slots), step, H, G, dk, dv, ws)
            torch.cuda.synchronize()
            ops.check_device_errors(d)
            got, want = out.cpu().to(F), torch.cat(want).reshape(T, -1)
            # A split product loses 2^-17 of an operand, twice; |q| <= 1, |k| = 1 and the states stay within a few times sqrt(dv): chains of
            # a few hundred such products stay below 1e-4 of the largest value
            assert float((got - want).abs().max()) < 1e-4 * float(want.abs().max())
            now = on_gpu.cpu().to(F)
            assert float((now - want_state).abs().max()) < 1e-4 * float(want_state.abs().max())
    finally:
        ops.DELTA_CHUNKS_HELD = before
    assert torch.equal(on_gpu[:, -extra:].cpu(), state[:, -extra:])


def test_what_the_rule_leaves_to_the_scan():
    from cppvllm_b200.csrc import ops
    state = torch.zeros(2, 128 * 128 + 1)
    ok = lambda dt=torch.bfloat16, dk=128, dv=128, w=128 * 128, n=33: ops.delta_chunks_supported(dt, dk, dv, state[:, :w], [1, n])     # noqa: E731
    assert ok() and ok(dv=64)
    assert not ok(dt=torch.float32) and not ok(dk=64) and not ok(dv=96) and not ok(w=128 * 128 + 1) and not ok(n=32)
