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


@pytest.mark.parametrize("H,G,dv,taps,lens,held,decay", [
    (2, 1, 128, 4, [[33], [64], [1]], 96, "mixed"), (4, 2, 64, 3, [[31, 65, 1], [40, 2, 97]], 96, "mixed"), (3, 3, 128, 1, [[200, 70]], 2, "mixed"),
    (2, 2, 128, 2, [[100]], 96, "one"), (2, 2, 128, 4, [[100]], 96, "zero"), (9, 3, 128, 4, [[50] * 8, [3] * 8], 96, "mixed")])
def test_against_the_rule_token_by_token(H, G, dv, taps, lens, held, decay):
    from cppvllm_b200.csrc import ops
    from cppvllm_b200.parts.base import Workspace
    dk, d = 128, torch.device("cuda:0")
    gen = torch.Generator().manual_seed(H * 1000 + dv)
    S, extra = len(lens[0]), 6
    slots = list(range(S, 0, -1))
    mat, C = H * dk * dv, 2 * G * dk + H * dv
    state = torch.randn(S + 1, mat + (taps - 1) * C + extra, generator=gen) * 0.1
    conv, dt_bias = torch.randn(C, taps, generator=gen) * 0.6, torch.randn(H, generator=gen)
    a_log = {"mixed": torch.randn(H, generator=gen) - 1, "one": torch.full((H,), -60.0), "zero": torch.full((H,), 8.0)}[decay]
    want_state = state.to(F).clone()
    on_gpu = state.to(d)
    ws = Workspace(d, 1024, 8)
    before, ops.DELTA_CHUNKS_HELD = ops.DELTA_CHUNKS_HELD, held
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=d)             # noqa: E731
    try:
        for step in lens:                                            # portions, one after the other
            T, off = sum(step), 2
            packed = torch.randn(T, off + C + 4, generator=gen).to(torch.bfloat16)
            a, b = torch.randn(T, H, generator=gen), torch.randn(T, H, generator=gen)
            cu, want = [0], []
            for s, n in enumerate(step):
                e = slice(cu[-1], cu[-1] + n)
                cu.append(cu[-1] + n)
                hist = want_state[slots[s], mat:mat + (taps - 1) * C].view(taps - 1, C)
                u = torch.cat([hist, packed[e, off:off + C].to(F)])
                y = sum(u[j:j + n] * conv[:, j].to(F) for j in range(taps))
                y = y / (1 + torch.exp(-y))
                unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)        # noqa: E731
                q, k, v = unit(y[:, :G * dk].view(n, G, dk)) * dk ** -0.5, unit(y[:, G * dk:2 * G * dk].view(n, G, dk)), y[:, 2 * G * dk:].view(n, H, dv)
                g = torch.exp(-torch.exp(a_log.to(F)) * torch.nn.functional.softplus(a[e].to(F) + dt_bias.to(F), threshold=60.0))
                M = want_state[slots[s], :mat].view(H, dk, dv)
                o, M = rule(q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1), v, g, torch.sigmoid(b[e].to(F)), M)
                want_state[slots[s], :mat] = M.reshape(-1)
                want_state[slots[s], mat:mat + (taps - 1) * C] = u[n:].reshape(-1)
                want.append(o)
            out = torch.full((T, H * dv), 9.0, device=d)
            dev = packed.to(d)
            ops.delta_chunks(out, dev, off, conv.to(d), torch.cat([b, a], 1).to(d), dt_bias.to(d), a_log.to(d), on_gpu, mat, i32(cu), i32(slots), step, H, G, dk, dv, ws)
            ops.conv_history(on_gpu, mat, dev, off, C, taps, i32(cu), i32(slots), S)
            torch.cuda.synchronize()
            ops.check_device_errors(d)
            got, want = out.cpu().to(F), torch.cat(want).reshape(T, -1)
            # A split product loses 2^-21 of an operand, twice; |q| <= 1, |k| = 1 and the states stay within a few times sqrt(dv): chains of
            # a few hundred such products stay below 1e-4 of the largest value, and on average, where their signs differ, below 1e-6 of the values
            assert float((got - want).abs().max()) < 1e-4 * float(want.abs().max())
            now = on_gpu.cpu().to(F)
            assert float((now - want_state).abs().max()) < 1e-4 * float(want_state.abs().max())
            assert float((got - want).norm()) < 1e-6 * float(want.norm()) and float((now - want_state).norm()) < 1e-6 * float(want_state.norm())
    finally:
        ops.DELTA_CHUNKS_HELD = before
    assert torch.equal(on_gpu[:, -extra:].cpu(), state[:, -extra:])


def test_what_the_rule_leaves_to_the_scan():
    from cppvllm_b200.csrc import ops
    state, row = torch.zeros(2, 128 * 128 + 1), torch.zeros(40, 513, dtype=torch.bfloat16)

    def ok(packed=row[:, :512].contiguous(), off=0, taps=4, H=4, dk=128, dv=128, w=128 * 128, n=64):
        return ops.delta_chunks_supported(packed, off, taps, H, 2, dk, dv, state[:, :w], [1, n])
    assert ok() and ok(dv=64) and ok(off=2)
    assert not ok(packed=row[:, :512].float()) and not ok(packed=row) and not ok(off=1) and not ok(taps=5)
    assert not ok(dk=64) and not ok(dv=96) and not ok(w=128 * 128 + 1) and not ok(n=63) and not ok(H=8)


@pytest.mark.parametrize("channel", ["q", "k", "v"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_bad_token_reaches_no_token_before_it(channel, bad):
    """As in the rule token by token: a bad query spoils the rows that its convolution reaches, a bad value its column from there on."""
    from cppvllm_b200.csrc import ops
    from cppvllm_b200.parts.base import Workspace
    gen, d = torch.Generator().manual_seed(6), torch.device("cuda:0")
    H, G, dk, dv, T, taps, at = 2, 1, 128, 128, 90, 4, 50
    mat, C = H * dk * dv, 2 * G * dk + H * dv
    packed = torch.randn(T, C, generator=gen).to(torch.bfloat16)
    conv, dt_bias, a_log = torch.randn(C, taps, generator=gen) * 0.6, torch.randn(H, generator=gen), torch.randn(H, generator=gen) - 1
    ba = torch.randn(T, 2 * H, generator=gen)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=d)             # noqa: E731

    def run():
        state, out = torch.zeros(1, mat + (taps - 1) * C, device=d), torch.zeros(T, H * dv, device=d)
        ops.delta_chunks(out, packed.to(d), 0, conv.to(d), ba.to(d), dt_bias.to(d), a_log.to(d), state, mat, i32([0, T]), i32([0]), [T], H, G, dk, dv,
                         Workspace(d, 1024, 8))
        return out.cpu()
    clean = run()
    packed[at, {"q": 3, "k": dk + 3, "v": 2 * dk + 3}[channel]] = bad
    got = run()
    assert torch.equal(got[:32], clean[:32])                         # the chunk in front; in its own a bad token's columns are summed another way
    assert float((got[:at] - clean[:at]).abs().max()) < 1e-6 * float(clean.abs().max()) and not bool(torch.isfinite(got[at:at + taps]).all())
    if channel == "q":
        assert torch.equal(got[at + taps:], clean[at + taps:])
    if channel == "v":
        others = [i for i in range(H * dv) if i != 3]
        assert torch.equal(got[:, others], clean[:, others]) and not bool(torch.isfinite(got[at:, 3]).any())


def test_steps_of_many_requests_stay_with_the_scan():
    from cppvllm_b200.csrc import ops
    state, row = torch.zeros(2, 128 * 128), torch.zeros(40, 512, dtype=torch.bfloat16)

    def ok(q_lens, H=16):
        return ops.delta_chunks_supported(row, 0, 4, H, H // 2, 128, 128, state, q_lens)
    assert ok([64] + [1] * 8) and not ok([64] + [1] * 9) and ok([1] * 64 + [512]) and not ok([1] * 65 + [512])
    assert ok([512] + [1] * 32, H=32) and not ok([512] + [1] * 33, H=32) and ok([200] * 8) and not ok([64] * 12)
