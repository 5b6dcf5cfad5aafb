"""The state-space recurrence in chunks of 128 tokens at the edges of its chunks, against the same recurrence in float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
N, P = 128, 64


def _run(q_lens, H, G, decay, kernel="tcgen05", seed=3, spoil=None):
    from cppvllm_b200.csrc import ops
    dev = torch.device("cuda:0")
    T, S = sum(q_lens), len(q_lens)
    g = torch.Generator().manual_seed(seed)
    u = torch.randn(T, H * P + 2 * G * N, generator=g).bfloat16()
    if spoil is not None:
        u[spoil] = float("nan")
    dt, skip = torch.rand(T, H, generator=g), torch.randn(H, generator=g)
    la = decay * torch.rand(T, H, generator=g)
    state = torch.randn(S + 1, H * N * P + 4, generator=g)
    slots = list(range(S, 0, -1))
    held = ops.ssd_held_chunks(max(T, 64))
    ends, decays = torch.full((held * H * N * P,), math.nan, device=dev), torch.full((held * H,), math.nan, device=dev)
    y, st = torch.full((T, H * P), math.nan, device=dev), state.to(dev)
    cu = [0]
    for n in q_lens:
        cu.append(cu[-1] + n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)                               # noqa: E731
    ops.ssd_chunks(y, u.to(dev), dt.to(dev), la.to(dev), skip.to(dev), st, i32(cu), i32(slots), q_lens, H, G, N, P, ends=ends, decays=decays, kernel=kernel)
    ops.check_device_errors(dev)
    return (u, dt, la, skip, state, slots, cu), y.cpu().view(T, H, P), st.cpu()


def _want(u, dt, la, skip, state, slots, cu, H, G):
    x, B, C = u[:, :H * P].double().view(-1, H, P), u[:, H * P:H * P + G * N].double().view(-1, G, N), u[:, H * P + G * N:].double().view(-1, G, N)
    B, C = (t.repeat_interleave(H // G, 1) for t in (B, C))
    y, after = torch.zeros_like(x), state.double().clone()
    for s, slot in enumerate(slots):
        M = state[slot, :H * N * P].double().view(H, N, P).clone()
        for t in range(cu[s], cu[s + 1]):
            M = torch.exp(la[t].double())[:, None, None] * M + (dt[t].double()[:, None] * B[t])[:, :, None] * x[t][:, None, :]
            y[t] = torch.einsum("hnp,hn->hp", M, C[t]) + skip.double()[:, None] * x[t]
        after[slot, :H * N * P] = M.reshape(-1)
    return y, after


@pytest.mark.parametrize("q_lens", [[1], [127], [128], [129], [300], [256, 1, 130], [1, 5, 128, 384], [33] * 5, [1] * 70 + [130, 2, 257]])
@pytest.mark.parametrize("H,G,decay", [(4, 2, -0.2), (3, 1, -1e-6), (2, 2, -60.0)])
def test_chunk_edges(q_lens, H, G, decay):
    args, y, st = _run(q_lens, H, G, decay)
    want, after = _want(*args, H, G)
    # operands are exact; the factors keep 16 bits (2^-17 of every addend), the running sums of up to 128 decays 2^-24 * 60 * 128 in the exponent
    # where a decay is that strong (and then the weight is 0): 3e-4 of the largest value covers hundreds of addends that do not cancel
    for got, ref in ((y, want), (st, after)):
        assert float((got.double() - ref).abs().max()) <= 3e-4 * float(ref.abs().max())
    assert torch.equal(st[0], args[4][0]) and torch.equal(st[:, H * N * P:], args[4][:, H * N * P:])


def test_as_close_as_chunks_of_64():
    args, y, st = _run([500, 77], 4, 2, -0.1)
    _, y2, st2 = _run([500, 77], 4, 2, -0.1, kernel="mma")
    want, after = _want(*args, 4, 2)
    for new, old, ref in ((y, y2, want), (st, st2, after)):
        a, b = (float((t.double() - ref).norm() / ref.norm()) for t in (new, old))
        assert a <= 1.25 * b, (a, b)                       # the same factors' rounding, over other partial sums


@pytest.mark.parametrize("q_lens", [[500, 77], [128]])
@pytest.mark.parametrize("decay", [-1e-3, -0.1, -0.8, -2.0, -8.0])
def test_no_further_off_than_chunks_of_64_at_any_decay(q_lens, decay):
    """Twice the tokens a chunk: the decays between them may not get coarser.  What is left is the factors' rounding to 16 bits, the same in
    both forms and 20 times that of the decays; means over six seeds, whose scatter is about 1 %."""
    mean = {}
    for kernel in ("tcgen05", "mma"):
        for seed in range(6):
            args, y, st = _run(q_lens, 4, 2, decay, kernel=kernel, seed=seed)
            for name, got, ref in zip(("y", "state"), (y, st), _want(*args, 4, 2)):
                mean[kernel, name] = mean.get((kernel, name), 0.0) + float((got.double() - ref).norm() / ref.norm()) / 6
    for name in ("y", "state"):
        assert mean["tcgen05", name] <= 1.03 * mean["mma", name], (name, mean)


def test_a_bad_token_reaches_no_token_before_it():
    args, clean, _ = _run([200], 2, 1, -0.1)
    _, y, _ = _run([200], 2, 1, -0.1, spoil=77)
    assert torch.isnan(y[77:]).all() and torch.isfinite(y[:77]).all()
    torch.testing.assert_close(y[:77], clean[:77], atol=1e-3 * float(clean.abs().max()), rtol=1e-3)
