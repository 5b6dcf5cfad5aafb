"""The grouped products of the experts at the edges of their tiles, against the same layer in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# rows per expert: none, one, around multiples of 16, 32 and the largest tile
COUNTS = {"edges": [0, 1, 15, 16, 17, 31, 32, 33, 0, 63, 64, 65], "tiles": [255, 256, 257, 0, 513, 5], "one": [0, 0, 3, 0]}
BF = torch.bfloat16


def _layer(x, ids, wts, wgu, wd, act, limit, alpha):
    """Rounded where the kernels round: both products, the activation and the sum."""
    T, D = x.shape
    y = torch.zeros(T, D, dtype=torch.float64, device=x.device)
    for k in range(ids.shape[1]):
        for e in range(wgu.shape[0]):
            t = (ids[:, k] == e).nonzero()[:, 0]
            if not len(t):
                continue
            h = (x[t].double() @ wgu[e].double().T).to(BF).double()
            if act == "relu2":
                h = torch.relu(h) ** 2
            else:
                g, u = h.chunk(2, -1)
                if act == "clamped":
                    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
                    h = g * torch.sigmoid(alpha * g) * (u + 1)
                else:
                    h = (g * torch.sigmoid(g)).to(BF).double() * u
            y[t] += wts[t, k].double()[:, None] * (h.to(BF).double() @ wd[e].double().T).to(BF).double()
    return y


@pytest.mark.parametrize("counts", sorted(COUNTS))
@pytest.mark.parametrize("act,D,F", [("silu", 136, 200), ("silu", 512, 256), ("relu2", 72, 264), ("clamped", 128, 72)])
@pytest.mark.parametrize("tile", [(256, 2), (256, 1), (64, 2), (32, 1)])
def test_expert_products_at_tile_edges(counts, act, D, F, tile):
    from cppvllm_b200.csrc import ops
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(hash((D, F)) % 1000)
    sizes = COUNTS[counts]
    E, T = len(sizes), sum(sizes)
    one = torch.cat([torch.full((n,), e) for e, n in enumerate(sizes)])[torch.randperm(T, generator=g)]
    ids = torch.stack([one, (one + 1) % E], 1).to(torch.int32)               # the second choice shifts every count by one expert
    wts = torch.rand(T, 2, generator=g)
    x = torch.randn(T, D, generator=g).to(BF)
    wgu = (torch.randn(E, F if act == "relu2" else 2 * F, D, generator=g) * D ** -0.5).to(BF)
    wd = (torch.randn(E, D, F, generator=g) * F ** -0.5).to(BF)
    x, ids, wts, wgu, wd = (t.to(dev) for t in (x, ids, wts, wgu, wd))
    R = ops.grouped_rows_tcgen05(T, 2, E)
    ints = dict(dtype=torch.int32, device=dev)
    scratch = [torch.full((n, m), float("nan"), dtype=BF, device=dev) for n, m in ((R, D), (R, F), (R, D))]
    y = torch.empty(T, D, dtype=BF, device=dev)
    ops.experts_grouped_tcgen05(y, x, ids, wts, wgu, wd, torch.empty(R // 128, **ints), torch.empty(R, **ints), torch.empty(T * 2, **ints), *scratch,
                                activation=act, limit=2.0, alpha=1.702, tile=tile)
    ops.check_device_errors(dev)
    ref = _layer(x, ids, wts, wgu, wd, act, 2.0, 1.702)
    # an intermediate may round the other way (float sums of up to 512 products against float64): one unit of bf16, 2^-8, on some of a row's
    # terms, and the last rounding; 2^-6 of the row's largest value covers both
    err = (y.double() - ref).abs().amax(1) / ref.abs().amax(1).clamp(min=1e-3)
    assert float(err.max()) < 2.0 ** -6, float(err.max())


@pytest.mark.parametrize("counts,beside", [([5, 0, 33, 2], 7), ([0, 0, 3, 0], 40), ([0, 0, 0, 0], 9), ([16, 17, 64, 1], 0)])
def test_pairs_whose_expert_is_the_input(counts, beside):
    """`beside` pairs have no row among the sorted ones; what the index scratch held before is no row of theirs either."""
    from cppvllm_b200.csrc import ops
    dev, D, F, E = torch.device("cuda:0"), 136, 72, len(counts)
    g = torch.Generator().manual_seed(beside)
    ids = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)] + [E + torch.randint(0, 3, (beside,), generator=g)])
    P = len(ids)
    ids = ids[torch.randperm(P, generator=g)].to(torch.int32).view(P, 1).to(dev)
    wts = torch.rand(P, 1, generator=g).to(dev)
    x = torch.randn(P, D, generator=g).to(BF).to(dev)
    wgu, wd = ((torch.randn(E, n, m, generator=g) * m ** -0.5).to(BF).to(dev) for n, m in ((2 * F, D), (D, F)))
    R = ops.grouped_rows_tcgen05(P, 1, E)
    ints = dict(dtype=torch.int32, device=dev)
    row_token = torch.full((R,), 1 << 30, **ints)
    scratch = [torch.full((R, m), float("nan"), dtype=BF, device=dev) for m in (D, F, D)]
    y = torch.empty(P, D, dtype=BF, device=dev)
    ops.experts_grouped_tcgen05(y, x, ids, wts, wgu, wd, torch.empty(R // 128, **ints), row_token, torch.empty(P, **ints), *scratch, identity=3)
    ops.check_device_errors(dev)
    own = (ids >= E).double()
    ref = _layer(x, ids, wts, wgu, wd, "silu", 0.0, 0.0) + own * wts.double() * x.double()
    err = (y.double() - ref).abs().amax(1) / ref.abs().amax(1).clamp(min=1e-3)
    assert float(err.max()) < 2.0 ** -6                        # as above
    assert row_token[P - beside:P].tolist() == [0] * beside
    assert int(row_token[:P].min()) >= 0 and int(row_token[:P].max()) < P


def test_scratch_is_as_large_as_the_pairs():
    """No room for padding: many experts with few pairs each ask for no more than the pairs and the experts' segments."""
    from cppvllm_b200.csrc import ops
    from cppvllm_b200.parts.base import Workspace
    dev, T, top, E, D, F = torch.device("cuda:0"), 40, 2, 64, 72, 40
    g = torch.Generator().manual_seed(1)
    ids = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).to(torch.int32).to(dev)
    wts, x = torch.rand(T, top, generator=g).to(dev), torch.randn(T, D, generator=g).to(BF).to(dev)
    wgu, wd = ((torch.randn(E, n, m, generator=g) * m ** -0.5).to(BF).to(dev) for n, m in ((2 * F, D), (D, F)))
    ws, y = Workspace(dev, T), torch.empty(T, D, dtype=BF, device=dev)
    ops.routed_experts(y, x, ids, wts, wgu, wd, workspace=ws, kernel="tcgen05")
    ops.check_device_errors(dev)
    assert sum(b.numel() * b.element_size() for b in ws._buffers.values()) <= T * top * (2 * (2 * D + F) + 2 * 4) + 2 * (E + 1) * 4
    ref = _layer(x, ids, wts, wgu, wd, "silu", 0.0, 0.0)
    err = (y.double() - ref).abs().amax(1) / ref.abs().amax(1).clamp(min=1e-3)
    assert float(err.max()) < 2.0 ** -6                        # as above


def test_a_call_makes_no_tensors():
    """Small steps wait for the host, where a view of the scratch costs as much as a launch's share of it."""
    from torch.utils._python_dispatch import TorchDispatchMode
    from cppvllm_b200.csrc import ops
    from cppvllm_b200.parts.base import Workspace
    dev, T, top, E, D, F = torch.device("cuda:0"), 40, 2, 8, 72, 40
    made = []

    class Count(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            made.append(str(func))
            return func(*args, **(kwargs or {}))
    ids, wts = torch.zeros(T, top, dtype=torch.int32, device=dev), torch.rand(T, top, device=dev)
    x, y, wgu, wd = (torch.zeros(*s, dtype=BF, device=dev) for s in ((T, D), (T, D), (E, 2 * F, D), (E, D, F)))
    ws = Workspace(dev, T)
    ops.routed_experts(y, x, ids, wts, wgu, wd, workspace=ws, kernel="tcgen05")       # makes the scratch
    with Count():
        ops.routed_experts(y, x, ids, wts, wgu, wd, workspace=ws, kernel="tcgen05")
    ops.check_device_errors(dev)
    assert made == []
