"""Exponentials of the prompt kernels: a NaN, a score far below the row's largest and a row's only key, at neighbouring columns (they are made in
pairs, and a tile's in two halves)."""
import pytest
import torch

from test_kernels import build_paged, dev

pytestmark = pytest.mark.gpu
H, KV, HD, PAGE, C, N, DT = 4, 2, 128, 32, 900, 130, torch.bfloat16


def _attend(q, k, v, scale, first=C):
    from cppvllm_b200.csrc import ops
    n, d = q.shape[0], dev()
    cache, tables = build_paged([k], [v], PAGE, -(-(first + n) // PAGE) + 1, KV, HD, DT, torch.Generator().manual_seed(1))
    tiles = ops.prefill_tiles_tcgen05([n], H, KV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=d)                                 # noqa: E731
    out = ops.attn_prefill_tcgen05(torch.zeros(n, H * HD, dtype=DT, device=d), q.view(n, -1).to(d), cache.to(d), tables.to(d), i32([0, n]),
                                   i32(list(range(first, first + n))), 1, tiles, H, KV, HD, PAGE, scale)
    ops.check_device_errors(d)
    return out.cpu().view(n, H, HD)


def _random(first, n):
    g = torch.Generator().manual_seed(3)
    k, v = (torch.randn(first + n, KV, HD, generator=g).to(DT) for _ in range(2))
    return torch.randn(n, H, HD, generator=g).to(DT), k, v


@pytest.mark.parametrize("key", range(948, 955))
def test_a_nan_key_spoils_the_rows_that_see_it(key):
    q, k, v = _random(C, N)
    k[key, 1, 3] = float("nan")
    bad = torch.isnan(_attend(q, k, v, 0.1))
    want = torch.zeros(N, H, dtype=torch.bool)
    want[key - C:, 2:] = True
    assert torch.equal(bad.all(-1), want) and not bad[~want].any()


@pytest.mark.parametrize("key", range(6))
def test_a_score_far_below_the_largest_has_no_weight(key):
    """Its value would show: 2^100 times the smallest number that is not 0 changes the last places."""
    q, k, v = _random(C, N)
    q[:, :, 0], k[:, :, 0] = 1.0, 0.0
    k[key, :, 0], v[key] = -30000.0, 0.0
    clean = _attend(q, k, v, 0.1)
    v[key] = 2.0 ** 100
    assert torch.equal(_attend(q, k, v, 0.1), clean)


def test_rows_with_one_key_give_its_value():
    """Whichever column the only probability of a row lies in."""
    q, k, v = _random(0, 1 + N)
    q[:, :, :], k[:, :, :] = 0.0, 0.0
    q[:, :, 0] = 32.0
    k[:, :, 0] = torch.arange(1 + N).to(DT)[:, None]         # the own key outweighs the one before by 2^46
    out = _attend(q, k, v, 1.0, first=0)
    # the scores reach 6,000 in base 2, where a float's last place is 2^-11: 2^-12 in the exponent, and the two roundings to bf16
    torch.testing.assert_close(out.float(), v.repeat_interleave(H // KV, 1).float(), atol=0.0, rtol=2.0 ** -7)


def test_a_keys_weight_does_not_depend_on_its_column():
    """Two keys with a weight, one of weight 1; the other one's probability is the same number wherever it lies in a tile.  Of 131,072 scores some
    have an exponential within 1e-7 of the middle between two bf16, where two ways to make it would round apart."""
    n, g = 32768, torch.Generator().manual_seed(11)
    q, k, v = torch.zeros(n, H, HD), torch.zeros(C + n, KV, HD), torch.zeros(C + n, KV, HD)
    q[:, :, 0], q[:, :, 2], q[:, :, 1] = 0.5 + 7.0 * torch.rand(n, H, generator=g), torch.rand(n, H, generator=g), 1.0
    k[:, :, 1] = -30000.0                                    # no weight
    k[60] = 0.0                                              # weight 1, value 0
    first = None
    for column in (0, 1, 2, 3, 4, 5, 64, 65, 66, 67, 68, 69):
        k2, v2 = k.clone(), v.clone()
        k2[column, :, 0], k2[column, :, 2], k2[column, :, 1] = -1.0, -2.0 ** -7, 0.0
        v2[column] = 1.0
        out = _attend(q.to(DT), k2.to(DT), v2.to(DT), 0.7)
        first = out if first is None else first
        assert torch.equal(out, first), (column, int((out != first).any(-1).sum()))
