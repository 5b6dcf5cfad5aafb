"""The float32 product on the tensor cores: edges of its tiles and stages, its error beside the library's, values without parts."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# around the rows of a block, the columns of a block and the 64 of K of a stage
SHAPES = [(1, 4, 4), (16, 128, 64), (31, 100, 60), (33, 130, 68), (65, 1, 128), (96, 257, 132), (127, 300, 516), (129, 96, 1024), (200, 640, 196)]


def _run(ops, x, w, tile=None):
    out = torch.full((x.shape[0], w.shape[0]), float("nan"), device=x.device)
    ops.gemm_f32_split(out, x, w, tile=tile)
    ops.check_device_errors(x.device)
    return out


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("rows", [32, 64, 96, 128])
@pytest.mark.parametrize("parts", [1, 2, 4, 8])
def test_edges(M, N, K, rows, parts):
    from cppvllm_b200.csrc import ops
    if parts > -(-K // 64):
        pytest.skip("fewer stages than parts")
    g = torch.Generator().manual_seed(M * 1000 + N)
    x, w = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
    out = _run(ops, x, w, (rows, parts))
    ref, mag = x.double() @ w.double().T, x.abs().double() @ w.abs().double().T
    # 2^-23 of every product for the parts left out; at most 9 truncated additions in tensor memory (128 of K by 16), 2^-23 each; as many
    # rounded additions as there are groups of 128 of K and parts, 2^-24 each
    bound = (1 + 9 + (K // 128 + 1 + parts) / 2) * 2.0 ** -23 * mag + 1e-37
    assert bool(((out.double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("M,N,K", [(17, 1024, 128), (33, 512, 320), (100, 256, 256), (17, 4096, 1024), (449, 1024, 2048), (300, 4096, 1024)])
def test_error_no_larger_than_the_library(M, N, K):
    from cppvllm_b200.csrc import ops
    ops.configure_library_matmul()
    g = torch.Generator().manual_seed(5)
    x, w = torch.randn(M, K, generator=g).cuda(), (torch.randn(N, K, generator=g) * 0.02).cuda()
    ref = x.double() @ w.double().T
    ours, lib = ((y.double() - ref).norm() / ref.norm() for y in (_run(ops, x, w), torch.mm(x, w.T)))
    assert float(ours) <= float(lib), (float(ours), float(lib))


def _one_sign(kind, shape, g):
    """Numbers from 1 up to 2 whose first part is a multiple of 2^-7, at the edges of the cuts."""
    a = 1 + torch.randint(0, 127, shape, generator=g) / 128.0
    if kind == "below a bf16":                   # cut off instead of rounded, all of the other two parts is there
        return a + 2.0 ** -7 - 2.0 ** -23 * torch.randint(1, 4, shape, generator=g)
    if kind == "below half a step":              # the second part is as large as it gets, the third of either sign
        return a + 2.0 ** -8 - 2.0 ** -17 + 2.0 ** -23 * torch.randint(-1, 2, shape, generator=g)
    return a + 2.0 ** -8 + 2.0 ** -17 * (1 - 2.0 ** -6)


@pytest.mark.parametrize("kind", ["below a bf16", "below half a step", "above half a step"])
@pytest.mark.parametrize("M,N,K", [(17, 200, 128), (40, 96, 384), (130, 300, 1024)])
def test_operands_of_one_sign_at_the_edges_of_the_cuts(kind, M, N, K):
    """Nothing cancels here, so what the cuts leave out adds up over K."""
    from cppvllm_b200.csrc import ops
    g = torch.Generator().manual_seed(K)
    x, w = _one_sign(kind, (M, K), g).cuda(), _one_sign(kind, (N, K), g).cuda()
    ref = x.double() @ w.double().T
    for tile in (None, (64, 1), (128, 2)):
        err = (_run(ops, x, w, tile).double() - ref) / ref
        # Sums of leading parts are exact in tensor memory (multiples of 2^-14 below 2^9), the others are below 2^-6 of them: 40 truncations of
        # 2^-23 of that at most.  2^-24 (1 + 2^-9) of every product is left out, a group of 128 of K is added with two roundings, each
        # of at most 2^-24 of what is there, and up to 8 parts of K with one.
        bound = (1 + 2.0 ** -9 + 40 * 2.0 ** -5 + 2 * -(-K // 128) + (0 if tile is None or tile[1] == 1 else 2)) * 2.0 ** -24
        if tile is None:
            bound += 8 * 2.0 ** -24
        assert float(err.abs().max()) <= bound
        assert abs(float(err.mean())) <= (1.5 + 40 * 2.0 ** -5) * 2.0 ** -24       # roundings to nearest leave no mean


@pytest.mark.parametrize("tile", [(32, 1), (64, 2), (128, 1)])
def test_infinities_and_nan(tile):
    """A row with a value that has no parts gives what float sums give; the other rows do not see it."""
    from cppvllm_b200.csrc import ops
    g = torch.Generator().manual_seed(7)
    x, w = torch.randn(40, 192, generator=g).cuda(), torch.randn(70, 192, generator=g).cuda()
    clean = _run(ops, x, w, tile)
    x[3, 5], x[17, 191], x[30, 64], x[39, 0] = float("inf"), float("-inf"), float("nan"), 3.4e38
    out, ref = _run(ops, x, w, tile), x.double() @ w.double().T
    assert bool(torch.isnan(out[30]).all()) and torch.equal(torch.isinf(out[3]), torch.isinf(ref[3])) and torch.equal(out[17].double(), ref[17])
    big = ref[39].abs() < 3.4e38
    assert bool(torch.isfinite(out[39][big]).all())
    rest = [i for i in range(40) if i not in (3, 17, 30, 39)]
    assert torch.equal(out[rest], clean[rest])


def test_a_long_kernel_in_front_does_not_run_out_the_waits():
    """The product may start beside the kernel before it, whose time is no part of its waits' limit (40 million cycles)."""
    from cppvllm_b200.csrc import ops
    dev, T, dim, vdim = torch.device("cuda:0"), 300000, 16, 64
    g = torch.Generator().manual_seed(9)
    q, k, v = (torch.randn(T, n, generator=g).to(dev) for n in (vdim, vdim, vdim))
    la, dt, skip = torch.full((T, 1), -0.5, device=dev), torch.full((T, 1), 0.1, device=dev), torch.ones(1, device=dev)
    out, state = torch.empty(T, vdim, device=dev), torch.zeros(1, dim * vdim, device=dev)
    cu, slots = (torch.tensor(x, dtype=torch.int32, device=dev) for x in ([0, T], [0]))
    x, w, y = out.view(-1)[-40 * 128:].view(40, 128), torch.randn(70, 128, generator=g).to(dev), torch.empty(40, 70, device=dev)

    def scan():                                # token by token in a block or two: the other SMs are free for the product
        ops.skip_scan(out, q[:, :dim], k[:, :dim], v, la, dt, skip, state, cu, slots, 1, 1, 1, dim, vdim)
    scan()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    scan()
    e1.record()
    torch.cuda.synchronize()
    assert e0.elapsed_time(e1) > 40.0          # more than the limit at any clock the GPU runs at under load
    out.zero_()
    scan()
    ops.gemm_f32_split(y, x, w)
    ops.check_device_errors(dev)
    torch.testing.assert_close(y.double(), x.double() @ w.double().T, rtol=1e-5, atol=1e-5 * float(x.abs().max()))
