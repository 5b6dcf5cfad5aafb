"""Which float32 products go through the tensor cores, and with what: the route alone, without a GPU."""
import pytest
import torch

from cppvllm_b200.csrc import ops


@pytest.fixture
def taken(monkeypatch):
    """What project_rows handed on: ("split", dependent) or ("library",)."""
    calls = []
    monkeypatch.setattr(ops, "gemm_f32_split", lambda out, x, w, tile=None, dependent=True: calls.append(("split", dependent)) or out)
    monkeypatch.setattr(ops, "linear", lambda x, w, out=None: calls.append(("library",)) or out)
    return calls


@pytest.mark.parametrize("dependent", [True, False])
def test_a_product_that_has_to_stay_behind_its_predecessor_stays_there(taken, dependent):
    x, w = torch.zeros(64, 1024), torch.zeros(512, 1024)
    ops.project_rows(x, w, torch.zeros(64, 512), 64, dependent=dependent)
    assert taken == [("split", dependent)]


@pytest.mark.parametrize("rows,n_out,k,split", [
    (17, 1024, 1024, True), (16, 1024, 1024, False), (64, 2, 512, True), (64, 1, 512, False), (500, 1, 4096, False),          # one output
    (4096, 16, 512, True), (4096, 16, 508, False), (2048, 16, 256, True), (2049, 16, 256, False), (2049, 128, 256, True),      # few outputs
    (2048, 1024, 252, True), (2047, 1024, 252, False), (16384, 128, 128, True), (32768, 64, 128, False), (2048, 1024, 124, False)])
def test_which_product_is_faster(taken, rows, n_out, k, split):
    """Either side of every line of the rule."""
    ops.project_rows(torch.zeros(rows, k), torch.zeros(n_out, k), torch.zeros(rows, n_out), rows)
    assert taken == [("split", True) if split else ("library",)]


@pytest.mark.parametrize("change", ["k of 4", "offset", "row stride", "weight's stride", "short out", "no outputs", "half out", "many rows"])
def test_what_the_kernel_does_not_take_is_the_librarys(taken, change):
    x, w, out = torch.zeros(64, 1024), torch.zeros(512, 1024), torch.zeros(64, 512)
    if change == "k of 4":
        x, w = torch.zeros(64, 1022), torch.zeros(512, 1022)
    elif change == "offset":
        x = torch.zeros(64 * 1024 + 1)[1:].view(64, 1024)
    elif change == "row stride":
        x = torch.zeros(64, 1028)[:, :1024]
    elif change == "weight's stride":
        w = torch.zeros(1024, 512).t()
    elif change == "short out":
        out = torch.zeros(63, 512)
    elif change == "no outputs":
        w, out = torch.zeros(0, 1024), torch.zeros(64, 0)
    elif change == "half out":
        out = out.bfloat16()
    elif change == "many rows":
        x, w, out = (torch.empty(n, m, device="meta") for n, m in ((65535 * 32 + 1, 256), (128, 256), (65535 * 32 + 1, 128)))
    ops.project_rows(x, w, out, x.shape[0])
    assert taken == [("library",)]
