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
