"""Dense dispatch from a gate result that only has the tensors its position mode reads."""
import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,absent", [(0, ("counts_k", "prob_sum")), (1, ("slot", "prob_sum"))])
def test_dispatch_scatter_of_a_partial_result(mode, absent):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import PikvError, ops
    g = ops.gate_fused(logits=torch.randn(50, 8, device="cuda"))
    want = ops.dispatch_scatter(g, 8, 30, mode)
    part = dataclasses.replace(g, **dict.fromkeys(absent))
    for got, full in zip(ops.dispatch_scatter(part, 8, 30, mode), want):
        assert torch.equal(got, full)
    with pytest.raises(PikvError):
        ops.dispatch_scatter(part, 8, 30, 1 - mode)
