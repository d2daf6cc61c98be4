"""Errors of the operators that only a GPU can show."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_out_of_memory_is_torchs_own_error():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import ops
    g = ops.gate_fused(logits=torch.randn(64, 8, device="cuda"))
    with pytest.raises(torch.OutOfMemoryError):
        ops.dispatch_scatter(g, 8, 1 << 30)              # 2 TB
    d, _ = ops.dispatch_scatter(g, 8, 128)                # and the next call works
    assert int(d.sum()) == 128
