"""The tensors of a gate result are independent of each other."""
import io

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_storage_each():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import ops
    g = ops.gate_fused(logits=torch.randn(4096, 64, device="cuda"))
    parts = [t for t in g.tensors() if t is not None]
    assert len({t.untyped_storage().data_ptr() for t in parts}) == len(parts)
    saved = io.BytesIO()
    torch.save(g.new_len, saved)                       # 256 bytes of values
    assert saved.getbuffer().nbytes < 8192
