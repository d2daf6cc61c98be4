"""Calls that the operators take beside the usual ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda")


def test_capacity_as_a_float(dev):
    import pikv_b200
    from pikv_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(0)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()        # noqa: E731
    act, w2 = randn(40, 64), randn(8, 64)
    factor = 1.25 * 40 * 2 / 8                                   # 12.5 rows
    whole = ops.gate_fused(act, w2, capacity=12)
    assert torch.equal(ops.gate_fused(act, w2, capacity=factor).slot, whole.slot)
    w1 = randn(64, 64)
    assert torch.equal(ops.gate_mlp_fused(act, w1, None, w2, None, capacity=factor).slot, ops.gate_mlp_fused(act, w1, None, w2, None, capacity=12).slot)
    cache = pikv_b200.PagedKVCache(8, 64, 1)
    k = randn(40, 128)
    assert torch.equal(cache.route_append(act, w2, None, k, k, capacity=factor).new_len, whole.new_len)
