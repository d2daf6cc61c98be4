"""The tensor-core gate on short batches, whose tiles' hidden dimension is shared by the CTAs of a cluster."""
import numpy as np
import pytest
import torch

from oracle import pikv_oracle as O

pytestmark = pytest.mark.gpu


# tiles from one to more than the GPU holds clusters for (every cluster size), k blocks that do not divide by the number
# of CTAs, a ragged last block, and every width of the tail
@pytest.mark.parametrize("T,H,E", [(1, 4096, 8), (128, 1096, 16), (129, 2048, 64), (1537, 1600, 8), (2800, 4096, 24),
                                   (4700, 1024, 64), (7000, 520, 8), (9473, 512, 4)])
def test_gate_shared_hidden_dimension(T, H, E):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pikv_b200
    from pikv_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(T)
    act = torch.randn(T, H, generator=gen, device="cuda").bfloat16()
    w2 = (torch.randn(E, H, generator=gen, device="cuda") / H ** 0.5).bfloat16()
    b2 = torch.randn(E, generator=gen, device="cuda")
    g = ops.gate_fused(act, w2, b2, top_k=2, capacity=T)
    torch.cuda.synchronize()
    assert pikv_b200.lib().pikv_gate_error_state() == 0
    probs = torch.softmax(act.double() @ w2.double().T + b2.double(), dim=1)
    # fp32 sums of H products of unit variance over sqrt(H): a few 1e-6 on the logit, so on the probability's exponent
    assert float((g.probs.double() - probs).abs().max()) < 2e-5
    idx = g.topk_idx.cpu().numpy()
    assert np.array_equal(idx, np.argsort(-g.probs.cpu().numpy(), axis=1, kind="stable")[:, :2])
    slot, counts = O.slot_assign_fast(idx, E, T)
    assert np.array_equal(g.slot.cpu().numpy(), slot) and np.array_equal(g.counts_k.cpu().numpy(), counts)
    assert np.allclose(g.prob_sum.cpu().numpy(), g.probs.double().sum(0).cpu().numpy(), rtol=1e-5)
