"""The two-layer gate net with its dense outputs at the edges of its tiles and of its two tail routes."""
import numpy as np
import pytest
import torch

from oracle import pikv_oracle as O

pytestmark = pytest.mark.gpu


# one token, ragged token pairs and hidden widths, the longest batch of the cluster tail and the first one past it, more
# blocks of hidden units than partial logits (K = H = 4608, T > 2048), every padded expert count, top-8
@pytest.mark.parametrize("T,K,H,E,k", [(1, 64, 64, 4, 2), (37, 72, 200, 3, 1), (255, 1024, 1000, 8, 2), (2048, 128, 4096, 16, 8),
                                       (2049, 256, 512, 8, 2), (2305, 64, 4608, 32, 2), (500, 64, 256, 64, 4)])
def test_gate_net_with_dense_outputs(T, K, H, E, k):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pikv_b200
    from pikv_b200 import ops
    gen = torch.Generator().manual_seed(T + H)
    rand = lambda *s: torch.rand(*s, generator=gen) * 2 - 1      # noqa: E731
    x, w1 = torch.randn(T, K, generator=gen).bfloat16(), (rand(H, K) / K ** 0.5).bfloat16()
    b1, w2, b2 = (rand(H) / K ** 0.5).bfloat16(), (rand(E, H) / H ** 0.5 * 4).bfloat16(), rand(E).bfloat16()
    cap = max(1, int(T * 1.5 * k / E))
    rows = min(cap, 40)
    args = [t.cuda() for t in (x, w1, b1, w2, b2)]
    for mode in (1, 0):
        g, (d, c, aux) = ops.gate_mlp_dense(*args, rows, mode, "entropy", 0.01, top_k=k, capacity=cap)
        torch.cuda.synchronize()
        assert pikv_b200.lib().pikv_gate_error_state() == 0
        hid = np.maximum(x.double().numpy() @ w1.double().numpy().T + b1.double().numpy(), 0).astype(np.float32)
        probs, _, _ = O.gate_tail(O.gate_logits(O.bf16_round(hid), w2.float().numpy(), b2.float().numpy()), k)
        # a hidden unit that rounds to the other bf16 (2^-8 of it) moves a logit by less than 1e-3 here
        assert np.abs(g.probs.cpu().numpy() - probs).max() < 2e-3
        got, tw, p = g.topk_idx.cpu().numpy(), g.topk_w.cpu().numpy(), g.probs.cpu().numpy()
        order = np.argsort(-p, axis=1, kind="stable")[:, :k]
        assert np.array_equal(got, order)                        # the kernel's own probabilities, ties to the lowest index
        slot, counts = O.slot_assign_fast(got, E, cap)
        assert np.array_equal(g.slot.cpu().numpy(), slot) and np.array_equal(g.counts_k.cpu().numpy(), counts)
        assert np.array_equal(g.new_len.cpu().numpy(), np.minimum(counts.sum(0), cap))
        assert np.allclose(g.prob_sum.cpu().numpy(), p.astype(np.float64).sum(0), rtol=1e-5)      # T additions in fp32
        wd, wc = np.zeros((T, E, rows), np.float32), np.zeros((T, E, rows), np.float32)
        for j in range(k):
            pos = slot[:, j] if mode == 0 else np.array([sum(counts[i, e] > 0 for i in range(j)) for e in got[:, j]])
            ok = (pos >= 0) & (pos < rows)
            wd[np.arange(T)[ok], got[ok, j], pos[ok]] = 1.0
            wc[np.arange(T)[ok], got[ok, j], pos[ok]] = tw[ok, j]
        assert np.array_equal(d.cpu().numpy(), wd) and np.array_equal(c.cpu().numpy(), wc)
        pm = p.astype(np.float64).mean(0)
        want = (pm * np.log(pm * E + 1e-9)).sum() + 0.01 * (pm * np.log(pm + 1e-9)).sum() / np.log(E)
        assert abs(float(aux) - want) < 1e-5 * max(1.0, abs(want))
