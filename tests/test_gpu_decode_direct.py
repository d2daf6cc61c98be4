"""Decode attention and its H2O update around the line between the two plans, against an fp32 reference on the cache's own
dequantised rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# most streams of a direct plan and one more; empty requests between others; lengths at page and block edges; one long
# stream (many blocks per request: the four-warp merge) and its planned counterpart; both formats, group sizes 1, 4 and 8
@pytest.mark.parametrize("B,ctx,n_q,n_kv,bits", [(512, 40, 4, 1, 8), (513, 40, 4, 1, 8), (7, 333, 8, 8, 8), (5, 1000, 16, 2, 4),
                                                 (3, 4097, 8, 2, 8), (1, 20000, 8, 2, 4), (1, 30000, 16, 2, 8), (2, 65, 4, 4, 8)])
@pytest.mark.parametrize("wide", [False, True])
def test_decode_attention_plans(B, ctx, n_q, n_kv, bits, wide):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pikv_b200
    gen = torch.Generator(device="cuda").manual_seed(B + ctx)
    seqs = B + 2
    # `wide` makes the page table so wide that the list cannot be taken for short: the same requests through the plan kernel
    cap = max(ctx, 64 * 2368 * 16 // (B * n_kv) + 64) if wide else ctx
    need = seqs * ((ctx + 15) // 16)
    cache = pikv_b200.PagedKVCache(seqs, cap, n_kv, bits=bits, symmetric=bits == 8, num_pages=need, identity_table=False)
    perm = torch.randperm(need, generator=gen, device="cuda").int().view(seqs, -1)
    cache.page_table[:, : perm.shape[1]] = perm
    pos = torch.arange(ctx, dtype=torch.int32, device="cuda")
    for s in range(seqs):
        k, v = (torch.randn(ctx, n_kv * 128, generator=gen, device="cuda").bfloat16() for _ in range(2))
        cache.append(k, v, torch.full_like(pos, s), pos)
    ids = torch.randperm(seqs, generator=gen, device="cuda")[:B].int()
    edge = torch.tensor([0, 1, 15, 16, 17, 63, 64, 65, ctx - 1, ctx], device="cuda")
    lens = edge[torch.randint(0, len(edge), (B,), generator=gen, device="cuda")].clamp(0, ctx).int()
    lens[-1] = ctx
    q = torch.randn(B, n_q, 128, generator=gen, device="cuda").bfloat16()
    out, lse = cache.decode_attention(q, seq_ids=ids, seq_len=lens, want_lse=True)
    acc = torch.zeros(B * n_kv, ctx + 1, device="cuda")          # rows at every 4-byte boundary
    if bits == 8:
        again = cache.decode_attention_h2o(q, acc, seq_ids=ids, seq_len=lens)
        assert torch.equal(again, out)
    cache.check_status()
    g = n_q // n_kv
    for b in range(0, B, max(1, B // 24)):
        n = int(lens[b])
        if n == 0:
            assert not out[b].any()
            continue
        rows = pos[:n]
        kd, vd = (cache.gather(torch.full_like(rows, int(ids[b])), rows, w).view(n, n_kv, 128) for w in ("k", "v"))
        s = torch.einsum("hgd,nhd->hgn", q[b].float().view(n_kv, g, 128), kd) / 128 ** 0.5
        p = torch.softmax(s, dim=-1)
        want = torch.einsum("hgn,nhd->hgd", p, vd).reshape(n_q, 128)
        # bf16 output (2^-8) and f16 probabilities (2^-11 each): 1e-2 of the largest value
        assert float((out[b].float() - want).abs().max()) <= 1e-2 * float(want.abs().max()) + 1e-6
        assert float((lse[b] - torch.logsumexp(s, -1).reshape(-1)).abs().max()) <= 2e-3
        if bits == 8:
            got = acc.view(B, n_kv, -1)[b]
            # f16 probabilities (2^-11) and the 15-bit query (2^-13 of a logit of order 10): 1e-2 of the probability
            assert float((got[:, :n] - p.sum(1)).abs().max()) <= 1e-2 * float(p.sum(1).max())
            assert not got[:, n:].any()
