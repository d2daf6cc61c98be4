"""Decode over a batch padded with stream ids outside the cache: zero rows, the status bit, and nothing else touched."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("wide", [False, True])      # short lists plan themselves, wide page tables take the plan kernel
def test_ids_outside_the_cache(bits, wide):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import pikv_b200
    gen = torch.Generator(device="cuda").manual_seed(3)
    seqs, n_kv, ctx = 5, 2, 70
    cap = 64 * 2368 * 16 // (6 * n_kv) + 64 if wide else ctx
    pages = (ctx + 15) // 16
    cache = pikv_b200.PagedKVCache(seqs, cap, n_kv, bits=bits, symmetric=bits == 8, num_pages=seqs * pages, identity_table=False)
    cache.page_table[:, :pages] = torch.arange(seqs * pages, dtype=torch.int32, device="cuda").view(seqs, -1)
    pos = torch.arange(ctx, dtype=torch.int32, device="cuda")
    for s in range(seqs):
        k, v = (torch.randn(ctx, n_kv * 128, generator=gen, device="cuda").bfloat16() for _ in range(2))
        cache.append(k, v, torch.full_like(pos, s), pos)
    cache.length.copy_(torch.tensor([70, 1, 33, 0, 64], dtype=torch.int32))
    ids = torch.tensor([2, -1, 0, seqs, 4, -2**31], dtype=torch.int32, device="cuda")
    good, bad = [0, 2, 4], [1, 3, 5]
    q = torch.randn(6, 8, 128, generator=gen, device="cuda").bfloat16()
    out, lse = cache.decode_attention(q, seq_ids=ids, want_lse=True)
    with pytest.raises(pikv_b200.PikvError, match="status"):
        cache.check_status()
    assert int(cache.status) == 1                    # PIKV_ST_BAD_SEQ alone
    cache.status.zero_()
    want, want_lse = cache.decode_attention(q[good].contiguous(), seq_ids=ids[good], seq_len=cache.length[ids[good].long()], want_lse=True)
    cache.check_status()
    assert not out[bad].any() and bool((lse[bad] == -float("inf")).all())
    # the list is cut elsewhere: bf16 results of the same f16 probabilities (2^-8 and 2^-11), 1e-2 of the largest value
    assert float((out[good].float() - want.float()).abs().max()) <= 1e-2 * float(want.abs().max())
    assert float((lse[good] - want_lse).abs().max()) <= 2e-3
    if bits == 8:
        acc = torch.full((6 * n_kv, ctx), 0.5, device="cuda")
        assert torch.equal(cache.decode_attention_h2o(q, acc, seq_ids=ids), out)
        rows = acc.view(6, n_kv, ctx)
        assert bool((rows[bad] == 0.5).all()) and bool(torch.isfinite(rows).all()) and bool((rows[good][:, :, 0] > 0.5).all())
