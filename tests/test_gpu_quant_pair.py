"""K and V of one forward through the paired block quantiser, against the numpy oracle."""
import numpy as np
import pytest
import torch

from oracle import pikv_oracle as O

pytestmark = pytest.mark.gpu


# row counts around a CTA's 32-row step and its warps; widths with a ragged last tile and last group; group sizes that
# are one chunk, a power-of-two number of chunks, an odd number of chunks, and not a multiple of a chunk (scalar loads)
@pytest.mark.parametrize("N,H,gs,bits,sym", [(1, 64, 64, 8, False), (31, 1000, 128, 8, False), (33, 1000, 200, 4, True),
                                             (257, 77, 7, 8, False), (4099, 256, 8, 4, False), (40, 2048, 2048, 8, True),
                                             (129, 130, 1, 8, False), (8192, 128, 100, 8, True)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_quant_block_pair_matches_oracle(N, H, gs, bits, sym, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import ops
    gen = torch.Generator().manual_seed(N + H)
    k, v = (torch.randn(N, H, generator=gen).mul(3).to(dtype) for _ in range(2))
    qmin, qmax = O.qrange(bits, sym)
    count = torch.tensor(3.0, device="cuda")
    dk, dv, mse = ops.quant_block_pair(k.cuda(), v.cuda(), gs, qmin, qmax, sym, sample_count=count, count_add=5.0)
    dq1, _, params, sq = ops.quant_block(v.cuda(), gs, qmin, qmax, sym)
    for got, x in ((dk, k), (dv, v)):
        want = torch.from_numpy(O.quant_block_forward(x.float().numpy(), bits, gs, sym)[0])
        assert torch.equal(got.cpu(), want.to(dtype))
    want, _, scale, zp, want_mse = O.quant_block_forward(v.float().numpy(), bits, gs, sym)
    assert np.array_equal(dq1.cpu().numpy(), want)
    assert np.array_equal(params.cpu().numpy(), np.stack([scale, zp], 1))
    # sums of at most N*gs squares in fp32, a few thousand terms deep per partial: 1e-5 of the sum on both sides
    ref = ((v.float().numpy().astype(np.float64) - want) ** 2)
    groups = (H + gs - 1) // gs
    for g in range(groups):
        s = ref[:, g * gs:(g + 1) * gs].sum()
        assert abs(float(sq[g]) - s) <= 1e-5 * s + 1e-20
    assert abs(float(mse) - ref[:, (groups - 1) * gs:].mean()) <= 1e-5 * ref[:, (groups - 1) * gs:].mean() + 1e-20
    assert float(count) == 8.0
