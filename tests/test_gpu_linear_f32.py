"""The split-operand fp32 linear layer against float64, and its error against a plain fp32 layer's."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _error(y, want):
    return float((y.double() - want).norm() / want.norm())


# rows and outputs around the tile, more tiles than SMs, every number of k blocks (one and three: halves of unequal length)
@pytest.mark.parametrize("M,N,K", [(1, 1, 64), (127, 129, 64), (128, 128, 128), (129, 50257, 256), (33, 4099, 192), (1000, 2051, 256), (641, 1000, 128)])
@pytest.mark.parametrize("bias", [True, False])
def test_no_further_off_than_fp32_sums(M, N, K, bias):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    # rows of very different size, and entries of very different size within a row
    x = torch.randn(M, K, generator=g, device="cuda") * torch.exp(torch.randn(M, 1, generator=g, device="cuda") * 4)
    w = torch.randn(N, K, generator=g, device="cuda") * torch.exp(torch.randn(N, K, generator=g, device="cuda"))
    b = torch.randn(N, generator=g, device="cuda") if bias else None
    want = x.double() @ w.double().T + (b.double() if bias else 0.0)
    y = ops.linear_f32(x, w, b)
    ours = _error(y, want)
    # what K roundings of half an ulp of the growing sum can add up to
    assert ours < 2.0 ** -24 * K ** 0.5
    # any single output: two operands to 2^-23 each, the dropped product of the low limbs 2^-22, K additions of 2^-23 of the sum
    # so far, the bias
    terms = x.abs().double() @ w.abs().double().T + (b.abs().double() if bias else 0.0)
    assert bool(((y.double() - want).abs() <= (2.0 ** -21 + (K + 1) * 2.0 ** -23) * terms).all())
    if M >= 100:                            # enough outputs for the errors to be compared
        plain = _error(F.linear(x, w, b), want)
        assert ours <= 1.05 * plain, (ours, plain)
    assert _lib.lib().pikv_lowrank_error_state() == 0


def test_infinities_nans_and_extreme_rows():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(1)
    x, w, b = (torch.randn(*s, generator=g, device="cuda") for s in ((200, 128), (300, 128), (300,)))
    x[3, 5], x[70, 0], x[199, 127], w[131, 9], w[299, 1] = float("inf"), float("nan"), float("-inf"), float("inf"), float("nan")
    x[10], x[11], x[12], w[40], w[41] = 0.0, x[11] * 1e-37, x[12] * 1e30, 0.0, w[41] * 1e-30
    x[13, 1:] *= 1e-12                      # low limbs far below the row's largest
    y, want = ops.linear_f32(x, w, b), F.linear(x.double(), w.double(), b.double()).float()
    assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.equal(torch.isinf(y), torch.isinf(want))
    assert torch.equal(y[torch.isinf(y)], want[torch.isinf(want)])
    fine = torch.isfinite(want)
    scale = x.abs().nan_to_num(0, 0, 0) @ w.abs().nan_to_num(0, 0, 0).T + b.abs()        # the sum of the terms' magnitudes
    assert bool(((y - want).abs()[fine] <= 1e-6 * scale[fine]).all())
    assert ops.linear_f32(x.view(2, 100, 128), w, b).shape == (2, 100, 300)


def test_refuses_what_it_does_not_take():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import PikvError, ops
    x = torch.zeros(4, 320, device="cuda")
    for a, w in ((x, torch.zeros(8, 320, device="cuda")), (x[:, :96].contiguous(), torch.zeros(8, 96, device="cuda")),
                 (x[:, :64].contiguous(), torch.zeros(8, 128, device="cuda")), (x.double(), torch.zeros(8, 320, device="cuda"))):
        with pytest.raises(PikvError):
            ops.linear_f32(a, w)
