"""The split-operand fp32 linear layer where a row's entries differ by many powers of two."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


# a large entry of one operand that meets a zero of the other leaves the small entries as the whole result; the spreads end on
# both sides of 2^27, where the limbs give way to plain sums
@pytest.mark.parametrize("spread", [12, 18, 24, 26, 27, 28, 29, 40, 60])
@pytest.mark.parametrize("side", ["x", "w", "some"])
def test_large_entries_that_meet_zeros(spread, side):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(spread)
    M, N, K = 300, 1000, 256
    x, w = (torch.randn(n, K, generator=g, device="cuda") for n in (M, N))
    big, other = (w, x) if side == "w" else (x, w)
    rows = slice(None) if side != "some" else slice(3, None, 41)
    big[rows, 77] = 2.0 ** spread
    other[:, 77] = 0.0
    want = x.double() @ w.double().T
    y = ops.linear_f32(x, w)
    error = lambda v: float((v.double() - want).norm() / want.norm())          # noqa: E731
    assert error(y) <= 1.05 * error(F.linear(x, w))
    # two operands to 2^-23 each, the dropped product of the low limbs 2^-22, K additions of 2^-23 of the sum so far
    assert bool(((y.double() - want).abs() <= (2.0 ** -21 + K * 2.0 ** -23) * (x.abs().double() @ w.abs().double().T)).all())


def test_entries_of_every_size():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(5)
    M, N, K = 200, 700, 192
    x, w = (torch.randn(n, K, generator=g, device="cuda") for n in (M, N))
    x *= torch.exp2(-torch.rand(M, K, generator=g, device="cuda") * 60)
    x[7], x[8, 3] = x[7] * 2.0 ** -130, 1e-42                                  # subnormal entries
    w[torch.rand(N, K, generator=g, device="cuda") < 0.9] = 0.0                # few terms each: nothing large to hide behind
    want, terms = x.double() @ w.double().T, x.abs().double() @ w.abs().double().T
    y = ops.linear_f32(x, w)
    # as above, and the smallest fp32 number's rounding per term
    assert bool(((y.double() - want).abs() <= (2.0 ** -21 + K * 2.0 ** -23) * terms + K * 2.0 ** -149).all())


@pytest.mark.parametrize("entries", [1, 2])
@pytest.mark.parametrize("M,N,K", [(1, 1, 64), (45, 131, 256), (3000, 700, 192)])
def test_tiny_entries(M, N, K, entries):
    """Entries far below their row's largest, in both operands and at the same place of both, as whole results: the large
    entries meet zeros."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(K)
    x, w = torch.zeros(M, K, device="cuda"), torch.zeros(N, K, device="cuda")
    x[:, 0], w[:, 1] = 3e8, 5e9
    rand = lambda n: torch.rand(n, entries, generator=g, device="cuda") + 0.3           # noqa: E731
    at = torch.tensor([K - 1, 17][:entries], device="cuda")
    x[:, at], w[:, at] = rand(M), rand(N)
    x[M // 2, at], w[N // 2, at] = 0.0, 0.0
    x[M // 2, 40], w[N // 2, 40] = 1.25, 0.75
    w[N - 1] = torch.rand(K, generator=g, device="cuda") + 0.3                             # a row without a large entry
    b = torch.zeros(N, device="cuda")
    want = x.double() @ w.double().T
    y = ops.linear_f32(x, w, b)
    terms = x.abs().double() @ w.abs().double().T
    assert bool(((y.double() - want).abs() <= 2.0 ** -21 * terms).all())                   # at most three terms each
