"""Shapes and layers of the low-rank compressors that are not the plain [rows, width] batch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda")


def test_one_dimensional_vectors(dev):
    from pikv_b200.compression import PyramidCompressor, SVDCompressor
    torch.manual_seed(0)
    x = torch.randn(3, 256, device=dev).bfloat16()
    with torch.no_grad():
        c = SVDCompressor(256, rank=32).to(dev).bfloat16()
        latent = c.project(x)
        assert torch.equal(c.project(x[1]), latent[1]) and torch.equal(c.reconstruct(latent[1]), c.reconstruct(latent)[1])
        p = PyramidCompressor(256).to(dev).bfloat16()
        assert torch.equal(p._chain(x[2], 1), p._chain(x, 1)[2])


@pytest.mark.parametrize("layers", ["fp32 projector", "fp32 bias", "no bias", "other rank"])
def test_round_trip_of_unlike_layers(dev, layers):
    """K and V through one kernel (4096 rows) and through the separate products (a few rows) take the same layers."""
    from pikv_b200.compression import SVDCompressor
    torch.manual_seed(1)
    c = SVDCompressor(256, rank=32).to(dev).bfloat16()
    for p in (c.key_projector, c.value_projector, c.key_reconstructor, c.value_reconstructor):
        torch.nn.init.normal_(p.bias)
    if layers == "fp32 projector":
        c.key_projector.float()
    elif layers == "fp32 bias":
        c.value_reconstructor.bias = torch.nn.Parameter(c.value_reconstructor.bias.float())
    elif layers == "no bias":
        c.key_projector.float().bias = None
    else:
        c.value_projector, c.value_reconstructor = (torch.nn.Linear(*s).to(dev).bfloat16() for s in ((256, 16), (16, 256)))
    k, v = (torch.randn(c.PAIR_ROWS, 256, device=dev).bfloat16() for _ in range(2))
    with torch.no_grad():
        rk, rv = c(k, v)
        few = c(k[:64], v[:64])
    # the same bf16 latent up to its rounding (2^-8 of a term), bf16 results
    for got, want in zip((rk[:64], rv[:64]), few):
        assert float((got.float() - want.float()).norm() / want.float().norm()) < 2 ** -8
