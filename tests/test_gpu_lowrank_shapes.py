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
