"""The quantiser's sample counter in every form that an in-place addition takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counter", [dict(size=()), dict(size=(1,)), dict(size=(3,)), dict(size=(), dtype=torch.float64), dict(size=(), device="cpu")])
def test_sample_count(counter):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200.compression import QuantizedCompressor
    q = QuantizedCompressor(64, group_size=32).cuda()
    q.sample_count = torch.full(**{"fill_value": 5.0, "device": "cuda", **counter})
    k = torch.randn(1, 20, 64, device="cuda")
    q(k, k)
    assert bool((q.sample_count == 9.0).all())           # two groups of K and two of V
