"""Where PiKVMoE's fused forward is taken, and its results beyond a serving batch."""
import copy
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(experts, hidden):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import config as C
    from pikv_b200.moe import PiKVMoE
    keep = dict(C.config)
    C.config.update(dict(num_experts=experts, hidden_size=hidden, num_layers=max(5, experts), vocab_size=301, cache_decrement=3))
    try:
        torch.manual_seed(0)
        with torch.device("cuda"):
            return PiKVMoE().eval()
    finally:
        C.config.clear()
        C.config.update(keep)


@pytest.fixture
def taken(monkeypatch):
    """Whether each forward offered to the host module was fused."""
    from pikv_b200 import moe
    own, log = moe.host(), []

    def offered(*a):
        r = own.moe(*a)
        log.append(r is not None)
        return r

    monkeypatch.setattr(moe, "host", lambda: types.SimpleNamespace(moe=offered))
    return log


# both sides of the lines: tokens x width^2 above a width of 512, sequence x width^2 above 256
@pytest.mark.parametrize("hidden,batch,seq,fused", [(1024, 1, 8192, True), (1024, 1, 8193, False), (1024, 8, 1025, False), (640, 3, 6990, True),
                                                    (640, 3, 6991, False), (512, 1, 45056, True), (512, 1, 45057, False), (512, 2, 24000, True),
                                                    (256, 1, 70001, True)])
def test_route_and_results(taken, hidden, batch, seq, fused):
    m = _model(2, hidden)
    other = copy.deepcopy(m)
    x = torch.randn(batch, seq, hidden, device="cuda")
    with torch.no_grad():
        got = m(x)
        assert taken == [fused]
        if fused:
            other._fused = lambda x: None
            want = other(x)
            # fp32 sums of up to 1024 terms in another order, and the tie-free softmax weights of both
            assert float((got - want).norm() / want.norm()) < 1e-5
            for a, b in zip(m.kv_caches, other.kv_caches):
                for n in ("keys", "values", "importance"):
                    assert float((getattr(a, n) - getattr(b, n)).norm()) <= 1e-4 * float(getattr(b, n).norm()) + 1e-6


def test_modules_run_where_the_workspace_does_not_fit(taken):
    m = _model(16, 128)
    other = copy.deepcopy(m)
    x = torch.randn(8, 16384, 128, device="cuda")
    needs = 16 * x.numel() * 4                            # all experts' outputs
    other._fused = lambda x: None
    with torch.no_grad():
        torch.cuda.empty_cache()
        torch.cuda.reset_peak_memory_stats()
        want = other(x).cpu()
        peak = torch.cuda.max_memory_reserved()
        torch.cuda.empty_cache()
        if peak + (64 << 20) >= torch.cuda.memory_reserved() + needs:
            pytest.skip("the modules need as much")
        torch.cuda.set_per_process_memory_fraction((peak + (64 << 20)) / torch.cuda.get_device_properties(0).total_memory)
        try:
            got = m(x).cpu()
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
    assert taken == [False]
    assert float((got - want).norm() / want.norm()) < 1e-5
