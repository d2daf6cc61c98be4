"""Which forwards of PiKVMoE are offered to the fused kernels."""
import types

import torch
from torch.overrides import TorchFunctionMode

from pikv_b200 import moe


class Watch(TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def test_function_modes_run_the_modules(monkeypatch):
    m = moe.PiKVMoE().eval()
    offered = []
    monkeypatch.setattr(moe, "host", lambda: types.SimpleNamespace(moe=lambda *a: offered.append(1)))
    x = torch.zeros(1, 2, moe.config["hidden_size"])
    with torch.no_grad():
        with Watch():
            assert m._fused(x) is None and not offered
        with torch.device("cpu"), Watch():
            assert m._fused(x) is None and not offered
        with torch.device("cpu"):                      # a default device only concerns new tensors
            m._fused(x)
        assert len(offered) == 1
        m._fused(x)
        assert len(offered) == 2
