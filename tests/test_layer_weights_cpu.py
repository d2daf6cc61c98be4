"""Layers whose weight is computed (weight norm, parametrisations) and named Sequentials are taken like plain ones."""
from collections import OrderedDict

import pytest
import torch
import torch.nn as nn
from torch.nn.utils import parametrizations

from pikv_b200 import compression, ops
from pikv_b200.routing import TopKBalancedRouter


def test_gate_net_weights_of_reparametrised_layers():
    r = TopKBalancedRouter(32, 4, top_k=2)
    plain = [t.detach().clone() for t in r._net_weights(r.router)]
    parametrizations.weight_norm(r.router[0])
    assert all(torch.allclose(a.float(), b.float(), atol=1e-2) for a, b in zip(r._net_weights(r.router), plain))
    named = nn.Sequential(OrderedDict(first=r.router[0], act=nn.ReLU(), last=r.router[2]))
    assert all(torch.allclose(a.float(), b.float(), atol=1e-2) for a, b in zip(r._net_weights(named), plain))
    assert r._fused_net(named, torch.zeros(1, 32, dtype=torch.bfloat16))


class _Shaped:
    """What _round_trip asks of a K/V tensor on the GPU."""

    def __init__(self, rows, width):
        self.shape, self.dtype, self.is_cuda = (rows, width), torch.bfloat16, True

    def numel(self):
        return self.shape[0] * self.shape[1]


@pytest.mark.parametrize("own", [False, True])
def test_low_rank_round_trip_of_reparametrised_layers(monkeypatch, own):
    class Own(compression.SVDCompressor):
        def project(self, x, which="key"):
            return which

        def reconstruct(self, latent, which="key"):
            return "own " + latent

    c = (Own if own else compression.SVDCompressor)(64, rank=16)
    parametrizations.weight_norm(c.key_projector)
    monkeypatch.setattr(ops, "lowrank_pair", lambda x, w1, b1, w2, b2: [tuple(t.shape) for t in (*w1, *b1, *w2, *b2)])
    x = _Shaped(c.PAIR_ROWS, 64)
    got = c._round_trip(x, x)
    if own:
        assert got == ("own key", "own value")
    else:
        assert got == [(16, 64)] * 2 + [(16,)] * 2 + [(64, 16)] * 2 + [(64,)] * 2
