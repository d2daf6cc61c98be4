"""The fused PiKVMoE forward against float64 arithmetic and against its own modules."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(experts=4, hidden=256, seed=0, **cfg):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pikv_b200 import config as C
    from pikv_b200.moe import PiKVMoE
    keep = dict(C.config)
    C.config.update(dict(num_experts=experts, hidden_size=hidden, num_layers=max(5, experts), vocab_size=301, cache_decrement=3, **cfg))
    try:
        torch.manual_seed(seed)
        m = PiKVMoE().eval().cuda()
    finally:
        C.config.clear()
        C.config.update(keep)
    g = torch.Generator(device="cuda").manual_seed(seed)
    with torch.no_grad():
        for n, p in m.named_parameters():
            if n.endswith("lora_B"):
                p.copy_(torch.randn(p.shape, generator=g, device="cuda") * 0.2)
        for c in m.kv_caches:
            c.values.copy_(torch.randn(c.values.shape, generator=g, device="cuda"))
            c.importance.copy_(torch.rand(c.importance.shape, generator=g, device="cuda"))
        m.cache_ptrs.copy_(torch.tensor([m.kv_caches[i].size - 1 - i for i in range(experts)]))
    m.router.load_balancing_router.temperature = 0.7
    return m


def _f64(m, x):
    """Weighted sum, logits, cache rows and auxiliary loss in float64."""
    d = lambda t: t.detach().double()                                              # noqa: E731
    lin = lambda l, v: v @ d(l.weight).T + d(l.bias)                               # noqa: E731
    lora = lambda l, v: v @ d(l.lora_A) @ d(l.lora_B) * l.scaling                  # noqa: E731
    x, r = x.double(), m.router
    sel = torch.softmax(lin(r.router_selector[2], torch.relu(lin(r.router_selector[0], x.mean(1)))), -1)
    gate = lambda g: torch.softmax(lin(g.router[2], torch.relu(lin(g.router[0], x))) / g.temperature, -1)   # noqa: E731
    a, b, pr = gate(r.load_balancing_router), gate(r.importance_router), r.importance_router.importance_predictor
    imp = torch.sigmoid(lin(pr[2], torch.relu(lin(pr[0], x))))
    b = b * imp
    w = sel[:, 0:1, None] * a + sel[:, 1:2, None] * b / b.sum(-1, keepdim=True)
    out, rows = torch.zeros_like(x), []
    for e, ex in enumerate(m.experts):
        c = m.kv_caches[e]
        xi = d(c.values) * d(c.importance)[:, None]
        p = c.compressor.compressor.compression_layers
        cv = xi + lin(p[1], lin(p[0], xi))
        y = torch.relu(lin(ex.dense, x) + lora(ex.lora, x)) + (cv + lora(c.value_lora, cv)).mean(0)
        rows.append((x.mean((0, 1)), y.mean((0, 1)), imp.mean()))
        out = out + y * w[..., e:e + 1]
    use = a.mean((0, 1))
    return lin(m.vocab_proj, out), rows, r.load_balancing_router.balance_weight * use.std() / use.mean(), w


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


# one token, part of a tile, whole tiles, one past them; two experts and the most; widths with one and many tiles
@pytest.mark.parametrize("B,S,E,H", [(1, 1, 4, 256), (3, 21, 4, 256), (1, 64, 2, 128), (5, 13, 16, 128), (2, 97, 3, 384), (8, 128, 4, 256),
                                     (1, 7, 2, 1024)])
def test_against_float64(B, S, E, H):
    m = _model(E, H)
    x = torch.randn(B, S, H, generator=torch.Generator(device="cuda").manual_seed(B * S), device="cuda")
    want, rows, loss, w = _f64(m, x)
    slots = m.cache_ptrs.tolist()
    with torch.no_grad():
        assert m._fused(x) is not None
        m.cache_ptrs.copy_(torch.tensor(slots)); m._host_ptrs = None
        for e, c in enumerate(m.kv_caches[:E]):                    # what the call above wrote into the ring
            c.values[slots[e]] = torch.randn(H, device="cuda")
        want, rows, loss, w = _f64(m, x)
        got, lb = m(x, return_loss=True)
    # fp32 sums of up to 1024 products, three layers deep
    assert _rel(got, want) < 2e-6
    for e in range(E):
        c = m.kv_caches[e]
        assert _rel(c.keys[slots[e]], rows[e][0]) < 2e-6 and _rel(c.values[slots[e]], rows[e][1]) < 2e-6
        assert abs(float(c.importance[slots[e]]) - float(rows[e][2])) < 1e-6
        assert int(m.cache_ptrs[e]) == (slots[e] + 1) % c.size == m._host_ptrs[e]
    assert abs(float(lb) - float(loss)) < 1e-5 * float(loss) + 1e-7
    assert _rel(m.router.last_gate.topk_w.sum(-1), torch.ones(B * S, device="cuda").double()) < 1e-6
    top = w.view(B * S, E).topk(2, -1).values
    assert torch.allclose(w.view(B * S, E).gather(1, m.router.last_gate.topk_idx.long()), top, atol=1e-6)


def test_same_as_the_modules_and_when_they_run(monkeypatch):
    """Both routes give the same state; hooks, a query, gradients, autocast, tangents, transforms and scheduled caches take the modules."""
    m, n = _model(), _model()
    x = torch.randn(2, 33, 256, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda")
    seen = []
    handle = n.experts[2].lora.register_forward_hook(lambda *a: seen.append(1))
    with torch.no_grad():
        for k in range(3):
            a, b = m(x + k), n(x + k)
            assert _rel(a, b.double()) < 2e-6
        assert len(seen) == 3
        for (name, p), (_, q) in zip(m.named_buffers(), n.named_buffers()):
            assert torch.allclose(p.float(), q.float(), rtol=1e-5, atol=1e-6), name
        for f in (lambda t: t.router.last_gate, lambda t: t.router.importance_router.last_gate, lambda t: t.router.load_balancing_router.last_gate):
            for p, q in zip(f(m).tensors()[:7], f(n).tensors()[:7]):
                assert (p is None) == (q is None) and (p is None or torch.allclose(p.float(), q.float(), rtol=1e-4, atol=1e-5))
        assert n._fused(x) is None
        handle.remove()
        assert n._fused(x) is not None
        with torch.autocast("cuda", torch.bfloat16):
            assert n._fused(x) is None
        assert n._fused(x[..., :128]) is None and n._fused(x.double()) is None
        assert n._fused(x.transpose(0, 1).contiguous().transpose(0, 1)) is not None
        n.kv_caches[1].use_scheduling = True
        assert n._fused(x) is None
        n.kv_caches[1].use_scheduling = False
        n.kv_caches[1].values = n.kv_caches[0].values               # shared storage is read behind its update by the modules
        assert n._fused(x) is None
        with torch.autograd.forward_ad.dual_level():
            assert m._fused(x) is None
        torch.func.vmap(lambda t: (seen.append(m._fused(t)), t)[1])(x[None])
        assert seen[-1] is None
    with torch.inference_mode():
        assert m._fused(x.clone()) is not None
    y = m(x)
    assert y.requires_grad
    assert math.isfinite(float(y.detach().sum()))
