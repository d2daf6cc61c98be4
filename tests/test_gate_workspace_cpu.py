"""Gate scratch is sized for the kernels that run: a step that binds its own only runs the gate tail."""
import ctypes
import types

import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from pikv_b200 import _lib, distributed, ops


def test_prepared_step_has_scratch_for_the_tail(monkeypatch):
    monkeypatch.setattr(ops, "_p", lambda t: None)
    T, H, E, k, n_kv = 131072, 64, 64, 2, 1
    cache = types.SimpleNamespace(max_pages=4, num_pages=4 * E, status=None)
    me = types.SimpleNamespace(_C=ctypes, _lib=_lib, num_experts=E, device="cuda", n_kv=n_kv, global_table=None, cache=cache, world=1, rank=0, per=E,
                               capacity=64, slot_base=None, mirror_k=None, mirror_v=None, seq=None, len_all=None, wait_limit_us=0,
                               _peer={n: [None] for n in ("k_codes", "v_codes", "k_scale", "v_scale")}, _peer_gather=[None], _peer_flags=[None])
    with FakeTensorMode():
        bf = lambda *s: torch.empty(*s, dtype=torch.bfloat16, device="cuda")                    # noqa: E731
        out = ops.GateResult(*[None] * 7)
        distributed.PeerShardedKVCache.prepare(me, bf(T, H), bf(E, H), None, bf(T, 128), bf(T, 128), top_k=k, out=out)
    assert out.workspace.numel() == _lib.lib().pikv_gate_tail_workspace_bytes(T, E, k) < 1 << 22
