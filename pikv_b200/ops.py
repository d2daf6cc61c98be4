"""Functional wrappers: torch CUDA tensors in, kernels launched through the C ABI.

Every function enqueues on the current torch CUDA stream and returns torch
tensors it allocated.  Inputs are borrowed and never modified unless the
docstring says so.  The operators of the hot path go through the native host
module (csrc/host/host.cpp), the rest through ctypes.  Nothing here computes on the CPU: a tensor that is not on
a CUDA device is an error.
"""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass
from typing import Optional

import torch

from . import _lib
from ._lib import PikvError, check, host, lib

PAGE_TOKENS = _lib.PAGE_TOKENS
HEAD_DIM = _lib.HEAD_DIM


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _p(t: Optional[torch.Tensor]):
    return None if t is None else C.c_void_p(t.data_ptr())


def _req(t: torch.Tensor, name: str, dtype=None) -> torch.Tensor:
    if not isinstance(t, torch.Tensor) or not t.is_cuda:
        raise PikvError(f"{name} must be a CUDA tensor (there is no CPU path)")
    if dtype is not None and t.dtype != dtype:
        raise PikvError(f"{name} must be {dtype}, got {t.dtype}")
    return t if t.is_contiguous() else t.contiguous()


def _written(t: torch.Tensor, name: str, dtype) -> torch.Tensor:
    """A tensor that is updated in place: a contiguous copy would take the update and be dropped."""
    if isinstance(t, torch.Tensor) and not t.is_contiguous():
        raise PikvError(f"{name} is updated in place and must be contiguous")
    return _req(t, name, dtype)


def _dtype_code(t: torch.Tensor, name: str) -> int:
    if t.dtype == torch.float32:
        return _lib.PIKV_F32
    if t.dtype == torch.bfloat16:
        return _lib.PIKV_BF16
    raise PikvError(f"{name}: dtype {t.dtype} not supported (float32 or bfloat16)")


_ws_cache: dict = {}


def _workspace(dev: torch.device, nbytes: int, tag: str) -> torch.Tensor:
    """Per-(device, stream, tag) scratch buffer, grown on demand and reused."""
    key = (dev.index, torch.cuda.current_stream().cuda_stream, tag)
    buf = _ws_cache.get(key)
    if buf is None or buf.numel() < nbytes:
        buf = torch.empty(max(nbytes, 1), dtype=torch.uint8, device=dev)
        _ws_cache[key] = buf
    return buf


# ------------------------------------------------------------------ gate
@dataclass
class GateResult:
    probs: Optional[torch.Tensor]      # [T,E] fp32
    topk_idx: torch.Tensor             # [T,k] int32
    topk_w: torch.Tensor               # [T,k] fp32
    slot: torch.Tensor                 # [T,k] int32, -1 = dropped at capacity
    counts_k: torch.Tensor             # [k,E] int32
    prob_sum: torch.Tensor             # [E] fp32
    new_len: torch.Tensor              # [E] int32
    workspace: Optional[torch.Tensor] = None   # gate scratch owned by this result (route_append)

    @property
    def counts(self) -> torch.Tensor:
        return self.counts_k.sum(0)

    def tensors(self):
        return (self.probs, self.topk_idx, self.topk_w, self.slot, self.counts_k, self.prob_sum, self.new_len, self.workspace)


def gate_fused(act: Optional[torch.Tensor] = None, w2: Optional[torch.Tensor] = None,
               b2: Optional[torch.Tensor] = None, *, logits: Optional[torch.Tensor] = None, top_k: int = 2,
               expert_mask: Optional[torch.Tensor] = None, mask_mode: int = _lib.MASK_SINGLE,
               correction: Optional[torch.Tensor] = None, temperature: float = 1.0, renorm_eps: float = 0.0,
               capacity: int = 0, slot_base: Optional[torch.Tensor] = None, want_probs: bool = True,
               out: Optional[GateResult] = None, phase: int = 0) -> GateResult:
    """Fused gate tail; see pikv_gate_fused in include/pikv_b200.h.

    Give either (act [T,H], w2 [E,H], b2 [E]) or logits [T,E] fp32.  phase 1 (scoring kernel only) and
    phase 2 (slot finalisation only, same arguments, ordered after phase 1 by the caller) keep their state
    in out.workspace, which is allocated on first use and must not be shared between batches in flight.
    """
    res = host().gate(act, w2, b2, logits, top_k, expert_mask, mask_mode, correction, temperature, renorm_eps, int(capacity),
                      slot_base, want_probs, None if out is None else out.tensors(), int(phase))
    if out is None:
        return GateResult(*res)
    out.workspace = res[7]
    return out


def gate_mlp_fused(x: torch.Tensor, w1: torch.Tensor, b1: Optional[torch.Tensor], w2: torch.Tensor,
                   b2: Optional[torch.Tensor], *, top_k: int = 2, expert_mask: Optional[torch.Tensor] = None,
                   mask_mode: int = _lib.MASK_SINGLE, correction: Optional[torch.Tensor] = None, temperature: float = 1.0,
                   renorm_eps: float = 0.0, capacity: int = 0, slot_base: Optional[torch.Tensor] = None,
                   want_probs: bool = True, out: Optional[GateResult] = None) -> GateResult:
    """The whole gate net on tensor cores: relu(x @ w1.T + b1) @ w2.T + b2, then the tail of gate_fused (same
    keyword arguments and result); bf16 x [T,K], w1 [H,K], w2 [E,H].  See pikv_gate_mlp_fused."""
    res = host().gate_mlp(x, w1, b1, w2, b2, top_k, expert_mask, mask_mode, correction, temperature, renorm_eps, int(capacity),
                          slot_base, want_probs, None if out is None else out.tensors(), 0, 0, 0, 0.0)
    return GateResult(*res) if out is None else out


BALANCE = {None: 0, "entropy": 1, "cv": 2, "l2": 3}


def gate_mlp_dense(x: torch.Tensor, w1: torch.Tensor, b1: Optional[torch.Tensor], w2: torch.Tensor, b2: Optional[torch.Tensor],
                   rows: int, position_mode: int, balance: Optional[str] = None, coefficient: float = 0.0, *, top_k: int = 2,
                   expert_mask: Optional[torch.Tensor] = None, mask_mode: int = _lib.MASK_SINGLE, renorm_eps: float = 0.0,
                   capacity: int = 0):
    """gate_mlp_fused on x [..., K] and dispatch_loss (`rows` = capacity dimension of the dense tensors) in one call: the
    dense tensors are cleared beside the tensor-core work.  Returns (gate result, (dispatch, combine, aux))."""
    res = host().gate_mlp(x, w1, b1, w2, b2, top_k, expert_mask, mask_mode, None, 1.0, renorm_eps, int(capacity), None, True, None,
                          rows, position_mode, BALANCE[balance], coefficient)
    return GateResult(*res[:8]), res[8:]


def dispatch_scatter(g: GateResult, num_experts: int, capacity: int, position_mode: int = 0):
    """Dense [T,E,capacity] fp32 dispatch and combine tensors from a gate result."""
    return dispatch_loss(g, num_experts, capacity, position_mode)[:2]


def dispatch_loss(g: GateResult, num_experts: int, capacity: int, position_mode: int = 0, balance: Optional[str] = None,
                  coefficient: float = 0.0):
    """dispatch_scatter and the router's auxiliary loss (0-dim): the base term of core/single/pikv_routing.py:155-159
    plus `coefficient` times the balance term of :185-222.  The loss is None for a result without probability sums."""
    return host().dispatch_loss(g.topk_idx, g.topk_w, g.slot, g.counts_k, g.prob_sum, num_experts, capacity, position_mode,
                                BALANCE[balance], coefficient)


# ------------------------------------------------------------------ block-wide fake quantisation
def quant_block(x: torch.Tensor, group_size: int, qmin: int, qmax: int, symmetric: bool,
                params_in: Optional[torch.Tensor] = None, want_codes: bool = False, want_err: bool = True):
    """Returns (dq [N,H] fp32, q or None, params [G,2] fp32 (scale, zero point), sq_err [G] or None)."""
    x = _req(x, "x")
    N, H = x.shape
    G = (H + group_size - 1) // group_size
    dev = x.device
    dq = torch.empty(N, H, dtype=torch.float32, device=dev)
    q = torch.empty(N, H, dtype=torch.float32, device=dev) if want_codes else None
    params = torch.empty(G, 2, dtype=torch.float32, device=dev)
    err = torch.empty(G, dtype=torch.float32, device=dev) if want_err else None
    if params_in is not None:
        params_in = _req(params_in, "params_in", torch.float32)
    ws = _workspace(dev, lib().pikv_quant_block_workspace_bytes(N, H, group_size), "qb")
    check(lib().pikv_quant_block(_p(x), _dtype_code(x, "x"), N, H, group_size, qmin, qmax, int(bool(symmetric)),
                                 _p(params_in), _p(params), _p(dq), _p(q), _p(err), _p(ws), ws.numel(), _stream()),
          "pikv_quant_block")
    return dq, q, params, err


def quant_block_pair(k: torch.Tensor, v: torch.Tensor, group_size: int, qmin: int, qmax: int, symmetric: bool,
                     params_in: Optional[torch.Tensor] = None, sample_count: Optional[torch.Tensor] = None,
                     count_add: float = 0.0):
    """quant_block on K and V [..., H] of one forward, both tensors in each launch when they agree in shape and dtype.
    Returns (dk, dv in the input's dtype, mean squared error of V's last group as a 0-dim tensor); sample_count grows by
    count_add."""
    if sample_count is not None and (sample_count.dtype != torch.float32 or sample_count.device != k.device or sample_count.numel() != 1):
        sample_count += count_add                     # not one word that the kernel can add to
        sample_count = None
    if k.shape != v.shape or k.dtype != v.dtype:
        kf, vf = k.reshape(-1, k.shape[-1]), v.reshape(-1, v.shape[-1])
        dk, _, _, _ = quant_block(kf, group_size, qmin, qmax, symmetric, params_in=params_in, want_err=False)
        dv, _, _, err = quant_block(vf, group_size, qmin, qmax, symmetric, params_in=params_in)
        if sample_count is not None:
            sample_count += count_add
        last = vf.shape[1] - (err.numel() - 1) * group_size
        return dk.to(k.dtype).view(k.shape), dv.to(v.dtype).view(v.shape), err[-1] / float(vf.shape[0] * last)
    return host().quant_pair(k, v, group_size, qmin, qmax, symmetric, params_in, sample_count, count_add)


# ------------------------------------------------------------------ fp32 linear layer
def linear_f32(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """x [..., K] @ w [N, K].T + bias in fp32 on the tensor cores (two f16 limbs per operand); K a multiple of 64 up to 256."""
    return host().linear_f32(x, w, bias)


# ------------------------------------------------------------------ H2O
def h2o_accumulate(acc: torch.Tensor, ts: torch.Tensor, idx: Optional[torch.Tensor], w: torch.Tensor, now: float,
                   decay: float = 1.0, status: Optional[torch.Tensor] = None) -> None:
    """In place: acc[idx] += w ; ts[idx] = now (acc *= decay first when decay != 1)."""
    acc = _written(acc, "acc", torch.float32)
    ts = _written(ts, "ts", torch.float32)
    w = _req(w, "w", torch.float32)
    if idx is not None:
        idx = _req(idx, "idx", torch.int32)
    check(lib().pikv_h2o_accumulate(_p(acc), _p(ts), acc.numel(), _p(idx), _p(w), w.numel(), float(now), float(decay),
                                    _p(status), _stream()), "pikv_h2o_accumulate")


def h2o_select(acc: torch.Tensor, ts: torch.Tensor, num_heavy: int, num_recent: int,
               seg_len: Optional[torch.Tensor] = None, n: Optional[int] = None, want_idx: bool = True,
               as_bool: bool = True):
    """acc, ts: [segments, stride] fp32.  Returns (evict_mask bool [segments,stride], keep_idx int32
    [segments, min(stride, heavy+recent)] ascending (unused tail undefined), kept_count int32 [segments]).
    as_bool=False returns the mask as uint8."""
    return host().select(acc, ts, num_heavy, num_recent, seg_len, -1 if n is None else n, want_idx, as_bool)


def h2o_accumulate_attn(scores: torch.Tensor, lse: torch.Tensor, seq_len: Optional[torch.Tensor], n_kv: int,
                        acc: torch.Tensor) -> None:
    """In place: acc[b*n_kv+h, pos] += sum over the group's query heads of exp(scores - lse)."""
    scores = _req(scores, "scores", torch.float32)
    lse = _req(lse, "lse", torch.float32)
    acc = _written(acc, "acc", torch.float32)
    B, n_q, stride = scores.shape
    check(lib().pikv_h2o_accumulate_attn(_p(scores), stride, _p(lse), _p(seq_len), B, n_q, n_kv, _p(acc),
                                         acc.shape[-1], _stream()), "pikv_h2o_accumulate_attn")


# ------------------------------------------------------------------ low-rank projection
def lowrank_project(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None, relu: bool = True,
                    residual: Optional[torch.Tensor] = None, out_dtype: torch.dtype = torch.bfloat16) -> torch.Tensor:
    """y[..., N] = act(x[..., K] @ w[N,K]^T + bias) (+ residual) on tcgen05 tensor cores; x, w bf16."""
    if w.dtype != torch.bfloat16:
        raise PikvError(f"w must be {torch.bfloat16}, got {w.dtype}")
    return host().lowrank(x, w, bias, relu, residual, out_dtype != torch.bfloat16)


def lowrank_pair(xs, w1s, b1s, w2s, b2s):
    """relu(x @ w1.T + b1) @ w2.T + b2 for the two (x, w1, b1, w2, b2) of K and V in one launch; bf16 x.  See
    pikv_lowrank_pair for the shapes it takes."""
    return host().lowrank_pair(*xs, *w1s, *b1s, *w2s, *b2s)


# ------------------------------------------------------------------ all-to-all records
def a2a_record_bytes(n_kv: int) -> int:
    return int(lib().pikv_a2a_record_bytes(n_kv))


def a2a_pack(k: torch.Tensor, v: torch.Tensor, n_kv: int, dst_seq: torch.Tensor, slot: torch.Tensor,
             n_records: int, send_pos: Optional[torch.Tensor] = None, seq_prefix: Optional[torch.Tensor] = None,
             out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Quantise (int8 symmetric, per token and head) and pack routed rows into records.  The record
    index of (token, j) is send_pos[t,j], or seq_prefix[dst_seq[t,j]] + slot[t,j] when send_pos is None."""
    k = _req(k, "k")
    v = _req(v, "v", k.dtype)
    T = k.shape[0]
    top_k = dst_seq.shape[1]
    nbytes = max(n_records, 1) * a2a_record_bytes(n_kv)
    buf = out if out is not None else torch.empty(nbytes, dtype=torch.uint8, device=k.device)
    if buf.numel() < nbytes:
        raise PikvError("a2a_pack: output buffer too small")
    if send_pos is not None:
        send_pos = _req(send_pos, "send_pos", torch.int32)
    if seq_prefix is not None:
        seq_prefix = _req(seq_prefix, "seq_prefix", torch.int32)
    check(lib().pikv_a2a_pack(_p(k), _p(v), _dtype_code(k, "k"), T, n_kv, top_k, _p(_req(dst_seq, "dst_seq", torch.int32)),
                              _p(_req(slot, "slot", torch.int32)), _p(seq_prefix), _p(send_pos), _p(buf), _stream()),
          "pikv_a2a_pack")
    return buf
