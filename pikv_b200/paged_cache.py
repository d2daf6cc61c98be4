"""Paged, quantised KV store in HBM and the kernels that write and read it.

A *sequence* owns one row of the page table: an expert's cache (routed append),
a decode stream, or an (expert, stream) pair on an expert-sharded GPU.  Pages
hold 16 tokens.  Pools (indexed by physical page id):

    k_codes, v_codes  uint8 [pages, n_kv, 16, 128*bits/8]   (chunk-swizzled rows)
    k_scale, v_scale  bf16  [pages, n_kv, 16]
    k_zp, v_zp        fp32  [pages, n_kv, 16]                (asymmetric only)

The row placement follows CacheSchedulingManager.update_cache
(core/single/cache_scheduling.py:430-436: contiguous rows, truncation at
capacity); the arithmetic of the stored codes is QuantizedCompressor.
_quantize_tensor (core/single/module/pikv_compression.py:945-1012) per
(token, head) slice of 128 channels.
"""
from __future__ import annotations

from typing import Optional

import torch

from . import _lib, ops
from ._lib import PikvError, check, host, lib
from .ops import _p, _req, _stream, PAGE_TOKENS, HEAD_DIM


class PagedKVCache(torch.nn.Module):
    """Page pools + page table + per-sequence lengths, all registered buffers
    (so state_dict() carries the cache)."""

    def __init__(self, num_seqs: int, capacity: int, n_kv: int, bits: int = 8, symmetric: bool = True,
                 device="cuda", num_pages: Optional[int] = None, identity_table: bool = True):
        super().__init__()
        if bits not in (4, 8):
            raise ValueError("bits must be 4 or 8")
        self.num_seqs, self.n_kv, self.bits, self.symmetric = num_seqs, n_kv, bits, bool(symmetric)
        self.max_pages = (capacity + PAGE_TOKENS - 1) // PAGE_TOKENS
        self.capacity = capacity
        self.num_pages = num_pages if num_pages is not None else num_seqs * self.max_pages
        row = HEAD_DIM * bits // 8
        dev = torch.device(device)
        z = lambda *s, dtype: torch.zeros(*s, dtype=dtype, device=dev)
        self.register_buffer("k_codes", z(self.num_pages, n_kv, PAGE_TOKENS, row, dtype=torch.uint8))
        self.register_buffer("v_codes", z(self.num_pages, n_kv, PAGE_TOKENS, row, dtype=torch.uint8))
        self.register_buffer("k_scale", z(self.num_pages, n_kv, PAGE_TOKENS, dtype=torch.bfloat16))
        self.register_buffer("v_scale", z(self.num_pages, n_kv, PAGE_TOKENS, dtype=torch.bfloat16))
        if not self.symmetric:
            self.register_buffer("k_zp", z(self.num_pages, n_kv, PAGE_TOKENS, dtype=torch.float32))
            self.register_buffer("v_zp", z(self.num_pages, n_kv, PAGE_TOKENS, dtype=torch.float32))
        else:
            self.k_zp = self.v_zp = None
        if identity_table:
            if self.num_pages < num_seqs * self.max_pages:
                raise ValueError("identity page table needs num_seqs * max_pages pages")
            pt = torch.arange(num_seqs * self.max_pages, dtype=torch.int32, device=dev).view(num_seqs, self.max_pages)
        else:
            pt = torch.full((num_seqs, self.max_pages), -1, dtype=torch.int32, device=dev)
        self.register_buffer("page_table", pt)
        self.register_buffer("length", z(num_seqs, dtype=torch.int32))
        self.register_buffer("status", z(1, dtype=torch.int32))

    # -- serialisation ---------------------------------------------------------------
    # The reference's checkpoint keeps one mean vector per cache (core/single/pikv_moe.py:456-505): the rows are
    # lost.  Here the cache itself is the state: pages, scales, zero points, page table and lengths are registered
    # buffers, so state_dict() / load_state_dict() move it, and these two calls add the geometry a loader needs
    # to rebuild the object, plus any score buffers of an eviction policy the caller passes along.
    def save_checkpoint(self, path, scores: Optional[dict] = None) -> None:
        torch.save({"format": "pikv_b200.paged_cache.v1",
                    "geometry": {"num_seqs": self.num_seqs, "capacity": self.capacity, "n_kv": self.n_kv, "bits": self.bits,
                                 "symmetric": self.symmetric, "num_pages": self.num_pages},
                    "state_dict": self.state_dict(),
                    "scores": {k: v.detach().clone() for k, v in (scores or {}).items()}}, path)

    @classmethod
    def load_checkpoint(cls, path, device="cuda"):
        """Returns (cache, scores): the cache rebuilt on `device` with every page, scale and length of the saved one."""
        blob = torch.load(path, map_location=torch.device(device), weights_only=False)
        if blob.get("format") != "pikv_b200.paged_cache.v1":
            raise PikvError(f"{path}: not a paged-cache checkpoint")
        g = blob["geometry"]
        cache = cls(g["num_seqs"], g["capacity"], g["n_kv"], bits=g["bits"], symmetric=g["symmetric"], device=device,
                    num_pages=g["num_pages"], identity_table=False)
        cache.load_state_dict(blob["state_dict"])
        return cache, blob.get("scores", {})

    # -- writes --------------------------------------------------------------------
    def append(self, k: torch.Tensor, v: torch.Tensor, dst_seq: torch.Tensor, slot: torch.Tensor) -> None:
        """Quantise and store k, v [T, n_kv*128] at (dst_seq[t,j], slot[t,j]); slot < 0 is skipped.
        Does not touch `length` (the gate's new_len, or the caller, owns it)."""
        host().append(self._buffers, self.num_seqs, self.n_kv, self.bits, self.symmetric, self.max_pages, self.num_pages,
                      k, v, dst_seq, slot)

    def append_rope(self, k: torch.Tensor, v: torch.Tensor, dst_seq: torch.Tensor, slot: torch.Tensor,
                    cos: torch.Tensor, sin: torch.Tensor, positions: Optional[torch.Tensor] = None) -> None:
        """append() with the rotary position embedding of core/single/pikv_attention.py:329-390 applied to K in
        registers before it is quantised (pikv_kv_append_rope).  cos, sin: [max_pos, 64] fp32 tables (the
        reference's cos_cached / sin_cached); positions [T] int32 (default: the token index).  bf16 K/V, int8
        symmetric cache."""
        host().append(self._buffers, self.num_seqs, self.n_kv, self.bits, self.symmetric, self.max_pages, self.num_pages,
                      k, v, dst_seq, slot, cos, sin, positions)

    def route_append(self, act: torch.Tensor, w2: torch.Tensor, b2: Optional[torch.Tensor], k: torch.Tensor,
                     v: torch.Tensor, top_k: int = 2, capacity: Optional[int] = None,
                     out: Optional["ops.GateResult"] = None, slot_base: Optional[torch.Tensor] = None,
                     want_probs: bool = True):
        """Gate the tokens and append their quantised K/V rows in one call (pikv_route_append): the
        same results as ops.gate_fused followed by append(), with the slot finalisation folded into the
        append kernel.  Sequences are the experts.  Returns the gate result."""
        res = host().route_append(self._buffers, self.num_seqs, self.n_kv, self.bits, self.symmetric, self.max_pages,
                                  self.num_pages, act, w2, b2, k, v, top_k, None, 0, None, 1.0, 0.0,
                                  self.capacity if capacity is None else int(capacity), slot_base, want_probs,
                                  None if out is None else out.tensors())
        if out is None:
            return ops.GateResult(*res)
        out.workspace = res[7]
        return out

    # -- reads ---------------------------------------------------------------------
    def gather(self, seq: torch.Tensor, pos: torch.Tensor, which: str = "k", codes: bool = False):
        """Dequantised rows [n, n_kv*128] fp32 (and int8 codes when codes=True) in logical order."""
        seq = _req(seq, "seq", torch.int32)
        pos = _req(pos, "pos", torch.int32)
        n = seq.numel()
        dev = seq.device
        out = torch.empty(n, self.n_kv * HEAD_DIM, dtype=torch.float32, device=dev)
        cod = torch.empty(n, self.n_kv * HEAD_DIM, dtype=torch.int8, device=dev) if codes else None
        pool, sc, zp = (self.k_codes, self.k_scale, self.k_zp) if which == "k" else (self.v_codes, self.v_scale, self.v_zp)
        check(lib().pikv_cache_gather(_p(seq), _p(pos), n, _p(self.page_table), self.num_seqs, self.max_pages,
                                      self.num_pages, self.n_kv, self.bits, _p(pool), _p(sc), _p(zp), _p(out), _p(cod),
                                      _p(self.status), _stream()), "pikv_cache_gather")
        return (out, cod) if codes else out

    def decode_attention(self, q: torch.Tensor, seq_ids: Optional[torch.Tensor] = None,
                         seq_len: Optional[torch.Tensor] = None, splits: int = 0, want_lse: bool = False,
                         scores: Optional[torch.Tensor] = None, max_ctx: Optional[int] = None):
        """softmax(q K^T / sqrt(128)) V over each stream's cached context; q [B, n_q, 128] bf16.  max_ctx: the
        longest context in the batch if the caller knows it.  splits and max_ctx are accepted for older callers: the
        kernel balances the pages over the GPU by itself.  Reads int8 symmetric (pikv_decode_attn_q8) and 4-bit asymmetric (pikv_decode_attn_q4) caches."""
        return host().decode(self._buffers, self.num_seqs, self.n_kv, self.bits, self.symmetric, self.max_pages, self.num_pages,
                             q, seq_ids, seq_len, want_lse, scores)

    def h2o_workspace(self, B: int, n_q: int, max_ctx: Optional[int] = None):
        """Scratch for decode_attention_h2o: f16 probabilities [B, n_q, ctx] and the step maxima [B, n_q, ctx/16]."""
        ctx = max_ctx or self.max_pages * PAGE_TOKENS
        dev = self.k_codes.device
        return (torch.empty(B, n_q, ctx, dtype=torch.float16, device=dev),
                torch.empty(B, n_q, (ctx + PAGE_TOKENS - 1) // PAGE_TOKENS, dtype=torch.float32, device=dev))

    def decode_attention_h2o(self, q: torch.Tensor, acc: torch.Tensor, workspace=None, seq_ids: Optional[torch.Tensor] = None,
                             seq_len: Optional[torch.Tensor] = None):
        """decode_attention plus the H2O update acc[b * n_kv + h, pos] += sum over the group's query heads of the
        attention probability (core/single/pikv_moe.py:241-245 column sums fed to
        core/single/cache_scheduling.py:69-73): the decode kernel leaves f16 probabilities relative to their softmax
        step, pikv_h2o_accumulate_probs normalises them with the final log-sum-exp.  int8 symmetric caches."""
        probs, step_max = self.h2o_workspace(q.shape[0], q.shape[1]) if workspace is None else workspace
        return host().decode(self._buffers, self.num_seqs, self.n_kv, self.bits, self.symmetric, self.max_pages, self.num_pages,
                             q, seq_ids, seq_len, acc, probs, step_max)

    # -- eviction ------------------------------------------------------------------
    def compact_into(self, dst: "PagedKVCache", keep_idx: torch.Tensor, kept_count: torch.Tensor, per_head: bool,
                     src_acc=None, src_ts=None, dst_acc=None, dst_ts=None) -> None:
        """Copy the kept rows (ascending original order) to positions 0.. of `dst`'s sequences."""
        host().compact(self._buffers, self.num_seqs, self.n_kv, self.bits, self.symmetric, self.max_pages, self.num_pages,
                       dst._buffers, dst.num_seqs, dst.n_kv, dst.bits, dst.symmetric, dst.max_pages, dst.num_pages,
                       keep_idx, kept_count, per_head, src_acc, src_ts, dst_acc, dst_ts)

    def unpack_records(self, recv_buf: torch.Tensor, n_records: int, seq_offset: int = 0,
                       seg_start: Optional[torch.Tensor] = None, seg_base: Optional[torch.Tensor] = None) -> None:
        """Store records received from the token all-to-all (see ops.a2a_pack) into the pages.  Record
        sequence ids are global: seq_offset is subtracted.  seg_start [S+1] / seg_base [S, num_seqs] add a
        per-(source segment, sequence) base to the record's slot; positions >= capacity are dropped."""
        if self.bits != 8 or not self.symmetric:
            raise PikvError("records carry int8 symmetric codes")
        recv_buf = _req(recv_buf, "recv_buf", torch.uint8)
        n_seg = 0
        if seg_start is not None:
            seg_start = _req(seg_start, "seg_start", torch.int32)
            seg_base = _req(seg_base, "seg_base", torch.int32)
            n_seg = seg_start.numel() - 1
        check(lib().pikv_a2a_unpack(_p(recv_buf), n_records, self.n_kv, _p(self.page_table), self.num_seqs,
                                    self.max_pages, self.num_pages, seq_offset, self.capacity, _p(seg_start), _p(seg_base),
                                    n_seg, _p(self.k_codes), _p(self.v_codes), _p(self.k_scale), _p(self.v_scale),
                                    _p(self.status), _stream()), "pikv_a2a_unpack")

    def check_status(self) -> None:
        """Raise if any kernel flagged a bad index, page or a wait that ran out (synchronises)."""
        s = int(self.status.item())
        if s:
            raise PikvError(f"cache status word = {s:#x} (see PIKV_ST_* in include/pikv_b200.h)")
