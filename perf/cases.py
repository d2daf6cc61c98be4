"""What a user of this framework has it do, as cases that can be timed.

Each case is one call (or the two calls that belong together) of a serving program on one GPU: routing a batch of
tokens and appending their quantised K/V, one decode step over a quantised cache, an H2O eviction, a router of the
operator surface, the low-rank and the quantising compressor, and the whole PiKVMoE forward.  Sizes are those of
the test suite and of bench.py, with ragged ones between them.
"""
from __future__ import annotations

import math

import torch

import pikv_b200
from pikv_b200 import ops
from pikv_b200.compression import QuantizedCompressor, SVDCompressor
from pikv_b200.config import config
from pikv_b200.moe import PiKVMoE
from pikv_b200.routing import TopKBalancedRouter

D = 128                 # head width of the cache
GROUP = 4               # query heads per KV head
CAPACITY_FACTOR = 1.5


def listed():
    return [
        # routing of one decode batch: one token of each of 64 streams, the smallest call of the append path
        dict(name="route_decode_64", kind="route", tokens=64, hidden=4096, experts=8, n_kv=8, bits=8),
        # a prefill batch, int8 cache: the headline workload
        dict(name="route_prefill_16384", kind="route", tokens=16384, hidden=4096, experts=8, n_kv=8, bits=8),
        # a ragged prefill batch of a model with many experts, 4-bit asymmetric cache
        dict(name="route_ragged_64_experts_q4", kind="route", tokens=5003, hidden=4096, experts=64, n_kv=8, bits=4),
        # one user, one short conversation: the latency of a decode step
        dict(name="decode_single", kind="decode", streams=1, context=1500, ragged=False, n_kv=8, bits=8, h2o=False),
        # a full decode batch over long contexts, the largest case
        dict(name="decode_64x32768", kind="decode", streams=64, context=32768, ragged=False, n_kv=8, bits=8, h2o=False),
        # a batch of requests of different lengths over the 4-bit cache
        dict(name="decode_ragged_q4", kind="decode", streams=24, context=6001, ragged=True, n_kv=8, bits=4, h2o=False),
        # a decode step that also accumulates the attention each position received, for a later eviction
        dict(name="decode_h2o_16x16384", kind="decode", streams=16, context=16384, ragged=False, n_kv=8, bits=8, h2o=True),
        # H2O eviction of long contexts to the 2048-token budget: select, then compact
        dict(name="evict_32x32768", kind="evict", streams=32, context=32768, ragged=False, n_kv=8, budget=2048),
        # the router of the operator surface on a serving batch
        dict(name="router_2048x4096", kind="router", tokens=2048, hidden=4096, experts=8),
        # low-rank compression of the K and V of a long batch
        dict(name="svd_262144x1024", kind="svd", tokens=262144, hidden=1024, rank=64),
        # block-wide 8-bit quantisation of the K and V of one layer
        dict(name="quantize_8192x1024", kind="quantize", tokens=8192, hidden=1024, bits=8, group=128, bf16=False),
        # PiKVMoE forward on the configuration its class is built with
        dict(name="moe_8x128", kind="moe", batch=8, seq=128),
    ]


def _between(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["route", "route", "decode", "decode", "evict", "router", "svd", "quantize", "moe"])
    if kind == "route":
        return dict(kind=kind, tokens=_between(rng, 1, 16384), hidden=rng.choice([1024, 2048, 4096]),
                    experts=rng.choice([4, 8, 16, 64]), n_kv=rng.choice([2, 4, 8]), bits=rng.choice([8, 8, 4]))
    if kind == "decode":
        bits, h2o = rng.choice([(8, False), (8, False), (4, False), (8, True)])
        streams = _between(rng, 1, 64)
        most = 64 * 32768 if bits == 8 and not h2o else 32 * 32768
        return dict(kind=kind, streams=streams, context=_between(rng, 100, min(32768, most // streams)),
                    ragged=rng.random() < 0.6, n_kv=rng.choice([2, 4, 8]), bits=bits, h2o=h2o)
    if kind == "evict":
        context = _between(rng, 1000, 32768)
        return dict(kind=kind, streams=_between(rng, 1, 32), context=context, ragged=rng.random() < 0.5,
                    n_kv=rng.choice([2, 4, 8]), budget=_between(rng, 100, min(2048, context // 2)))
    if kind == "router":
        hidden = rng.choice([256, 512, 1024, 2048, 4096])
        return dict(kind=kind, tokens=_between(rng, 8, 2048 if hidden == 4096 else 4096), hidden=hidden,
                    experts=rng.choice([4, 8, 16]))
    if kind == "svd":
        hidden = rng.choice([512, 1024, 2048])
        return dict(kind=kind, tokens=_between(rng, 64, 262144 * 1024 // max(hidden, 1024)), hidden=hidden,
                    rank=rng.choice([16, 32, 64]))
    if kind == "quantize":
        return dict(kind=kind, tokens=_between(rng, 8, 8192), hidden=rng.choice([256, 512, 1024, 1000]),
                    bits=rng.choice([8, 8, 4]), group=rng.choice([64, 128]), bf16=rng.random() < 0.5)
    return dict(kind=kind, batch=rng.randint(1, 8), seq=_between(rng, 1, 128))


# ----------------------------------------------------------------------------- inputs
def _kv(gen, tokens, n_kv):
    """K or V rows: N(0,1) with 1 % of the channels scaled by 20."""
    x = torch.randn(tokens, n_kv * D, generator=gen, device="cuda")
    cols = torch.randperm(n_kv * D, generator=gen, device="cuda")[: max(1, round(0.01 * n_kv * D))]
    x[:, cols] *= 20.0
    return x.bfloat16()


def _stream_cache(gen, streams, context, n_kv, bits, capacity):
    """A cache whose streams hold `context` rows each, written through append()."""
    cache = pikv_b200.PagedKVCache(streams, capacity, n_kv, bits=bits, symmetric=(bits == 8))
    pos = torch.arange(context, dtype=torch.int32, device="cuda")
    for b in range(streams):
        cache.append(_kv(gen, context, n_kv), _kv(gen, context, n_kv), torch.full_like(pos, b), pos)
    return cache


def _lengths(gen, streams, context, ragged):
    """Rows held by each stream: all `context`, or anything from a tenth of it."""
    if not ragged:
        return torch.full((streams,), context, dtype=torch.int32, device="cuda")
    return torch.randint(max(1, context // 10), context + 1, (streams,), generator=gen, device="cuda", dtype=torch.int32)


def _rope_tables(positions):
    freq = 1.0 / (10000.0 ** (torch.arange(0, D, 2, device="cuda", dtype=torch.float32) / D))
    ang = torch.arange(positions, device="cuda", dtype=torch.float32)[:, None] * freq[None]
    return ang.cos().contiguous(), ang.sin().contiguous()


def prepare(case, seed):
    torch.manual_seed(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")   # noqa: E731
    kind, s = case["kind"], {"kind": case["kind"]}
    if kind == "route":
        T, H, E = case["tokens"], case["hidden"], case["experts"]
        bound = 1.0 / math.sqrt(H)                                     # nn.Linear's default initialisation
        s["w2"] = ((torch.rand(E, H, generator=gen, device="cuda") * 2 - 1) * bound).bfloat16()
        s["b2"] = (torch.rand(E, generator=gen, device="cuda") * 2 - 1) * bound
        s["act"], s["k"], s["v"] = randn(T, H).bfloat16(), _kv(gen, T, case["n_kv"]), _kv(gen, T, case["n_kv"])
        s["capacity"] = 64 + max(16, int(T * CAPACITY_FACTOR * 2 / E))  # rows held, and room for this batch
        s["held"] = torch.randint(0, 64, (E,), generator=gen, device="cuda", dtype=torch.int32)
        s["cache"] = pikv_b200.PagedKVCache(E, s["capacity"], case["n_kv"], bits=case["bits"], symmetric=(case["bits"] == 8))
    elif kind == "decode":
        B, ctx, n_kv = case["streams"], case["context"], case["n_kv"]
        s["cache"] = _stream_cache(gen, B, ctx, n_kv, case["bits"], ctx + 1)
        s["held"] = _lengths(gen, B, ctx, case["ragged"])              # the new token goes behind these rows
        s["seq_len"] = s["held"] + 1
        s["stream"] = torch.arange(B, dtype=torch.int32, device="cuda")
        s["q"], s["k"], s["v"] = randn(B, n_kv * GROUP, D).bfloat16(), _kv(gen, B, n_kv), _kv(gen, B, n_kv)
        s["rope"] = _rope_tables(ctx + 1) if case["bits"] == 8 else None
        s["h2o"] = None
        if case["h2o"]:
            s["acc"] = torch.rand(B * n_kv, ctx + 1, generator=gen, device="cuda")
            s["h2o"] = s["cache"].h2o_workspace(B, n_kv * GROUP)
    elif kind == "evict":
        B, ctx, n_kv, budget = case["streams"], case["context"], case["n_kv"], case["budget"]
        seg = B * n_kv
        s["cache"] = _stream_cache(gen, B, ctx, n_kv, 8, ctx)
        s["dst"] = pikv_b200.PagedKVCache(B, ctx, n_kv)
        s["seg_len"] = _lengths(gen, B, ctx, case["ragged"]).repeat_interleave(n_kv).contiguous()
        # attention received: a few heavy hitters, a long tail
        s["acc"] = (-torch.log(torch.rand(seg, ctx, generator=gen, device="cuda") + 1e-9)) ** 3
        s["ts"] = torch.arange(ctx, dtype=torch.float32, device="cuda").repeat(seg, 1)
        s["recent"] = max(1, budget // 8)
        s["heavy"] = budget - s["recent"]
        s["dst_acc"] = torch.zeros(seg, budget, device="cuda")
        s["dst_ts"] = torch.zeros(seg, budget, device="cuda")
    elif kind == "router":
        with torch.device("cuda"):
            s["router"] = TopKBalancedRouter(case["hidden"], case["experts"], top_k=2).bfloat16().eval()
        s["x"] = randn(1, case["tokens"], case["hidden"]).bfloat16()
    elif kind == "svd":
        with torch.device("cuda"):
            s["svd"] = SVDCompressor(case["hidden"], rank=case["rank"]).bfloat16().eval()
        s["k"] = randn(1, case["tokens"], case["hidden"]).bfloat16()
        s["v"] = randn(1, case["tokens"], case["hidden"]).bfloat16()
    elif kind == "quantize":
        dt = torch.bfloat16 if case["bf16"] else torch.float32
        s["quant"] = QuantizedCompressor(case["hidden"], bits=case["bits"], group_size=case["group"]).cuda().eval()
        s["k"], s["v"] = randn(1, case["tokens"], case["hidden"]).to(dt), randn(1, case["tokens"], case["hidden"]).to(dt)
    else:
        with torch.device("cuda"):
            s["moe"] = PiKVMoE().eval()
        s["x"] = randn(case["batch"], case["seq"], config["hidden_size"])
    return s


# ----------------------------------------------------------------------------- one pass
@torch.no_grad()
def run(s):
    kind = s["kind"]
    if kind == "route":
        cache = s["cache"]
        g = cache.route_append(s["act"], s["w2"], s["b2"], s["k"], s["v"], top_k=2, capacity=s["capacity"], slot_base=s["held"])
        return [g.probs, g.topk_idx, g.topk_w, g.slot, g.counts_k, g.prob_sum, g.new_len,
                cache.k_codes, cache.v_codes, cache.k_scale, cache.v_scale, cache.k_zp, cache.v_zp]
    if kind == "decode":
        cache = s["cache"]
        if s["rope"] is not None:
            cache.append_rope(s["k"], s["v"], s["stream"], s["held"], *s["rope"], positions=s["held"])
        else:
            cache.append(s["k"], s["v"], s["stream"], s["held"])
        if s["h2o"] is not None:
            out = cache.decode_attention_h2o(s["q"], s["acc"], s["h2o"], seq_len=s["seq_len"])
        else:
            out = cache.decode_attention(s["q"], seq_len=s["seq_len"])
        return [out, s.get("acc"), cache.k_codes, cache.v_codes, cache.k_scale, cache.v_scale, cache.k_zp, cache.v_zp]
    if kind == "evict":
        mask, keep, count = ops.h2o_select(s["acc"], s["ts"], s["heavy"], s["recent"], seg_len=s["seg_len"])
        dst = s["dst"]
        s["cache"].compact_into(dst, keep, count, True, s["acc"], s["ts"], s["dst_acc"], s["dst_ts"])
        return [mask, count, dst.k_codes, dst.v_codes, dst.k_scale, dst.v_scale, s["dst_acc"], s["dst_ts"]]
    if kind == "router":
        return list(s["router"](s["x"]))
    if kind == "svd":
        return list(s["svd"](s["k"], s["v"]))
    if kind == "quantize":
        return [*s["quant"](s["k"], s["v"]), s["quant"].quantization_error]
    moe = s["moe"]
    return [moe(s["x"]), moe.cache_ptrs, [[c.keys, c.values, c.importance] for c in moe.kv_caches]]


# ----------------------------------------------------------------------------- what a pass cannot do without
def _row_bytes(n_kv, bits):
    """One cached token: K and V codes, bf16 scales, and fp32 zero points where the cache is asymmetric."""
    return 2 * n_kv * (D * bits // 8 + 2 + (4 if bits == 4 else 0))


def work(case):
    kind = case["kind"]
    if kind == "route":
        T, H, E, n_kv = case["tokens"], case["hidden"], case["experts"], case["n_kv"]
        b = T * (H * 2 + 2 * n_kv * D * 2) + E * H * 2 + T * (E * 4 + 2 * 12) + 2 * T * _row_bytes(n_kv, case["bits"])
        return {"bytes": b, "flops": 2.0 * T * H * E}
    if kind == "decode":
        B, n_kv = case["streams"], case["n_kv"]
        rows = B * case["context"] * (0.55 if case["ragged"] else 1.0)
        b = rows * _row_bytes(n_kv, case["bits"]) + B * n_kv * D * 2 * (2 + 2 * GROUP)
        if case["h2o"]:
            b += rows * n_kv * 8
        return {"bytes": b, "flops": 4.0 * rows * n_kv * GROUP * D}
    if kind == "evict":
        seg = case["streams"] * case["n_kv"]
        scored = seg * case["context"] * (0.55 if case["ragged"] else 1.0)
        kept = seg * case["budget"]
        return {"bytes": scored * 8 + seg * case["context"] + kept * 4 + 2 * kept * (_row_bytes(1, 8) + 8), "flops": 0}
    if kind == "router":
        T, H, E = case["tokens"], case["hidden"], case["experts"]
        cap = max(1, int(T * CAPACITY_FACTOR * 2 / E))
        return {"bytes": T * H * 2 + H * H * 2 + E * H * 2 + T * E * 4 + 2 * T * E * cap * 4,
                "flops": 2.0 * T * H * H + 2.0 * T * H * E}
    if kind == "svd":
        M, H, R = case["tokens"], case["hidden"], case["rank"]
        return {"bytes": 4 * M * H * 2 + 4 * H * R * 2, "flops": 8.0 * M * H * R}
    if kind == "quantize":
        return {"bytes": 4 * case["tokens"] * case["hidden"] * (2 if case["bf16"] else 4), "flops": 0}
    T, H, V, E = case["batch"] * case["seq"], config["hidden_size"], config["vocab_size"], config["num_experts"]
    # experts, the three H x H layers of the router (and its half-width ones), the vocabulary projection
    layers = E * H * H + 3 * H * H
    return {"bytes": 4 * (T * H + T * V + V * H + layers + E * config["kv_cache_size"] * 2 * H),
            "flops": 2.0 * T * (layers + V * H)}


def tolerance(case):
    kind = case["kind"]
    if kind == "route":         # fp32 sums of bf16 products; codes and slots are whole, up to ties of the top-k
        return {"rel": 1e-5, "differ": 1e-3}
    if kind in ("decode", "router", "svd"):                            # bf16 results
        return {"rel": 1e-2, "max": 0.1}
    if kind == "evict":                                                # chosen and moved, not computed
        return "exact"
    if kind == "quantize":                                             # fp32, or bf16 results of the same codes
        return {"rel": 4e-3 if case["bf16"] else 1e-5}
    return {"rel": 1e-5}
