"""What the native host module refuses before anything reaches the GPU: fake CUDA tensors stand for the real ones.  One child
process imports the package and forks for every call, as a check that is missing may end the process instead of raising."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import json, os, sys
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
import pikv_b200
from pikv_b200 import ops
bf, f32, i32 = torch.bfloat16, torch.float32, torch.int32
def t(*shape, dtype=bf):
    return torch.empty(*shape, dtype=dtype, device="cuda")
with FakeTensorMode():               # what it imports on first use, once
    t(1)
for call in json.loads(sys.argv[1]):
    r, w = os.pipe()
    pid = os.fork()
    if pid == 0:
        text = "not refused"
        with FakeTensorMode():
            try:
                exec(call)
            except Exception as e:
                text = type(e).__name__ + ": " + str(e)
        os.write(w, text[:400].encode())
        os._exit(0)
    os.close(w)
    status = os.waitpid(pid, 0)[1]
    print(json.dumps([call, os.read(r, 4096).decode() if status == 0 else "the process ended with status %d" % status]))
"""

ZERO_WIDTH = [
    "ops.lowrank_project(t(4, 0), t(16, 0))",
    "ops.lowrank_pair((t(4, 0), t(4, 0)), [t(16, 0)] * 2, [None] * 2, [t(32, 16)] * 2, [None] * 2)",
    "ops.linear_f32(t(4, 0, dtype=f32), t(16, 0, dtype=f32))",
    "ops.gate_mlp_fused(t(4, 0), t(16, 0), None, t(8, 16), None)",
    "ops.quant_block_pair(t(4, 0), t(4, 0), 64, 0, 255, False)",
]
CACHE = "c = object.__new__(pikv_b200.PagedKVCache); torch.nn.Module.__init__(c); c.num_seqs, c.n_kv, c.bits, c.symmetric, c.max_pages, c.num_pages = 4, 2, 8, True, 2, 8; "
CACHE += "[c.register_buffer(n, t(4, 2, dtype=i32)) for n in ('length', 'page_table')]; "
# each lacks elements that a kernel would read or write
SHORT = [
    "ops.lowrank_project(t(4, 64), t(32, 64), t(31))",
    "ops.lowrank_project(t(4, 64), t(32, 64), residual=t(3, 32))",
    "ops.lowrank_pair((t(4, 64), t(4, 64)), [t(16, 64)] * 2, [t(16), t(15)], [t(32, 16)] * 2, [None] * 2)",
    "ops.lowrank_pair((t(4, 64), t(4, 64)), [t(16, 64)] * 2, [None] * 2, [t(32, 16)] * 2, [t(32), t(16)])",
    "ops.gate_mlp_fused(t(4, 64), t(16, 64), t(8), t(8, 16), None)",
    "ops.gate_mlp_fused(t(4, 64), t(16, 64), None, t(8, 16), t(4))",
    "ops.gate_fused(t(4, 64), t(8, 64), t(7))",
    "ops.gate_fused(t(4, 64), t(8, 64), expert_mask=t(7, dtype=f32))",
    "ops.gate_fused(logits=t(4, 8, dtype=f32), correction=t(4, dtype=f32))",
    "ops.gate_fused(logits=t(4, 8, dtype=f32), slot_base=t(4, dtype=i32))",
    "ops.dispatch_loss(ops.GateResult(None, t(4, 2, dtype=i32), t(4, 1, dtype=f32), t(4, 2, dtype=i32), t(2, 8, dtype=i32), t(8, dtype=f32), None), 8, 4)",
    "ops.dispatch_loss(ops.GateResult(None, t(4, 2, dtype=i32), t(4, 2, dtype=f32), t(4, 2, dtype=i32), t(2, 4, dtype=i32), t(8, dtype=f32), None), 8, 4)",
    "ops.quant_block_pair(t(4, 64), t(4, 64), 32, 0, 255, False, params_in=t(1, 2, dtype=f32))",
    CACHE + "c.decode_attention_h2o(t(4, 8, 128), t(7, 32, dtype=f32), (t(4, 8, 32, dtype=torch.float16), t(4, 8, 2, dtype=f32)))",
    CACHE + "c.decode_attention_h2o(t(4, 8, 128), t(8, 32, dtype=f32), (t(3, 8, 32, dtype=torch.float16), t(4, 8, 2, dtype=f32)))",
    CACHE + "c.decode_attention_h2o(t(4, 8, 128), t(8, 32, dtype=f32), (t(4, 8, 32, dtype=torch.float16), t(4, 4, 2, dtype=f32)))",
    CACHE + "c.decode_attention(t(4, 8, 128), scores=t(4, 4, 32, dtype=f32))",
    CACHE + "c.compact_into(c, t(7, 4, dtype=i32), t(8, dtype=i32), True)",
    CACHE + "c.compact_into(c, t(4, 4, dtype=i32), t(3, dtype=i32), False)",
]
TORCH_ERROR = CACHE + "c.append(t(4, 256), t(4, 256), t((), dtype=i32), t(4, dtype=i32))"      # a dst_seq without a dimension
# a result given to be written into, one of its members unfit
RESULT = "r = ops.GateResult(t(4, 8, dtype=f32), t(4, 2, dtype=i32), t(4, 2, dtype=f32), t(4, 2, dtype=i32), t(2, 8, dtype=i32), t(8, dtype=f32), t(8, dtype=i32)); "
MEMBERS = [RESULT + "r.%s = %s; ops.gate_fused(t(4, 64), t(8, 64), out=r)" % m for m in [
    ("topk_idx", "__import__('numpy').zeros((4, 2), 'int32')"), ("new_len", "[0] * 8"), ("workspace", "bytearray(1 << 20)"),
    ("topk_w", "t(4, 2)"), ("slot", "t(2, 4, dtype=i32).t()"), ("counts_k", "t(1, 8, dtype=i32)"),
    ("probs", "torch.empty(4, 8)"), ("prob_sum", "t(4, dtype=f32)")]]
# what is updated in place, as a strided view
WRITTEN = [
    CACHE + "c.decode_attention_h2o(t(4, 8, 128), t(8, 64, dtype=f32)[:, :32], (t(4, 8, 32, dtype=torch.float16), t(4, 8, 2, dtype=f32)))",
    CACHE + "c.decode_attention(t(4, 8, 128), scores=t(4, 8, 64, dtype=f32)[:, :, :32])",
    CACHE + "c.compact_into(c, t(8, 4, dtype=i32), t(8, dtype=i32), True, t(8, 32, dtype=f32), None, t(8, 64, dtype=f32)[:, :32], None)",
    CACHE + "c.compact_into(c, t(8, 4, dtype=i32), t(8, dtype=i32), True, None, t(8, 32, dtype=f32), None, t(8, 64, dtype=f32)[:, :32])",
    "ops.h2o_accumulate(t(64, dtype=f32)[::2], t(32, dtype=f32), None, t(32, dtype=f32), 1.0)",
    "ops.h2o_accumulate(t(32, dtype=f32), t(64, dtype=f32)[::2], None, t(32, dtype=f32), 1.0)",
    "ops.h2o_accumulate_attn(t(4, 8, 32, dtype=f32), t(4, 8, dtype=f32), None, 2, t(8, 64, dtype=f32)[:, :32])",
]
CALLS = WRITTEN + MEMBERS + ZERO_WIDTH + SHORT + [TORCH_ERROR]


@pytest.fixture(scope="module")
def answers():
    r = subprocess.run([sys.executable, "-c", CHILD, json.dumps(CALLS)], capture_output=True, text=True, cwd=ROOT,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0, r.stderr[-2000:]
    return dict(json.loads(line) for line in r.stdout.splitlines())


@pytest.mark.parametrize("call", ZERO_WIDTH)
def test_zero_width(answers, call):
    assert answers[call].startswith("PikvError: ") and "last dimension" in answers[call], answers[call]


@pytest.mark.parametrize("call", SHORT)
def test_short_operands(answers, call):
    assert answers[call].startswith("PikvError: ") and "are needed" in answers[call], answers[call]


def test_torch_errors_keep_their_type(answers):
    assert answers[TORCH_ERROR].startswith("IndexError: "), answers[TORCH_ERROR]


@pytest.mark.parametrize("call", MEMBERS)
def test_members_of_a_given_result(answers, call):
    assert answers[call].startswith("PikvError: ") and ("must be a" in answers[call] or "are needed" in answers[call]), answers[call]


@pytest.mark.parametrize("call", WRITTEN)
def test_strided_views_that_are_written(answers, call):
    assert answers[call].startswith("PikvError: ") and "must be contiguous" in answers[call], answers[call]
