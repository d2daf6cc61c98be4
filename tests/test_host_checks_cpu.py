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
CALLS = ZERO_WIDTH


@pytest.fixture(scope="module")
def answers():
    r = subprocess.run([sys.executable, "-c", CHILD, json.dumps(CALLS)], capture_output=True, text=True, cwd=ROOT,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0, r.stderr[-2000:]
    return dict(json.loads(line) for line in r.stdout.splitlines())


@pytest.mark.parametrize("call", ZERO_WIDTH)
def test_zero_width(answers, call):
    assert answers[call].startswith("PikvError: ") and "last dimension" in answers[call], answers[call]
