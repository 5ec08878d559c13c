"""Device memory of attention plans."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import torch
from raptor_t_b200 import capi, metadata, ops
cfg = capi.make_config(hidden=768, heads=12, ffn=3072, layers=1, max_pos=16384, vocab=97)
lens = [16384]
ptr, idx = metadata.build_block_csr(cfg, 0, lens)
torch.zeros(1, device="cuda")
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
plans = [ops.AttentionPlan(cfg, lens, ptr, idx) for _ in range(6)]
held = before - torch.cuda.mem_get_info()[0]
for p in plans:
    p.close()
left = before - torch.cuda.mem_get_info()[0]
print(held, left)
assert held > 16 << 20 and left <= 2 << 20, (held, left)
"""


def test_memory_goes_back_with_the_last_plan():
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]
