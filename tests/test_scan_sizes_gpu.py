"""Heads whose rows of a step need more shared memory than a kernel has by default: a call that rotates more dimensions than the first one
of its process (in a process of its own: the size is given once)."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import torch
from tensorline_b200 import ops
H, d, dv, T = 1, 256, 16, 40
g = torch.Generator().manual_seed(1)
proj = torch.randn(T, 2 * d + dv, generator=g).cuda()
i32 = dict(dtype=torch.int32, device="cuda")
start, slots, pos = torch.tensor([0, T], **i32), torch.zeros(1, **i32), torch.arange(T, **i32)
for rot in (2, 256, 0):
    outs = []
    for cuts in ([0, T], [0, 7, T]):
        state, out = torch.zeros(1, ops.scan_state_floats(d, False), device="cuda"), torch.empty(T, dv, device="cuda")
        inv = (10000.0 ** (-torch.arange(0, rot, 2).float() / max(rot, 1))).cuda()
        for a, b in zip(cuts, cuts[1:]):
            ops.linear_scan(proj[a:b], 0, d, 2 * d, H, d, dv, state, torch.tensor([0, b - a], **i32), slots, pos[a:b].contiguous(), out[a:b], B=1,
                            decay=torch.tensor([0.9], device="cuda"), inv_freq=inv if rot else None, rot=rot)
        outs.append(out)
    assert torch.equal(*outs) and bool(outs[0].isfinite().all())
print("ok")
"""


def test_more_rotated_dimensions_than_in_the_first_call():
    run = subprocess.run([sys.executable, "-c", PROGRAM], cwd=Path(__file__).resolve().parents[1], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout.strip() == "ok", run.stdout + run.stderr
