"""Device memory of a render's path states: 232 bytes a path (13 float4 and 6
words), and 42 more for the slots of parked traversals only in a process that
gives traversals a step budget.  The memory that a render of two states of 2^21
paths takes, read in a process of its own; 20 bytes a path either way are the
image, the tables and the allocator's rounding."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

_CODE = """
import torch
import pt_gb300 as P
from pt_gb300 import scenes
raw, cam = scenes.tiny_raw("two_tris")
hs = P.HostScene.from_raw(raw, cam)
torch.zeros(1, device="cuda")
with P.Context(0) as ctx:
    ctx.upload(hs.pack())
    ctx.build_accel()
    ctx.render(hs.render_params(16, 16, 2, 2))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ctx.render(hs.render_params(2048, 1024, 2, 2))
    torch.cuda.synchronize()
    print("bytes a path", (before - torch.cuda.mem_get_info()[0]) / 2**22)
"""


@pytest.mark.parametrize("env,per_path", [({}, 232), ({"PT_EXTEND_BUDGET_MIN_LOG2": "0"}, 274), ({"PT_SHADOW_BUDGET": "48"}, 274)],
                         ids=["default", "extend_budget", "shadow_budget"])
def test_bytes_a_path(env, per_path):
    pytest.importorskip("torch")
    env = {k: v for k, v in os.environ.items() if not k.startswith(("PT_EXTEND", "PT_SHADOW", "PT_WAVE"))} | env
    r = subprocess.run([sys.executable, "-c", _CODE], cwd=Path(__file__).resolve().parent.parent, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    got = float(r.stdout.split()[-1])
    assert abs(got - per_path) < 20, got
