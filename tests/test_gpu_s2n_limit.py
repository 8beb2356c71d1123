"""Number fluctuations where the kernel's dynamic shared memory just fits the 48 KB that need no opt-in, but not
together with its static shared memory; each size in a process of its own, whose first such call it is."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ONE = """
import sys
import numpy as np, torch
from oracle import orc
from trj_analysis_b200 import engine, frames
lsmax = int(sys.argv[1])
fr = frames.FCCSpec(cells=(5, 5, 5), sigma=0.1, seed=11).frame(0)
rc = float(min(fr.box)) / 2
dr = rc / (lsmax - 1)
ctx = engine.Context(0)
stage = engine.FrameStage(ctx, fr.n, 1)
plan = engine.RdfPlan(ctx, 1, dr, rc, fr.box, fr.n)
assert plan.lsmax == lsmax, plan.lsmax
n = stage.upload_and_pack(fr.xyz, fr.types - 1, fr.box)
plan.accumulate(stage.packed, n, fr.box, plan.new_hist())
gi, g2i = plan.new_s2n()
pts = torch.zeros(30, dtype=torch.float32, device=ctx.torch_device)
plan.s2n(10, gi, g2i, points=pts)
ctx.check()
pos, _, _ = orc.layout(fr.xyz, fr.types - 1, fr.box, 1)
a, b = orc.s2n_counts(pos, fr.box, plan.side2, np.float32(dr), plan.lsmax, pts.cpu().numpy().reshape(-1, 3))
assert np.array_equal(gi.cpu().numpy(), a) and np.array_equal(g2i.cpu().numpy(), b)
"""


@pytest.mark.parametrize("lsmax", [12275, 12280, 12287, 12288, 28000])
def test_s2n_shared_memory_limit(lsmax):
    r = subprocess.run([sys.executable, "-c", ONE, str(lsmax)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
