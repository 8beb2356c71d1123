"""Number fluctuations at the edges of the kernel's loops: bins around the 256 threads of the block scan, one
group per cell and many, split and unsplit axes.  Exact against the oracle at the kernel's own points."""
import numpy as np
import pytest
import torch

from oracle import orc
from trj_analysis_b200 import frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,rc,lsmax", [((2, 2, 2), 0.0, 2), ((5, 5, 5), 0.0, 255), ((8, 8, 8), 2.0, 256),
                                            ((8, 8, 16), 4.0, 257), ((14, 14, 14), 7.0, 1030)])
def test_s2n_sizes(cells, rc, lsmax):
    from trj_analysis_b200 import engine
    fr = frames.FCCSpec(cells=cells, sigma=0.1, fractions=(0.5, 0.5), seed=11).frame(0)
    dr = (rc or float(min(fr.box)) / 2) / (lsmax - 1)
    ctx = engine.Context(0)
    stage = engine.FrameStage(ctx, fr.n, 2)
    plan = engine.RdfPlan(ctx, 2, dr, rc, fr.box, fr.n)
    assert abs(plan.lsmax - lsmax) <= 1
    n = stage.upload_and_pack(fr.xyz, fr.types - 1, fr.box)
    plan.accumulate(stage.packed, n, fr.box, plan.new_hist())
    gi, g2i = plan.new_s2n()
    pts = torch.zeros(3 * 50, dtype=torch.float32, device=ctx.torch_device)
    plan.s2n(50, gi, g2i, points=pts)
    ctx.check()
    pos, _, _ = orc.layout(fr.xyz, fr.types - 1, fr.box, 2)
    a, b = orc.s2n_counts(pos, fr.box, plan.side2, np.float32(dr), plan.lsmax, pts.cpu().numpy().reshape(-1, 3))
    np.testing.assert_array_equal(gi.cpu().numpy(), a)
    np.testing.assert_array_equal(g2i.cpu().numpy(), b)
