"""Floor bins against the oracle at several thousand bins, where q = r/deltar is large and the window around a bin
edge in which a pair is looked at exactly is widest: counts, edge statistics and the charged form."""
import numpy as np
import pytest
import torch

from oracle import orc
from trj_analysis_b200 import frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,nsp,rmax,nbins", [((9, 9, 9), 1, 7.1, 7001), ((9, 9, 9), 2, 3.0, 12011),
                                                  ((10, 10, 10), 1, 8.3, 40000), ((6, 6, 6), 3, 2.9, 5)])
def test_floor_bins_bit_exact(cells, nsp, rmax, nbins):
    from trj_analysis_b200 import engine
    fr = frames.FCCSpec(cells=cells, sigma=0.1, fractions=(1.0,) * nsp, replace_frac=0.02, seed=21).frame(0)
    n, sp = fr.n, fr.types - 1
    ctx = engine.Context(0)
    stage = engine.FrameStage(ctx, n, nsp)
    plan = engine.RdfPlan(ctx, nsp, 0.0, rmax, fr.box, n, floor_bins=nbins)
    stage.upload_and_pack(fr.xyz, sp, fr.box)
    pos, sps, _ = orc.layout(fr.xyz, sp, fr.box, nsp)
    dr = np.float32(rmax) / np.float32(nbins)
    side2 = np.float32(rmax) * np.float32(rmax)
    h_o, e_o = orc.rdf_counts(pos, sps, fr.box, side2, dr, plan.lsmax, nsp, cells=False, floor_bins=True)
    edge = torch.zeros(4, dtype=torch.int64, device="cuda")
    with_edges, without = plan.new_hist(), plan.new_hist()
    plan.accumulate(stage.packed, n, fr.box, with_edges, edge)
    plan.accumulate(stage.packed, n, fr.box, without)
    ctx.check()
    assert np.array_equal(with_edges.cpu().numpy().astype(np.uint64), h_o)
    assert np.array_equal(without.cpu().numpy().astype(np.uint64), h_o)
    assert np.array_equal(edge.cpu().numpy()[:3].astype(np.uint64), e_o)
    if nbins * (4 * plan.nit + 8) < 200000:  # the charge sums take shared memory as well
        q = torch.linspace(-1.0, 1.0, n, device="cuda", dtype=torch.float32)
        charged, gqq = plan.new_hist(), plan.new_gqq()
        plan.accumulate(stage.packed, n, fr.box, charged, qpacked=q, gqq=gqq)
        ctx.check()
        assert np.array_equal(charged.cpu().numpy().astype(np.uint64), h_o)
    plan.close()
    ctx.close()
