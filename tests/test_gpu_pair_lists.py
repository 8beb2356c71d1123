"""Work items whose neighbour list holds more than 32 groups of one cell, so that a warp fills its table of group
starts several times: a simple cubic lattice, whose exact pair counts follow from its displacement vectors."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def lattice_counts(m, rc, deltar, lsmax):
    """Pairs per bin of m^3 atoms at integer coordinates of a periodic box of edge m, by the reference's FP32 steps."""
    k = int(rc)
    assert 2 * k < m
    g = np.arange(-k, k + 1)
    r2 = (g[:, None, None] ** 2 + g[None, :, None] ** 2 + g[None, None, :] ** 2).ravel().astype(np.float32)
    r2 = r2[(r2 < np.float32(rc) * np.float32(rc)) & (r2 > 0)]
    q = np.sqrt(r2) / np.float32(deltar)  # FP32, each operation rounded once
    bins = np.floor(q.astype(np.float64) + 0.5).astype(np.int64)
    h = np.bincount(bins, minlength=lsmax + 1)[1:lsmax + 1]
    return h.astype(np.uint64) * np.uint64(m ** 3) // np.uint64(2)


@pytest.mark.parametrize("m,rc", [(40, 12.9), (40, 19.9)], ids=["three_cells", "one_cell"])
def test_lists_of_many_groups(m, rc):
    from trj_analysis_b200 import engine
    deltar = 0.05
    box = np.full(3, m, np.float32)
    g = np.arange(m, dtype=np.float32)
    xyz = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
    ctx = engine.Context(0)
    stage = engine.FrameStage(ctx, m ** 3, 1)
    plan = engine.RdfPlan(ctx, 1, deltar, rc, box, m ** 3)
    n = stage.upload_and_pack(xyz, np.zeros(m ** 3, np.int32), box)
    hist = plan.new_hist()
    plan.accumulate(stage.packed, n, box, hist)
    ctx.check()
    assert np.array_equal(hist.cpu().numpy().astype(np.uint64)[0], lattice_counts(m, rc, deltar, plan.lsmax))
    plan.close()
    ctx.close()
