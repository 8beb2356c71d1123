"""Frames of so many pairs that CTAs move their 32-bit rows to the frame's histogram on the way: a simple cubic
lattice, whose counts are known exactly.  96^3 atoms have 2e11 pairs within half the box, which take the GPU some 0.35 s,
and the rows are moved every 35 ms."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

M = 96  # sites per axis; spacing 1, so that every squared distance is a whole number below 2^24


def expected(plan, floor):
    """Counts per row (species = parity of x) and bin, by the pair's displacement."""
    d = np.arange(M)
    d = np.minimum(d, M - d).astype(np.int64)
    rr2 = (d[:, None, None] ** 2 + d[None, :, None] ** 2 + d[None, None, :] ** 2).astype(np.float32)
    odd = np.broadcast_to((np.arange(M) % 2 == 1)[:, None, None], rr2.shape)
    q = (np.sqrt(rr2).astype(np.float32) / np.float32(plan_dr)).astype(np.float32)
    ind = np.floor(q).astype(np.int64) + 1 if floor else np.floor(q.astype(np.float64) + 0.5).astype(np.int64)
    ok = (rr2 < np.float32(plan.side2)) & (ind >= 1) & (ind <= plan.lsmax)
    ok[0, 0, 0] = False
    n = M ** 3
    out = np.zeros((3, plan.lsmax), np.int64)
    same = np.bincount(ind[ok & ~odd] - 1, minlength=plan.lsmax)
    out[0] = out[2] = same * (n // 4)
    out[1] = np.bincount(ind[ok & odd] - 1, minlength=plan.lsmax) * (n // 2)
    return out


plan_dr = 4.0  # coarse bins: the fullest ones


@pytest.mark.parametrize("floor,edge,fused", [(False, False, False), (False, True, False), (True, True, False),
                                              (False, False, True), (False, True, True)])
def test_rows_are_moved_on_the_way(floor, edge, fused):
    from trj_analysis_b200 import engine
    ctx = engine.Context(0)
    g = np.arange(M, dtype=np.float32)
    xyz = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    sp = (xyz[:, 0].astype(np.int32) % 2).astype(np.int32)
    n, box = M ** 3, np.full(3, float(M), np.float32)
    plan = engine.RdfPlan(ctx, 2, plan_dr, 1e9, box, 0 if fused else n)
    plan.set_binning(floor)
    hist = plan.new_hist()
    stats = torch.zeros(4, dtype=torch.int64, device="cuda") if edge else None
    if fused:
        batch = engine.Batch(ctx, 1, n)
        batch.begin(0)
        batch.stage(0, 0, xyz, sp)
        batch.add(0, plan, None, 0, n, box, hist, None, stats)
        batch.launch(0)
        batch.mark(0)
        ctx.check()
        batch.close()
    else:
        packed = torch.tensor(np.concatenate([xyz, sp.view(np.float32)[:, None]], 1), device="cuda")
        plan.accumulate(packed, n, box, hist, stats)
        ctx.check()
    want = expected(plan, floor)
    assert np.array_equal(hist.cpu().numpy(), want)
    if edge:
        assert int(stats[2]) == int(want.sum())
    plan.close()
    ctx.close()
