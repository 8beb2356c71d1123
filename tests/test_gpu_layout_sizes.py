"""Frame layout and cell sort at the sizes where their launch forms change, against the host layout."""
import numpy as np
import pytest

from oracle import orc
from trj_analysis_b200 import refsem
from trj_analysis_b200._lib import TrjError

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from trj_analysis_b200 import engine
    c = engine.Context(0)
    yield c
    c.close()


def frame(n, nsp, seed=0):
    rng = np.random.default_rng([n, nsp, seed])
    box = np.array([20.0, 21.0, 23.0], np.float32)
    xyz = (rng.uniform(-1, 2, (n, 3)) * box).astype(np.float32)
    return xyz, rng.integers(0, nsp, n).astype(np.int32), box


@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 8192, 8193, 131072, 131073])
@pytest.mark.parametrize("nsp", [1, 16])
def test_layout_sizes(ctx, n, nsp):
    import torch
    from trj_analysis_b200 import engine
    xyz, sp, box = frame(n, nsp)
    q = np.arange(n, dtype=np.float32)
    pos, sps, off = orc.layout(xyz, sp, box, nsp)
    stage = engine.FrameStage(ctx, n, nsp, charged=True)
    stage.upload_and_pack(xyz, sp, box, charges=q)
    ctx.check()
    got = stage.packed[:n].cpu().numpy()
    assert np.array_equal(got[:, :3], pos)
    assert np.array_equal(got[:, 3].view(np.int32), sps)
    assert np.array_equal(stage.counts.cpu().numpy(), np.diff(off))
    assert np.array_equal(stage.qpacked[:n].cpu().numpy(), q[np.argsort(sp, kind="stable")])
    lut = torch.tensor([-1] + list(range(nsp)), dtype=torch.int32, device="cuda")
    plain = engine.FrameStage(ctx, n, nsp)
    plain.upload_and_pack_types(xyz, sp + 1, box, lut)
    ctx.check()
    assert np.array_equal(plain.packed[:n].cpu().numpy().view(np.int32), got.view(np.int32))


@pytest.mark.parametrize("n", [700, 8192, 8193])
def test_bad_data_is_reported_at_every_size(ctx, n):
    from trj_analysis_b200 import engine
    for bad in ("species", "nan"):
        xyz, sp, box = frame(n, 2, seed=1)
        if bad == "species":
            sp[n // 2] = 7
        else:
            xyz[n - 1, 2] = np.nan
        stage = engine.FrameStage(ctx, n, 2)
        rdf = engine.RdfPlan(ctx, 2, 0.05, 3.0, box, n)
        stage.upload_and_pack(xyz, sp, box)
        rdf.accumulate(stage.packed, n, box, rdf.new_hist())
        with pytest.raises(TrjError) as ei:
            ctx.check()
        assert ei.value.code == -5
        rdf.close()


@pytest.mark.parametrize("n,rc", [(8191, 2.0), (8192, 9.0), (8193, 2.0), (8193, 9.0)])
def test_sort_sizes_bit_exact(ctx, n, rc):
    from trj_analysis_b200 import engine
    xyz, sp, box = frame(n, 2, seed=2)
    pos, sps, _ = orc.layout(xyz, sp, box, 2)
    p = refsem.rdf_params(2, 0.05, rc, box)
    want, _ = orc.rdf_counts(pos, sps, box, p.side2, p.deltar, p.lsmax, 2)
    q = np.random.default_rng(5).normal(size=n).astype(np.float32)
    stage = engine.FrameStage(ctx, n, 2, charged=True)
    stage.upload_and_pack(xyz, sp, box, charges=q)
    plan = engine.RdfPlan(ctx, 2, 0.05, rc, box, n)
    hist, gqq = plan.new_hist(), plan.new_gqq()
    plan.accumulate(stage.packed, n, box, hist, qpacked=stage.qpacked, gqq=gqq)
    ctx.check()
    assert np.array_equal(hist.cpu().numpy().astype(np.uint64), want)
    order = np.argsort(sp, kind="stable")
    _, _, sums = orc.rdf_charged(pos, sps, q[order], box, p.side2, p.deltar, p.lsmax, 2, cells=False)
    avq2 = np.float64(np.float32((q.astype(np.float64) ** 2).sum() / n))
    # FP64 sums of at most a few thousand products in another order
    np.testing.assert_allclose(gqq.cpu().numpy(), sums / avq2, rtol=0, atol=1e-11 * np.abs(sums / avq2).max())
    plan.close()
