"""The tensor-core S(Q) at the edges of its stages (32 atoms), runs (256 atoms) and tile widths.

Tolerance per vector: the split BF16 factors keep about 16 bits each, at most 3e-5 per atom of the species,
plus 1e-5 (as for the other split sums).
"""
import numpy as np
import pytest

from oracle import orc
from trj_analysis_b200 import refsem

pytestmark = pytest.mark.gpu

COUNTS = [(1,), (31, 1), (32, 33), (255, 256, 257), (512, 97)]


@pytest.mark.parametrize("cols", [32, 112, 208, 224])
@pytest.mark.parametrize("counts", COUNTS, ids=lambda c: "-".join(map(str, c)))
def test_split_sum_at_stage_edges(counts, cols):
    from trj_analysis_b200 import engine
    nsp, n = len(counts), sum(counts)
    rng = np.random.default_rng(n + cols)
    box = np.array([9.0, 7.0, 11.0], dtype=np.float32)
    xyz = (rng.random((n, 3)) * box).astype(np.float32)
    sp = np.repeat(np.arange(nsp), counts).astype(np.int32)
    ks = refsem.make_kset("full", box, 9.0)
    assert ks.dense.any()
    ctx = engine.Context(0)
    try:
        ctx.set_sq_tile_cols(cols)
        stage = engine.FrameStage(ctx, n, nsp)
        plan = engine.SqPlan(ctx, nsp, ks, np.array(counts))
        out = plan.new_out()
        stage.upload_and_pack(xyz, sp, box)
        plan.accumulate(stage.packed, n, box, out, engine.METHODS["split"])
        rho = plan.rho().cpu().numpy()
        ctx.check()
        plan.close()
    finally:
        ctx.close()
    pos, _, off = orc.layout(xyz, sp, box, nsp)
    ref = orc.rho_fp64(pos, off, box, ks.vectors)
    for a in range(nsp):
        assert np.abs(rho[a] - ref[a]).max() <= 3e-5 * counts[a] + 1e-5
