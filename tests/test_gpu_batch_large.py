"""Large frames in a fused turn: the number of pair work items stays in range, and frames whose neighbour lists are
cut by that bound have the counts of the single-request call."""
import numpy as np
import pytest
import torch

from trj_analysis_b200 import frames

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from trj_analysis_b200 import engine
    c = engine.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [6_200_000, 8_600_000, 9_200_000])
def test_pair_items_of_a_large_frame(ctx, n):
    """Described only, not launched: cutoff half the box, the frame's groups all in one cell."""
    from trj_analysis_b200 import engine
    box = np.full(3, (n / 0.8) ** (1.0 / 3.0), np.float32)
    batch = engine.Batch(ctx, 1, n)
    plan = engine.RdfPlan(ctx, 1, 0.5, 1e9, box, 0)
    batch.begin(0)
    batch.add(0, plan, None, 0, n, box, plan.new_hist(), None)
    _, units = batch.info(0)
    assert n // 32 <= units[1] <= max(1 << 20, n // 8 + 64)
    plan.close()
    batch.close()


def test_capped_lists_match_single_request(ctx):
    from trj_analysis_b200 import engine
    fr = frames.FCCSpec(cells=(33, 33, 33), sigma=0.1, fractions=(0.5, 0.5), seed=31).frame(0)
    sp = (fr.types - 1).astype(np.int32)
    plan = engine.RdfPlan(ctx, 2, 0.05, 1e9, fr.box, fr.n)
    stage = engine.FrameStage(ctx, fr.n, 2)
    stage.upload_and_pack(fr.xyz, sp, fr.box)
    one, fused = plan.new_hist(), plan.new_hist()
    plan.accumulate(stage.packed, fr.n, fr.box, one)
    batch = engine.Batch(ctx, 1, fr.n)
    batch.begin(0)
    batch.stage(0, 0, fr.xyz, sp)
    batch.add(0, plan, None, 0, fr.n, fr.box, fused, None)
    batch.launch(0)
    batch.mark(0)
    ctx.check()
    batch.wait(0)
    assert int(one.sum()) > 0 and torch.equal(one, fused)
    plan.close()
    batch.close()
