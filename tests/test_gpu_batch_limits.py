"""Batches of different histogram sizes side by side: the shared memory that one asks for does not limit another."""
import numpy as np
import pytest
import torch

from trj_analysis_b200 import frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("words", [(24576, 64), (8192, 4096, 1)])
def test_smaller_batch_made_later(words):
    from trj_analysis_b200 import engine
    fr = frames.FCCSpec(cells=(5, 5, 5), sigma=0.1, seed=3).frame(0)
    sp = np.zeros(fr.n, np.int32)
    ctx = engine.Context(0)
    batches = [engine.Batch(ctx, 1, fr.n, w) for w in words]
    half = float(min(fr.box)) / 2
    plans = [engine.RdfPlan(ctx, 1, 1.01 * half / max(w - 2, 0.5), 0.0, fr.box, 0) for w in words]
    hists = [p.new_hist() for p in plans]
    for b, p, h in zip(batches, plans, hists):
        b.begin(0)
        b.stage(0, 0, fr.xyz, sp)
        b.add(0, p, None, 0, fr.n, fr.box, h, None)
        b.launch(0)
        b.mark(0)
    ctx.check()
    stage = engine.FrameStage(ctx, fr.n, 1)
    stage.upload_and_pack(fr.xyz, sp, fr.box)
    for b, p, h in zip(batches, plans, hists):
        one = engine.RdfPlan(ctx, 1, np.float32(1.01 * half / max(b.hist_words - 2, 0.5)), 0.0, fr.box, fr.n)
        want = one.new_hist()
        one.accumulate(stage.packed, fr.n, fr.box, want)
        ctx.check()
        assert torch.equal(want, h)
        one.close()
        p.close()
        b.close()
    ctx.close()
