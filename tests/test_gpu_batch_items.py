"""Work items of a fused turn: enough of them for the GPU's warps where the turn has room for few frames, and every
unit of a table of many items finds its own frame."""
from contextlib import closing

import numpy as np
import pytest
import torch

from oracle import orc
from trj_analysis_b200 import refsem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from trj_analysis_b200 import engine
    c = engine.Context(0)
    yield c
    c.close()


def ball(n, edge, seed=1):
    rng = np.random.default_rng(seed)
    r = (3.0 * n / (4.0 * np.pi * 0.8)) ** (1.0 / 3.0)
    v = rng.normal(size=(n, 3))
    x = edge / 2 + r * rng.uniform(0, 1, (n, 1)) ** (1.0 / 3.0) * v / np.linalg.norm(v, axis=1, keepdims=True)
    return x.astype(np.float32), np.full(3, edge, np.float32)


@pytest.mark.parametrize("n,edge,rc", [(16000, 200.0, 8.0), (1000, 40.0, 5.0)])
def test_one_frame_fills_the_gpu(ctx, n, edge, rc):
    """At least an item per warp, or four times what a turn of 64 such frames takes of each (before: the same)."""
    from trj_analysis_b200 import engine
    xyz, box = ball(n, edge)
    with closing(engine.RdfPlan(ctx, 1, 0.02, rc, box, 0)) as plan, closing(engine.Batch(ctx, 1, n)) as one, \
            closing(engine.Batch(ctx, 64, 64 * n)) as many:
        units = []
        for b in (one, many):
            b.begin(0)
            b.add(0, plan, None, 0, n, box, plan.new_hist(), None)
            units.append(b.info(0)[1][1])
        warps = 24 * ctx.lib.trj_ctx_sm_count(ctx.h)
        assert units[0] >= min(warps, 4 * units[1])


@pytest.mark.parametrize("items", [1, 2, 31, 32, 33, 64, 1000, 1025, 2100])
def test_every_unit_finds_its_frame(ctx, items):
    from trj_analysis_b200 import engine
    rng = np.random.default_rng(items)
    sizes = rng.integers(1, 40, items)
    sizes[items // 2] = 1500  # several units
    off = np.concatenate([[0], np.cumsum(sizes)])
    box = np.full(3, 5.0, np.float32)
    p = refsem.rdf_params(1, 0.1, 2.5, box)
    with closing(engine.Batch(ctx, items, int(off[-1]))) as batch, closing(engine.RdfPlan(ctx, 1, 0.1, 2.5, box, 0)) as plan:
        hists = torch.zeros((items, plan.nit, plan.lsmax), dtype=torch.int64, device="cuda")
        xyz = rng.uniform(0, 5.0, (int(off[-1]), 3)).astype(np.float32) % box
        batch.begin(0)
        batch.stage(0, 0, xyz, np.zeros(len(xyz), np.int32))
        for k in range(items):
            batch.add(0, plan, None, int(off[k]), int(sizes[k]), box, hists[k], None)
        batch.launch(0)
        batch.mark(0)
        ctx.check()
        got = hists.cpu().numpy().astype(np.uint64)
    for k in range(items) if items <= 64 else (*range(0, items, 37), items // 2, items - 1):
        x = xyz[off[k]:off[k + 1]]
        want, _ = orc.rdf_counts(x, np.zeros(len(x), np.int32), box, p.side2, p.deltar, p.lsmax, 1, cells=False)
        assert np.array_equal(got[k], want), k
