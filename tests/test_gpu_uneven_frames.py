"""Frames of uneven density: a ball, clumps and a film in a much larger box, whose groups hold anything from no atom
to most of them.  Counts against the oracle, alone and in a fused turn; and the work is spread over the GPU, so that
such a frame does not take many times as long as an even one with as many atoms."""
import ctypes
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


def ball(n, box, rho=0.8, seed=1):
    rng = np.random.default_rng(seed)
    a = (1.0 / rho) ** (1.0 / 3.0)
    m = int(2.0 * (3.0 * n / rho / 4.0 / np.pi) ** (1.0 / 3.0) / a) + 3
    g = (np.arange(m) - m / 2) * a
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    x = x[np.argsort((x ** 2).sum(1), kind="stable")[:n]] + rng.normal(0.0, 0.1 * a, (n, 3)) + box / 2
    b = np.full(3, box, np.float32)
    return (x % b).astype(np.float32), rng.integers(0, 2, n).astype(np.int32), b


def clumps(n, box, k, sigma, seed=2):
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, box, (k, 3))[rng.integers(0, k, n)] + rng.normal(0, sigma, (n, 3))
    b = np.full(3, box, np.float32)
    return (x % b).astype(np.float32), rng.integers(0, 2, n).astype(np.int32), b


def film(n, edge, height, thick, seed=3):
    rng = np.random.default_rng(seed)
    b = np.array([edge, edge, height], np.float32)
    x = rng.uniform(0, 1, (n, 3)) * [edge, edge, thick]
    return (x % b).astype(np.float32), rng.integers(0, 2, n).astype(np.int32), b


def even(n, rho=0.8, seed=4):
    rng = np.random.default_rng(seed)
    b = np.full(3, (n / rho) ** (1.0 / 3.0), np.float32)
    return (rng.uniform(0, 1, (n, 3)) * b).astype(np.float32) % b, rng.integers(0, 2, n).astype(np.int32), b


CASES = [("ball_4k", ball(4000, 200.0), 10.0), ("ball_9k_few_groups", ball(9000, 60.0), 19.0),
         ("ball_20k", ball(20000, 250.0), 4.0), ("one_point", clumps(3000, 30.0, 1, 0.3), 3.0),
         ("clumps", clumps(10007, 60.0, 8, 0.6), 3.0), ("film", film(20000, 25.0, 100.0, 10.0), 4.0),
         ("lone_pair", (np.array([[1, 1, 1], [2, 1, 1]], np.float32), np.zeros(2, np.int32),
                        np.full(3, 300.0, np.float32)), 3.0)]


@pytest.mark.parametrize("name,data,rc", CASES, ids=[c[0] for c in CASES])
def test_uneven_counts(ctx, name, data, rc):
    from trj_analysis_b200 import engine
    xyz, sp, box = data
    n = xyz.shape[0]
    pos, sps, _ = orc.layout(xyz, sp, box, 2)
    p = refsem.rdf_params(2, 0.02, rc, box)
    h_o, e_o = orc.rdf_counts(pos, sps, box, p.side2, p.deltar, p.lsmax, 2, cells=False)
    stage = engine.FrameStage(ctx, n, 2)
    stage.upload_and_pack(xyz, sp, box)
    edge = torch.zeros(4, dtype=torch.int64, device="cuda")
    with closing(engine.RdfPlan(ctx, 2, 0.02, rc, box, n)) as plan, closing(engine.Batch(ctx, 2, n + 2)) as batch:
        alone, fused = plan.new_hist(), plan.new_hist()
        plan.accumulate(stage.packed, n, box, alone, edge)
        batch.begin(0)
        batch.stage(0, 1, xyz, sp)  # an odd offset
        batch.add(0, plan, None, 1, n, box, fused, None)
        batch.launch(0)
        batch.mark(0)
        ctx.check()
        assert np.array_equal(alone.cpu().numpy().astype(np.uint64), h_o)
        assert np.array_equal(edge.cpu().numpy()[:3].astype(np.uint64), e_o)
        assert np.array_equal(fused.cpu().numpy().astype(np.uint64), h_o)


def pair_ms(ctx, data, rc):
    from trj_analysis_b200 import engine
    xyz, sp, box = data
    n = xyz.shape[0]
    stage = engine.FrameStage(ctx, n, 2)
    stage.upload_and_pack(xyz, sp, box)
    ms, best = ctypes.c_float(), float("inf")
    ctx.lib.trj_ctx_set_timing(ctx.h, 1)
    with closing(engine.RdfPlan(ctx, 2, 0.02, rc, box, n)) as plan:
        hist = plan.new_hist()
        for _ in range(3):
            plan.accumulate(stage.packed, n, box, hist)
            ctx.lib.trj_rdf_kernel_ms(plan.h, ctypes.byref(ms))
            best = min(best, ms.value)
        ctx.check()
    ctx.lib.trj_ctx_set_timing(ctx.h, 0)
    return best


@pytest.mark.parametrize("n,box,rc", [(4000, 200.0, 10.0), (62500, 400.0, 8.0)])
def test_a_ball_is_spread_over_the_gpu(ctx, n, box, rc):
    """12 and 1,200 times the even frame's time with a warp per group."""
    assert pair_ms(ctx, ball(n, box), rc) < 0.2 + 10.0 * pair_ms(ctx, even(n), rc)
