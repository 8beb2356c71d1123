"""A plan's device arrays come in few allocations (each costs up to 0.3 ms, and plans are made per request), and the
time-correlation plan orders its vectors without sorting: any order and range of the components gives the same sums."""
import ctypes
import time
from contextlib import closing

import numpy as np
import pytest
import torch

from trj_analysis_b200 import frames, refsem

pytestmark = pytest.mark.gpu


@pytest.fixture
def ctx():
    from trj_analysis_b200 import engine
    from trj_analysis_b200.serve import ALLOC_FN, FREE_FN
    c = engine.Context(0)
    live, made = {}, []

    def alloc(nbytes, user):
        t = torch.empty(max(int(nbytes), 1), dtype=torch.uint8, device="cuda")
        live[t.data_ptr()] = t
        made.append(int(nbytes))
        return t.data_ptr()

    def free(ptr, user):
        del live[int(ptr)]
    a, f = ALLOC_FN(alloc), FREE_FN(free)
    engine.check(c.lib.trj_ctx_set_allocator(c.h, ctypes.cast(a, ctypes.c_void_p), ctypes.cast(f, ctypes.c_void_p), None),
                 c.h, "trj_ctx_set_allocator")
    c.made, c.live = made, live
    yield c
    c.close()
    assert not live


def sqw(vectors, nbins=1):
    v = np.asarray(vectors, np.int64)
    b = np.arange(len(v)) % nbins
    return refsem.SqwSet(qw=np.arange(nbins, dtype=np.float32) + 1, dq=0.1, vectors=v, bins=b,
                         nw=np.bincount(b, minlength=nbins))


def test_allocations_of_plans(ctx):
    from trj_analysis_b200 import engine
    fr = frames.FCCSpec(cells=(12, 12, 12), seed=3).frame(0)
    plan = engine.SqPlan(ctx, 1, refsem.make_kset("full+axes", fr.box, 8.0, 3.0), np.array([fr.n]))
    assert plan.n_tiles > 0 and sum(ctx.made) >= plan.scratch_bytes
    big = [b for b in ctx.made if b > 1 << 20]
    assert len(big) <= 2, big
    plan.close()
    ctx.made.clear()
    with closing(engine.DynPlan(ctx, 1, fr.n, 10, 20, sqw([[1, 0, 0], [0, 1, 0], [2, 1, 0]]), (1.0,))) as dyn:
        assert len(ctx.made) == 1 and ctx.made[0] == dyn.scratch_bytes


def test_plan_of_many_vectors_is_made_quickly(ctx):
    """200,000 vectors: 50 ms of sorting before, about 3 of counting."""
    from trj_analysis_b200 import engine
    rng = np.random.default_rng(1)
    w = sqw(rng.integers(-40, 41, (200000, 3)))
    best = float("inf")
    for _ in range(3):
        t = time.perf_counter()
        with closing(engine.DynPlan(ctx, 1, 64, 1, 2, w, (1.0,))):
            torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    assert best < 0.030


@pytest.mark.parametrize("which", ["shuffled", "far_apart", "one", "none", "negative", "two_far"])
def test_vector_orders(ctx, which):
    """Self term and coherent term of one step against FP64 sums for vectors in any order."""
    from trj_analysis_b200 import engine
    rng = np.random.default_rng(5)
    v = {"shuffled": rng.integers(-9, 10, (333, 3)), "far_apart": rng.integers(-30000, 30001, (130, 3)),
         "one": np.array([[3, -2, 5]]), "none": np.zeros((0, 3)), "negative": -rng.integers(1, 6, (97, 3)),
         "two_far": np.array([[0, 0, 1], [2 ** 30, 0, 0], [-2 ** 30, 1, 0]])}[which].astype(np.int64)
    n, box = 700, np.array([10.0, 11.0, 12.0], np.float32)
    nb = 3
    x0 = (rng.uniform(0, 1, (n, 3)) * box).astype(np.float32)
    x1 = (rng.uniform(0, 1, (n, 3)) * box).astype(np.float32)
    pk = [torch.tensor(np.concatenate([x, np.zeros((n, 1), np.float32)], 1), device="cuda") for x in (x0, x1)]
    with closing(engine.DynPlan(ctx, 1, n, 1, 3, sqw(v, nb), (1.0,))) as dyn:
        fkt, fskt, r2t = dyn.new_totals()
        dyn.accumulate(pk[0], n, box, np.array([0], np.int32), np.array([1], np.uint8))
        dyn.accumulate(pk[1], n, box, np.array([1], np.int32), np.array([0], np.uint8))
        dyn.flush(np.array([1], np.uint8), fkt, fskt, r2t)
        ctx.check()
        fkt, fskt = fkt.cpu().numpy(), fskt.cpu().numpy()
    # phases as the kernel takes them: 32-bit fractions of the box, whole turns dropped exactly
    u = [np.rint(x.astype(np.float64) / box.astype(np.float64) % 1.0 * 2.0 ** 32).astype(np.int64) for x in (x0, x1)]

    def angles(w):
        return ((w[:, None, :] * v[None, :, :]).sum(-1) % 2 ** 32) * (2 * np.pi / 2 ** 32)
    rho = [np.exp(1j * angles(w)).sum(0) for w in u]
    fc = (rho[1] * rho[0].conj()).real
    fs = np.cos(angles(u[1] - u[0])).sum(0)
    # every term is within 2^-20 (the fast sine's absolute error), sums of n terms in runs of 64
    tol = n * 2.0 ** -20 + (n + 63) // 64 * 64 * 64 * 2.0 ** -24
    for b in range(nb):
        pick = np.arange(len(v)) % nb == b
        assert abs(fskt[1, b] - fs[pick].sum()) <= tol * max(1, pick.sum())
        size = (np.abs(rho[0]) + np.abs(rho[1]) + tol)[pick]
        assert abs(fkt[1, b] - fc[pick].sum()) <= (2 * tol * size).sum() + 1e-9
