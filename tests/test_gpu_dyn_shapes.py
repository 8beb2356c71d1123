"""Launch shapes of the time-correlation sums (slots, runs, parts) against direct FP64 sums.

Bounds per term: cos/sin.approx 2^-20.5, the phase's two FP32 roundings 2 pi 2^-24, and the FP32 sum of 64 terms
32.5 * 2^-24 (partial sums of at most 64): together below 3.1e-6 per atom for a cosine sum, and per component
of rho.
"""
import numpy as np
import pytest

from trj_analysis_b200 import refsem

pytestmark = pytest.mark.gpu

EPS = 3.1e-6


@pytest.fixture(scope="module")
def ctx():
    from trj_analysis_b200 import engine
    c = engine.Context(0)
    yield c
    c.close()


def vectors(kind, nvec, rng):
    if kind == "scattered":  # no two vectors share a component: the unshared form
        return np.stack([rng.permutation(nvec) - nvec // 2 for _ in range(3)], axis=1).astype(np.int32)
    v = rng.integers(0, 6, (nvec, 3)).astype(np.int32)
    v[:, 1 if kind == "rows_y" else 2] = np.sort(rng.integers(0, 2, nvec))
    return v


@pytest.mark.parametrize("n,nvec,nbuf,kind", [
    (1, 1, 2, "rows_y"), (63, 3, 2, "rows_z"), (65, 129, 3, "scattered"), (1025, 640, 2, "rows_y"),
    (2500, 1029, 4, "scattered"), (4097, 33, 5, "rows_z"),
])
def test_dyn_sums(ctx, n, nvec, nbuf, kind):
    import torch
    from trj_analysis_b200 import engine
    rng = np.random.default_rng([n, nvec, nbuf])
    box = np.array([9.0, 10.5, 12.25], np.float32)
    vec, bins, bsc = vectors(kind, nvec, rng), rng.integers(0, 3, nvec).astype(np.int32), (1.0, 0.6)
    sqw = refsem.SqwSet(qw=np.ones(3, np.float32), dq=0.1, vectors=vec, bins=bins, nw=np.bincount(bins, minlength=3))
    sp = np.sort(rng.integers(0, 2, n)).astype(np.int32)
    frames = []
    for _ in range(nbuf + 1):
        f = np.zeros((n, 4), np.float32)
        f[:, :3] = rng.uniform(0, 1, (n, 3)) * box
        f[:, 3] = sp.view(np.float32)
        frames.append(f)
    plan = engine.DynPlan(ctx, 2, n, nbuf, nbuf + 2, sqw, bsc)
    fkt, fskt, r2t = plan.new_totals()
    dev = [torch.from_numpy(f).cuda() for f in frames]
    for f in range(nbuf + 1):  # buffer b starts at frame b
        lags = np.array([f - b for b in range(nbuf)], np.int32)
        plan.accumulate(dev[f], n, box, np.maximum(lags, -1), (lags == 0).astype(np.uint8))
    plan.flush(np.ones(nbuf, np.uint8), fkt, fskt, r2t)
    ctx.check()
    u = [f[:, :3].astype(np.float64) / box.astype(np.float64) for f in frames]
    w = np.asarray(bsc)[sp]
    rho = [(w * np.exp(2j * np.pi * (vec @ x.T))).sum(1) for x in u]
    want_f, want_s = np.zeros((nbuf + 2, 3)), np.zeros((nbuf + 2, 3))
    tol_f, tol_s = np.zeros((nbuf + 2, 3)), np.zeros((nbuf + 2, 3))
    d = 1.5 * EPS * n
    for b in range(nbuf):
        for f in range(b, nbuf + 1):
            np.add.at(want_f[f - b], bins, (rho[b] * rho[f].conj()).real)
            np.add.at(tol_f[f - b], bins, d * (np.abs(rho[b]) + np.abs(rho[f])) + d * d)
            np.add.at(want_s[f - b], bins, np.cos(2 * np.pi * (vec @ (u[f] - u[b]).T)).sum(1))
            np.add.at(tol_s[f - b], bins, EPS * n)
    assert np.all(np.abs(fkt.cpu().numpy() - want_f) <= tol_f)
    assert np.all(np.abs(fskt.cpu().numpy() - want_s) <= tol_s)
    plan.close()
