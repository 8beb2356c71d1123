"""The direct sum's launch shapes (vectors and run lanes per block, parts of a slice) against the FP64 oracle.

Bound per atom and vector, from the operations: a run of 64 terms is summed in FP32 with partial sums of at
most 64, so its rounding is below (1 + 2 + .. + 64) 2^-24 = 32.5 * 2^-24 per term; a term itself (table entry,
two polynomials, rotation: at most seven roundings of values <= 1) is within 4 * 2^-24 of its exact value, and
the 32-bit phase within pi 2^-32 (|nx| + |ny| + |nz|) < 2^-24.  Together below 38 * 2^-24 = 2.3e-6 per atom.
"""
import numpy as np
import pytest

from oracle import orc
from trj_analysis_b200 import refsem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from trj_analysis_b200 import engine
    c = engine.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("counts,nvec", [
    ((1,), 1), ((63,), 31), ((65, 0), 65), ((64, 129), 511), ((4097,), 1), ((2049, 700, 1), 513),
    ((9000, 333), 257), ((3001,), 1025), ((70001,), 40), ((20011, 5), 2100),
])
def test_direct_sum_shapes(ctx, counts, nvec):
    import torch
    from trj_analysis_b200 import engine
    rng = np.random.default_rng([sum(counts), nvec])
    n, nsp = sum(counts), len(counts)
    box = np.array([11.0, 12.5, 14.25], np.float32)
    pos = (rng.uniform(0, 1, (n, 3)) * box).astype(np.float32)
    packed = np.zeros((n, 4), np.float32)
    packed[:, :3] = pos
    packed[:, 3] = np.repeat(np.arange(nsp, dtype=np.int32), counts).view(np.float32)
    vec = rng.integers(-40, 41, (nvec, 3)).astype(np.int32)
    bins = rng.integers(0, 5, nvec).astype(np.int32)
    ks = refsem.KSet(mode="test", dq=1.0, nqmax=4, vectors=vec, bins=bins, weights=np.ones(nvec),
                     dense=np.zeros(nvec, np.uint8), nq=np.bincount(bins, minlength=5).astype(np.int64))
    plan = engine.SqPlan(ctx, nsp, ks, counts)
    dev = torch.from_numpy(packed).cuda()
    out = plan.new_out()
    plan.accumulate(dev, n, box, out, engine.METHODS["plain"])
    rho = plan.rho().cpu().numpy()
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    groups = plan.rho_groups(dev, n, box, off).cpu().numpy()
    ctx.check()
    want = orc.rho_fp64(pos, off, box, vec)
    bound = 2.3e-6 * np.maximum(1, np.asarray(counts))[:, None]
    assert np.all(np.abs(rho - want) <= bound)
    assert np.all(np.abs(groups - want) <= bound)
    got = out.cpu().numpy()
    row = 0
    for a in range(nsp):
        for b in range(a, nsp):
            s = np.bincount(bins, weights=(rho[a] * rho[b].conj()).real, minlength=5)
            np.testing.assert_allclose(got[:, row], s, rtol=1e-12, atol=1e-12 * n * n)
            row += 1
    plan.close()
