"""Direct sums over many atom groups: the groups are shared out between blocks, whatever their number and sizes.
Against FP64 sums, empty and one-atom groups included, and many small groups take no longer than a few times what two
large ones of the same atoms take.  Bound of a group's sum of m FP32 terms added in runs of 64: 64 roundings of a sum of
at most 64, 64 * 64 * 2^-24 per run, and 2^-21 per term."""
import numpy as np
import pytest
import torch

from trj_analysis_b200 import frames, refsem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup():
    from trj_analysis_b200 import engine
    fr = frames.FCCSpec(cells=(16, 16, 16), density=0.7, sigma=0.1, seed=7).frame(0)
    n = fr.n
    ctx = engine.Context(0)
    dev = np.zeros((n, 4), np.float32)
    dev[:, :3] = np.mod(fr.xyz, fr.box).astype(np.float32)
    plan = engine.SqPlan(ctx, 1, refsem.make_kset("ref", fr.box, 12.0, 3.0), np.array([n]))
    yield plan, torch.tensor(dev, device="cuda"), n, fr.box
    plan.close()
    ctx.close()


def offsets(n, sizes):
    return np.concatenate([[0], np.cumsum(sizes), [n]]).astype(np.int64)


@pytest.mark.parametrize("which", ["one", "two", "three_ragged", "sixty_four", "small_and_empty"])
def test_rho_groups(setup, which):
    plan, dev, n, box = setup
    off = {"one": np.array([0, n], np.int64), "two": offsets(n, [n // 3]), "three_ragged": offsets(n, [1, 65]),
           "sixty_four": np.linspace(0, n, 65).astype(np.int64),
           "small_and_empty": offsets(n, [0, 1, 0, 63, 64, 65, 0] * 40)}[which]
    got = plan.rho_groups(dev, n, box, off).cpu().numpy()
    x = dev[:, :3].cpu().numpy().astype(np.float64) / np.asarray(box, np.float64)
    k = np.arange(0, plan.kset.nvec, 7)
    e = np.exp(2j * np.pi * (x @ plan.kset.vectors[k].astype(np.float64).T))
    for g in range(len(off) - 1):
        m = int(off[g + 1] - off[g])
        bound = ((m + 63) // 64) * 64 * 64 * 2.0 ** -24 + m * 2.0 ** -21
        assert np.abs(got[g, k] - e[off[g]:off[g + 1]].sum(0)).max(initial=0.0) <= bound


def ms(plan, dev, n, box, off):
    best = float("inf")
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        plan.rho_groups(dev, n, box, off)
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


def test_many_groups_fill_the_gpu(setup):
    """280 us against 60 with every block summing all groups one after the other."""
    plan, dev, n, box = setup
    two, many = offsets(n, [n // 2]), np.linspace(0, n, 65).astype(np.int64)
    assert ms(plan, dev, n, box, many) < 2.5 * ms(plan, dev, n, box, two)
