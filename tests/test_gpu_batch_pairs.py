"""Pair histograms of a fused turn over frames of every sort and image form, against the single-request calls."""
import numpy as np
import pytest

from trj_analysis_b200 import frames

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from trj_analysis_b200 import engine
    c = engine.Context(0)
    yield c
    c.close()


def lattice(cells, nsp, seed, centred=False, density=0.8):
    spec = frames.FCCSpec(cells=cells, density=density, sigma=0.1, fractions=(1.0,) * nsp, replace_frac=0.05, seed=seed)
    fr = spec.frame(0)
    x = fr.xyz
    if centred:
        x = (x - fr.box * np.floor(x / fr.box + 0.5)).astype(np.float32)
    return x, (fr.types - 1).astype(np.int32), fr.box


def test_fused_pairs_match_single_requests(ctx):
    import torch
    from trj_analysis_b200 import engine
    reqs = [
        # (frame, nsp, deltar, cutoff, floor bins, edge statistics)
        (lattice((9, 9, 9), 3, 1), 3, 0.02, 2.5, None, True),
        (lattice((9, 9, 9), 3, 2), 3, 0.02, 2.5, None, False),
        (lattice((6, 6, 6), 2, 3, centred=True), 2, 0.01, 1e9, None, True),
        (lattice((4, 4, 16), 2, 4, centred=True), 2, 0.02, 1e9, None, True),
        (lattice((8, 8, 8), 1, 5), 1, 0.0, 3.0, 150, True),          # floor bins
        (lattice((6, 6, 6), 12, 6), 12, 0.05, 1e9, None, True),     # row table
        (lattice((12, 12, 12), 2, 7), 2, 0.01, 0.5, None, True),    # many more cells than groups
        (lattice((2, 2, 2), 1, 8), 1, 0.05, 1e9, None, True),
    ]
    one = (np.array([[1.0, 2.0, 3.0]], np.float32), np.zeros(1, np.int32), np.full(3, 9.0, np.float32))
    reqs.append((one, 1, 0.05, 2.0, None, True))
    total = sum(r[0][0].shape[0] for r in reqs)
    batch = engine.Batch(ctx, len(reqs), total, hist_words=8192)
    st, off = [], 0
    for frame, nsp, deltar, rc, nbins, edges in reqs:
        xyz, sp, box = frame
        n = xyz.shape[0]
        plan = engine.RdfPlan(ctx, nsp, deltar, rc, box, n, floor_bins=nbins)
        st.append(dict(n=n, nsp=nsp, box=box, xyz=xyz, sp=sp, plan=plan, off=off, hist=plan.new_hist(),
                       edge=torch.zeros(4, dtype=torch.int64, device="cuda") if edges else None))
        off += n
    for turn in range(2):  # both staging buffers, counts add up
        batch.begin(turn)
        for e in st:
            batch.stage(turn, e["off"], e["xyz"], e["sp"])
            batch.add(turn, e["plan"], None, e["off"], e["n"], e["box"], e["hist"], None, e["edge"])
        batch.launch(turn)
        batch.mark(turn)
    ctx.check()
    for e in st:
        stage = engine.FrameStage(ctx, e["n"], e["nsp"])
        stage.upload_and_pack(e["xyz"], e["sp"], e["box"])
        hist, edge = e["plan"].new_hist(), torch.zeros(4, dtype=torch.int64, device="cuda")
        e["plan"].accumulate(stage.packed, e["n"], e["box"], hist, edge)
        ctx.check()
        assert torch.equal(e["hist"], 2 * hist)
        if e["edge"] is not None:
            assert torch.equal(e["edge"][:3], 2 * edge[:3])
        e["plan"].close()
    batch.close()
