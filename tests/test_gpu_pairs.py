"""The pair kernel's paths, each bit-exact against the oracle: image forms, group sizes, row layouts."""
import numpy as np
import pytest
import torch

from oracle import orc
from trj_analysis_b200 import frames, refsem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from trj_analysis_b200 import engine
    c = engine.Context(0)
    yield c
    c.close()


def lattice(cells, nsp=2, sigma=0.1, seed=1, density=0.8):
    spec = frames.FCCSpec(cells=cells, density=density, sigma=sigma, fractions=(1.0,) * nsp, replace_frac=0.02, seed=seed)
    fr = spec.frame(0)
    return fr.xyz, fr.types - 1, fr.box


def centred(*a, **k):  # coordinates in [-L/2, L/2), as centred boxes are stored
    x, t, b = lattice(*a, **k)
    return (x - b * np.floor(x / b + 0.5)).astype(np.float32), t, b


def both_signs(*a, **k):  # coordinates all over (-L, L)
    x, t, b = lattice(*a, **k)
    rng = np.random.default_rng(3)
    return (x - b * rng.integers(0, 2, x.shape)).astype(np.float32), t, b


def clumps(n, box, nsp=3, seed=4):  # groups of far more than 32 atoms beside empty ones
    rng = np.random.default_rng(seed)
    b = np.full(3, box, np.float32)
    c = rng.uniform(0, box, (6, 3))
    x = c[rng.integers(0, 6, n)] + rng.normal(0, 0.35, (n, 3))
    return (x % b).astype(np.float32), rng.integers(0, nsp, n).astype(np.int32), b


def crystal(cells, nsp=2):  # many pairs exactly on bin edges
    return lattice(cells, nsp=nsp, sigma=0.0, density=0.5)


CASES = [
    ("split_shift", lattice((9, 9, 9)), 2, 0.02, 3.0),
    ("split_sparse", lattice((12, 12, 12)), 2, 0.01, 0.95),      # cells merged up to about 28 atoms
    ("split_2_cells_apart", lattice((7, 8, 15)), 2, 0.02, 3.6),  # three cells on one axis
    ("split_centred", centred((9, 9, 9)), 2, 0.02, 3.0),
    ("split_both_signs", both_signs((9, 9, 9)), 2, 0.02, 3.0),
    ("whole_half_box", lattice((6, 6, 6), nsp=3), 3, 0.01, 1e9),
    ("whole_centred", centred((6, 6, 6), nsp=3), 3, 0.01, 1e9),
    ("whole_both_signs", both_signs((6, 6, 6), nsp=3), 3, 0.01, 1e9),
    ("mixed_axes_centred", centred((4, 4, 16)), 2, 0.02, 1e9),   # z split, x and y not
    ("clumps_split", clumps(3001, 12.0), 3, 0.02, 2.0),
    ("clumps_whole", clumps(1999, 6.0), 3, 0.02, 1e9),
    ("crystal_edges", crystal((6, 6, 6)), 2, 0.1, 1e9),
    ("row_table", lattice((6, 6, 6), nsp=12), 12, 0.0125, 1e9),  # 144 square rows do not fit
    ("one_group", lattice((2, 2, 2), nsp=1), 1, 0.05, 1e9),
]


@pytest.mark.parametrize("name,data,nsp,deltar,rc", CASES, ids=[c[0] for c in CASES])
def test_pair_paths_bit_exact(ctx, name, data, nsp, deltar, rc):
    from trj_analysis_b200 import engine
    xyz, sp, box = data
    n = xyz.shape[0]
    pos, sps, _ = orc.layout(xyz, sp, box, nsp)
    p = refsem.rdf_params(nsp, deltar, rc, box)
    h_o, e_o = orc.rdf_counts(pos, sps, box, p.side2, p.deltar, p.lsmax, nsp, cells=False)
    stage = engine.FrameStage(ctx, n, nsp)
    plan = engine.RdfPlan(ctx, nsp, deltar, rc, box, n)
    stage.upload_and_pack(xyz, sp, box)
    edge = torch.zeros(4, dtype=torch.int64, device="cuda")
    with_edges, without = plan.new_hist(), plan.new_hist()
    plan.accumulate(stage.packed, n, box, with_edges, edge)
    plan.accumulate(stage.packed, n, box, without)
    q = torch.linspace(-1.0, 1.0, n, device="cuda", dtype=torch.float32)
    charged, gqq = plan.new_hist(), plan.new_gqq()
    plan.accumulate(stage.packed, n, box, charged, qpacked=q, gqq=gqq)
    ctx.check()
    assert np.array_equal(with_edges.cpu().numpy().astype(np.uint64), h_o)
    assert np.array_equal(edge.cpu().numpy()[:3].astype(np.uint64), e_o)
    assert np.array_equal(without.cpu().numpy().astype(np.uint64), h_o)
    assert np.array_equal(charged.cpu().numpy().astype(np.uint64), h_o)
    plan.close()
