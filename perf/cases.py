"""Performance cases: the work a user of this package has it do, through its public entry points.

Five kinds of case, each one pass of what a trajectory program repeats frame after frame:

* ``gr``      frame layout and pair histogram of one frame that is resident on the device
              (``engine.pack_frame`` + ``engine.RdfPlan.accumulate``), optionally charge-weighted;
* ``sq``      the S(Q) shell sums of one packed frame (``engine.SqPlan.accumulate``), tensor-core
              ("split") or direct ("plain") method;
* ``batch``   one fused turn over many small requests (``engine.Batch``), staged from host memory;
* ``dyn``     one frame of the multiple-origin time correlations (``engine.DynPlan``);
* ``session`` one frame of the whole path from host arrays to host results (``analysis.Session``).

Frames are face-centred-cubic lattices with Gaussian displacements and a few re-placed atoms, the
synthetic trajectories of ``frames.FCCSpec``, drawn on the device from the seed.
"""
import functools
import math

import numpy as np
import torch

from trj_analysis_b200 import engine, refsem
from trj_analysis_b200.analysis import Config, Session
from trj_analysis_b200.frames import Frame

FRACTIONS = {1: (1.0,), 2: (0.8, 0.2), 3: (0.5, 0.3, 0.2)}
CHARGES = (1.0, -0.8, 0.5)
BSC = (1.0, 0.8, 0.5)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # Smallest call: one frame of a 4,000-atom liquid out to half the box (every pair is a
        # candidate), where launches and latency count.
        dict(name="gr_4k", kind="gr", cells="10,10,10", drop=0, density=0.8, nsp=1, deltar=0.02, rc=1e9,
             charged=False),
        # Ordinary binary mixture at high radial resolution: 62,500 atoms, four cells per axis.
        dict(name="gr_62k", kind="gr", cells="25,25,25", drop=0, density=0.8, nsp=2, deltar=0.01, rc=10.0,
             charged=False),
        # The headline frame: a million atoms, three species.
        dict(name="gr_1m", kind="gr", cells="63,63,63", drop=0, density=0.8, nsp=3, deltar=0.01, rc=8.0,
             charged=False),
        # Largest frame: a 1:1:4 slab of four million atoms with vacancies (ragged counts).
        dict(name="gr_slab_4m", kind="gr", cells="63,63,252", drop=752, density=0.8, nsp=2, deltar=0.02, rc=6.0,
             charged=False),
        # Ions: the charge-weighted g_qq(r) beside the counts, an odd number of atoms.
        dict(name="gr_ions_256k", kind="gr", cells="40,40,40", drop=37, density=0.8, nsp=3, deltar=0.01, rc=8.0,
             charged=True),
        # S(Q) of the headline frame, tensor-core method: every vector below Q = 3, axis vectors above.
        dict(name="sq_split_1m", kind="sq", cells="63,63,63", drop=0, density=0.8, nsp=3, kset="full+axes",
             qmax=10.0, qmin=3.0, method="split"),
        # S(Q) of the binary mixture: dense shells on the tensor cores, 200 sampled vectors per shell above.
        dict(name="sq_split_62k", kind="sq", cells="25,25,25", drop=0, density=0.8, nsp=2, kset="full+sampled",
             qmax=15.0, qmin=5.0, method="split"),
        # S(Q) of a small request by the direct sum, the reference's vector set.
        dict(name="sq_plain_16k", kind="sq", cells="16,16,16", drop=5, density=0.7, nsp=2, kset="ref", qmax=12.0,
             qmin=3.0, method="plain"),
        # One serving turn: 64 small requests packed into one launch sequence.
        dict(name="batch_64", kind="batch", requests=64, n_lo=1000, n_hi=16384, pick=3),
        # Dynamics: F(Q,t), Fs(Q,t) and the displacements over ten time origins, steady state.
        dict(name="dyn_62k", kind="dyn", cells="25,25,25", drop=0, density=0.8, nsp=2, nbuffer=10,
             qw="1.0,2.0,4.0,7.0"),
        # Whole call, small: host frame in, counts and S(Q) sums out, default (reference) vector set.
        dict(name="session_4k", kind="session", cells="10,10,10", drop=0, density=0.8, nsp=1, deltar=0.02, rc=0.0,
             kset="ref", qmax=10.0, qmin=3.0, method="split"),
        # Whole call, the headline frame from host memory to host results.
        dict(name="session_1m", kind="session", cells="63,63,63", drop=0, density=0.8, nsp=3, deltar=0.01, rc=8.0,
             kset="full+axes", qmax=10.0, qmin=3.0, method="split"),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_cells(rng, n):
    """FCC cells per axis of about n atoms: cubic, or a slab elongated along z."""
    if rng.random() < 0.35:
        ratio = rng.choice((2, 4))
        c = max(2, round((n / (4.0 * ratio)) ** (1.0 / 3.0)))
        return (c, c, ratio * c)
    c = max(3, round((n / 4.0) ** (1.0 / 3.0)))
    return (c, c, c)


def _draw_frame(rng, lo, hi):
    cells = _draw_cells(rng, _log_uniform(rng, lo, hi))
    sites = 4 * cells[0] * cells[1] * cells[2]
    return dict(cells=",".join(str(c) for c in cells), drop=rng.randrange(0, max(2, sites // 50)),
                density=round(_log_uniform(rng, 0.5, 1.0), 3), nsp=rng.randint(1, 3))


def _edges(case):
    a = (4.0 / case["density"]) ** (1.0 / 3.0)
    return [int(c) * a for c in case["cells"].split(",")]


def draw(rng):
    kind = rng.choice(("gr", "gr", "gr", "sq", "sq", "sq", "batch", "dyn", "session"))
    if kind == "gr":
        case = dict(kind="gr", **_draw_frame(rng, 1e3, 2e6))
        n, half = _atoms(case), min(_edges(case)) / 2.0
        # half the box for small frames (as the reference does by default), a cutoff above
        rc = 1e9 if n <= 2e4 and rng.random() < 0.5 else min(half, rng.uniform(2.5, 9.0))
        if n * case["density"] * min(rc, half) ** 3 > 5e8:
            rc = (5e8 / (n * case["density"])) ** (1.0 / 3.0)
        return dict(case, deltar=rng.choice((0.01, 0.02, 0.05)), rc=round(rc, 3),
                    charged=n <= 3e5 and rng.random() < 0.3)
    if kind == "sq":
        method = rng.choice(("split", "split", "plain"))
        if method == "plain":
            return dict(kind="sq", **_draw_frame(rng, 1e3, 1e5), kset="ref", qmax=round(rng.uniform(8.0, 14.0), 2),
                        qmin=round(rng.uniform(2.0, 4.0), 2), method=method)
        case = dict(kind="sq", **_draw_frame(rng, 4e3, 5e5), kset=rng.choice(("full+axes", "full+sampled", "ref")),
                    qmax=round(rng.uniform(8.0, 14.0), 2), method=method)
        if case["kset"] == "full+sampled" and _atoms(case) > 8e4:
            case["kset"] = "full+axes"  # sampling every shell of a large box takes the host seconds
        # at most ~2e11 atom-vector terms: vectors ~ V qmin^3 / (12 pi^2)
        n, v = _atoms(case), math.prod(_edges(case))
        qtop = (2e11 / n * 12.0 * math.pi ** 2 / v) ** (1.0 / 3.0)
        return dict(case, qmin=round(min(rng.uniform(2.0, 5.0), qtop), 2))
    if kind == "batch":
        return dict(kind="batch", requests=rng.randint(8, 64), n_lo=1000, n_hi=rng.choice((4096, 8192, 16384)),
                    pick=rng.randrange(1000))
    if kind == "dyn":
        shells = sorted(rng.uniform(0.8, 6.0) for _ in range(rng.randint(1, 4)))
        return dict(kind="dyn", **_draw_frame(rng, 1e3, 5e4), nbuffer=rng.randint(2, 10),
                    qw=",".join("%.2f" % q for q in shells))
    case = dict(kind="session", **_draw_frame(rng, 1e3, 2e5))
    half = min(_edges(case)) / 2.0
    return dict(case, deltar=rng.choice((0.01, 0.02)), rc=round(min(half, rng.uniform(4.0, 8.0)), 3),
                kset=rng.choice(("ref", "full+axes")), qmax=round(rng.uniform(8.0, 12.0), 2),
                qmin=round(rng.uniform(2.0, 3.0), 2), method=rng.choice(("split", "plain")))


# ---------------------------------------------------------------------------
# frames
# ---------------------------------------------------------------------------

def _atoms(case):
    c = [int(x) for x in case["cells"].split(",")]
    return 4 * c[0] * c[1] * c[2] - case["drop"]


def _box(case):
    return np.array(_edges(case), np.float64).astype(np.float32)


@functools.lru_cache(maxsize=None)
def _context():
    return engine.Context(0)


def _rng(seed, tag):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + tag) % (1 << 62))
    return g


def _species(case, g):
    """Species ids in a shuffled order with the mixture's exact counts."""
    n, fr = _atoms(case), FRACTIONS[case["nsp"]]
    counts = [int(f * n + 0.5) for f in fr]
    counts[-1] = n - sum(counts[:-1])
    ids = torch.repeat_interleave(torch.arange(case["nsp"], dtype=torch.int32, device="cuda"),
                                  torch.tensor(counts, device="cuda"))
    return ids[torch.randperm(n, generator=g, device="cuda")].contiguous(), counts


def _positions(case, g, sigma=0.1, replaced=0.02):
    """Raw coordinates (not folded): lattice sites with Gaussian displacements, some atoms re-placed."""
    cells = [int(c) for c in case["cells"].split(",")]
    a = (4.0 / case["density"]) ** (1.0 / 3.0)
    dev = "cuda"
    grid = torch.stack(torch.meshgrid(*[torch.arange(c, device=dev, dtype=torch.float64) for c in cells],
                                      indexing="ij"), dim=-1).reshape(-1, 1, 3)
    basis = torch.tensor([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]], device=dev, dtype=torch.float64)
    x = ((grid + basis) * a).reshape(-1, 3)
    if case["drop"]:
        keep = torch.randperm(x.shape[0], generator=g, device=dev)[case["drop"]:].sort().values
        x = x[keep]
    x = x + torch.randn(x.shape, generator=g, device=dev, dtype=torch.float64) * (sigma * a)
    m = int(round(replaced * x.shape[0]))
    if m:
        box = torch.tensor(_box(case).astype(np.float64), device=dev)
        where = torch.randperm(x.shape[0], generator=g, device=dev)[:m]
        x[where] = torch.rand((m, 3), generator=g, device=dev, dtype=torch.float64) * box
    return x.to(torch.float32).contiguous()


def _frame(case, seed):
    g = _rng(seed, 1)
    sp, counts = _species(case, g)
    return _positions(case, g), sp, counts, g


@functools.lru_cache(maxsize=32)
def _kset(kset, edges, qmax, qmin):
    return refsem.make_kset(kset, np.array(edges, np.float32), qmax, qmin)


def _case_kset(case):
    return _kset(case["kset"], tuple(float(v) for v in _box(case)), case["qmax"], case["qmin"])


def _pack(ctx, xyz, sp, nsp, box, charges=None):
    n = xyz.shape[0]
    packed = torch.empty((n, 4), dtype=torch.float32, device="cuda")
    counts = torch.zeros(nsp, dtype=torch.int64, device="cuda")
    engine.pack_frame(ctx, xyz, sp, nsp, box, packed, counts)
    return packed, counts


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def _prepare_gr(case, seed):
    ctx, box, nsp = _context(), _box(case), case["nsp"]
    xyz, sp, _, g = _frame(case, seed)
    n = xyz.shape[0]
    plan = engine.RdfPlan(ctx, nsp, case["deltar"], case["rc"], box, n)
    st = dict(kind="gr", ctx=ctx, xyz=xyz, sp=sp, nsp=nsp, box=box, n=n, plan=plan, hist=plan.new_hist(),
              packed=torch.empty((n, 4), dtype=torch.float32, device="cuda"),
              counts=torch.zeros(nsp, dtype=torch.int64, device="cuda"), q=None, qpacked=None, gqq=None)
    if case["charged"]:
        per = torch.tensor(CHARGES, dtype=torch.float32, device="cuda")
        st["q"] = per[sp.long()] + 0.05 * torch.randn(n, generator=g, device="cuda")
        st["qpacked"] = torch.empty(n, dtype=torch.float32, device="cuda")
        st["gqq"] = plan.new_gqq()
    return st


def _run_gr(st):
    # a frame's own histogram: the accumulators start from zero
    st["hist"].zero_()
    if st["gqq"] is None:
        engine.pack_frame(st["ctx"], st["xyz"], st["sp"], st["nsp"], st["box"], st["packed"], st["counts"])
        st["plan"].accumulate(st["packed"], st["n"], st["box"], st["hist"])
        return {"hist": st["hist"], "counts": st["counts"]}
    st["gqq"].zero_()
    engine.pack_frame(st["ctx"], st["xyz"], st["sp"], st["nsp"], st["box"], st["packed"], st["counts"],
                      charges=st["q"], qpacked=st["qpacked"])
    st["plan"].accumulate(st["packed"], st["n"], st["box"], st["hist"], qpacked=st["qpacked"], gqq=st["gqq"])
    return {"hist": st["hist"], "counts": st["counts"], "gqq": st["gqq"]}


def _prepare_sq(case, seed):
    ctx, box, nsp = _context(), _box(case), case["nsp"]
    xyz, sp, counts, _ = _frame(case, seed)
    packed, _ = _pack(ctx, xyz, sp, nsp, box)
    plan = engine.SqPlan(ctx, nsp, _case_kset(case), counts)
    return dict(kind="sq", box=box, n=xyz.shape[0], packed=packed, plan=plan, out=plan.new_out(),
                method=engine.METHODS[case["method"]])


def _run_sq(st):
    st["out"].zero_()
    st["plan"].accumulate(st["packed"], st["n"], st["box"], st["out"], st["method"])
    return {"s": st["out"]}


def _requests(case):
    """Sizes, shapes and mixtures of a turn's requests (the serving workload's distributions)."""
    rng = np.random.default_rng([case["pick"], 0x5e7])
    out = []
    for _ in range(case["requests"]):
        n = math.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))
        rho = round(math.exp(rng.uniform(math.log(0.5), math.log(1.0))), 3)
        nsp = int(rng.integers(1, 4))
        if rng.random() < 0.5:
            c = max(1, int((n / 8.0) ** (1 / 3)))
            cells = (c, c, 2 * c)
        else:
            c = max(1, int((n / 4.0) ** (1 / 3)))
            cells = (c, c, c)
        r = dict(cells=",".join(str(v) for v in cells), drop=int(rng.integers(0, 4)), density=rho, nsp=nsp,
                 kset="ref", qmax=12.0, qmin=3.0)
        r["rc"] = min(min(_edges(r)) / 2.0, 8.0)
        out.append(r)
    return out


def _prepare_batch(case, seed):
    ctx = _context()
    reqs, items, off = _requests(case), [], 0
    hist_words = sq_words = 0
    for k, r in enumerate(reqs):
        box, nsp, n = _box(r), r["nsp"], _atoms(r)
        g = _rng(seed, 100 + k)
        sp, counts = _species(r, g)
        it = dict(box=box, n=n, nsp=nsp, off=off, xyz=_positions(r, g).cpu().numpy(), sp=sp.cpu().numpy(),
                  rdf=engine.RdfPlan(ctx, nsp, 0.02, r["rc"], box, n), sq=engine.SqPlan(ctx, nsp, _case_kset(r), counts))
        it["h0"], it["s0"] = hist_words, sq_words
        hist_words += it["rdf"].nit * it["rdf"].lsmax
        sq_words += it["sq"].kset.nbins * it["sq"].nit
        off += n
        items.append(it)
    hist = torch.zeros(hist_words, dtype=torch.int64, device="cuda")
    s = torch.zeros(sq_words, dtype=torch.float64, device="cuda")
    for it in items:  # each request's accumulators: its part of the turn's result arrays
        it["hist"] = hist[it["h0"]:it["h0"] + it["rdf"].nit * it["rdf"].lsmax].view(it["rdf"].nit, it["rdf"].lsmax)
        it["out"] = s[it["s0"]:it["s0"] + it["sq"].kset.nbins * it["sq"].nit].view(it["sq"].kset.nbins, it["sq"].nit)
    return dict(kind="batch", batch=engine.Batch(ctx, len(items), off), items=items, hist=hist, s=s, turn=0)


def _run_batch(st):
    b, buf = st["batch"], st["turn"] & 1
    st["turn"] += 1
    st["hist"].zero_()
    st["s"].zero_()
    b.begin(buf)
    for it in st["items"]:
        b.stage(buf, it["off"], it["xyz"], it["sp"])
        b.add(buf, it["rdf"], it["sq"], it["off"], it["n"], it["box"], it["hist"], it["out"])
    b.launch(buf)
    b.mark(buf)
    return {"hist": st["hist"], "s": st["s"]}


DYN_STEP = 0.2  # displacement per frame and axis


def _dyn_frames(case, seed):
    """Origin frames of every buffer and the current frame of a random walk, on the device."""
    g = _rng(seed, 7)
    sp, counts = _species(case, g)
    x, out = _positions(case, g, replaced=0.0).double(), []
    for _ in range(case["nbuffer"] + 1):
        out.append(x.to(torch.float32).contiguous())
        x = x + DYN_STEP * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64)
    return out, sp, counts


@functools.lru_cache(maxsize=32)
def _sqw(edges, qw):
    box = np.array(edges, np.float32)
    shells = [float(q) for q in qw.split(",")]
    return refsem.sqw_kset(box, shells, refsem.sq_init_params(box, max(shells), max(shells)).dq)


def _case_sqw(case):
    return _sqw(tuple(float(v) for v in _box(case)), case["qw"])


def _prepare_dyn(case, seed):
    ctx, box, nsp, nbuf = _context(), _box(case), case["nsp"], case["nbuffer"]
    frames, sp, _ = _dyn_frames(case, seed)
    n = frames[0].shape[0]
    plan = engine.DynPlan(ctx, nsp, n, nbuf, nbuf + 10, _case_sqw(case), BSC[:nsp])
    packed = [_pack(ctx, f, sp, nsp, box)[0] for f in frames]
    fkt, fskt, r2t = plan.new_totals()
    # every buffer's origin is seen: buffer b starts at frame b and is at lag f - b in frame f
    for f in range(nbuf):
        lags = np.array([f - b for b in range(nbuf)], np.int32)
        plan.accumulate(packed[f], n, box, np.maximum(lags, -1), (lags == 0).astype(np.uint8))
    plan.flush(np.ones(nbuf, np.uint8), fkt, fskt, r2t)
    return dict(kind="dyn", plan=plan, packed=packed[nbuf], n=n, box=box, fkt=fkt, fskt=fskt, r2t=r2t,
                lags=np.array([nbuf - b for b in range(nbuf)], np.int32), none=np.zeros(nbuf, np.uint8),
                all=np.ones(nbuf, np.uint8))


def _run_dyn(st):
    for t in (st["fkt"], st["fskt"], st["r2t"]):
        t.zero_()
    st["plan"].accumulate(st["packed"], st["n"], st["box"], st["lags"], st["none"])
    st["plan"].flush(st["all"], st["fkt"], st["fskt"], st["r2t"])
    return {"fkt": st["fkt"], "fskt": st["fskt"], "r2t": st["r2t"]}


def _prepare_session(case, seed):
    nsp = case["nsp"]
    xyz, sp, _, _ = _frame(case, seed)
    # type ids in order of first appearance, so that species numbers do not depend on the shuffle
    order = [int(v) for v in sorted(range(nsp), key=lambda s: int((sp == s).nonzero()[0]))]
    types = torch.empty_like(sp)
    for t, s in enumerate(order):
        types[sp == s] = t + 1
    frame = Frame(xyz=xyz.cpu().numpy(), types=types.cpu().numpy(), box=_box(case))
    cfg = Config(nsp=nsp, sp_types_selected=list(range(1, nsp + 1)), deltar=case["deltar"], rcrdf=case["rc"],
                 qmax=case["qmax"], qmin=case["qmin"], bsc=BSC[:nsp], kset=case["kset"], method=case["method"])
    s = Session(cfg, ctx=_context(), n_max=frame.n)
    s.add_frame(frame)  # the trajectory's first frame makes the plans
    return dict(kind="session", session=s, frame=frame)


def _run_session(st):
    s = st["session"]
    # this frame's own results: the accumulators start from zero
    s.hist.zero_()
    s.sq_out.zero_()
    s.add_frame(st["frame"])
    return {"hist": s.rdf_transfer(), "s": s.sq_transfer_gpu_cpu()}


_PREPARE = dict(gr=_prepare_gr, sq=_prepare_sq, batch=_prepare_batch, dyn=_prepare_dyn, session=_prepare_session)
_RUN = dict(gr=_run_gr, sq=_run_sq, batch=_run_batch, dyn=_run_dyn, session=_run_session)


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------

def _gr_work(case):
    n, e, nsp = _atoms(case), _edges(case), case["nsp"]
    rc = min(case["rc"], min(e) / 2.0) if case["rc"] > 0 else min(e) / 2.0
    pairs = 0.5 * n * (n / math.prod(e)) * 4.0 / 3.0 * math.pi * rc ** 3
    bins = nsp * (nsp + 1) // 2 * (int(rc / case["deltar"]) + 2)
    charged = case.get("charged", False)
    # per pair: three differences, squared distance (5), root, division, rounding; the charge product
    return {"bytes": (20.0 if charged else 16.0) * n + 8.0 * bins, "flops": (13.0 if charged else 11.0) * pairs}


def _sq_work(case):
    n, ks, nsp = _atoms(case), _case_kset(case), case["nsp"]
    # a complex multiply-add per atom and vector
    return {"bytes": 16.0 * n + 8.0 * ks.nbins * nsp * (nsp + 1) / 2, "flops": 8.0 * n * ks.nvec}


def work(case):
    kind = case["kind"]
    if kind == "gr":
        return _gr_work(case)
    if kind == "sq":
        return _sq_work(case)
    if kind == "dyn":
        n, nvec, nb = _atoms(case), _case_sqw(case).nvec, case["nbuffer"]
        # per atom and vector: rho (complex term) once, a cosine term per origin
        return {"bytes": n * (16.0 + nb * 44.0), "flops": (8.0 + 4.0 * nb) * n * nvec}
    if kind == "batch":
        parts = [(_gr_work(dict(r, deltar=0.02)), _sq_work(r)) for r in _requests(case)]
    else:
        parts = [(_gr_work(case), _sq_work(case))]
    return {"bytes": sum(a["bytes"] + b["bytes"] for a, b in parts),
            "flops": sum(a["flops"] + b["flops"] for a, b in parts)}


# ---------------------------------------------------------------------------
# exact values (plain torch, 64 bits)
# ---------------------------------------------------------------------------

def exact(case, seed):
    """What ``run`` returns, in 64 bits.  Pair counts (and the charge products binned with them) are
    defined by the FP32 binning of each pair, so they have no 64-bit value."""
    kind = case["kind"]
    if kind == "gr":
        return None
    if kind == "sq":
        xyz, sp, _, _ = _frame(case, seed)
        return {"s": _exact_sq(xyz, sp, case["nsp"], _box(case), _case_kset(case))}
    if kind == "session":
        xyz, sp, _, _ = _frame(case, seed)
        order = sorted(range(case["nsp"]), key=lambda s: int((sp == s).nonzero()[0]))
        rank = torch.empty(case["nsp"], dtype=torch.int64, device="cuda")
        for t, s in enumerate(order):
            rank[s] = t
        out = _exact_sq(xyz, rank[sp.long()], case["nsp"], _box(case), _case_kset(case))
        return {"hist": None, "s": out.cpu().numpy()}
    if kind == "batch":
        parts = []
        for k, r in enumerate(_requests(case)):
            g = _rng(seed, 100 + k)
            sp, _ = _species(r, g)
            parts.append(_exact_sq(_positions(r, g), sp, r["nsp"], _box(r), _case_kset(r)).reshape(-1))
        return {"hist": None, "s": torch.cat(parts)}
    return _exact_dyn(case, seed)


def _turns(xyz, box):
    return torch.remainder(xyz.double() / torch.tensor(np.asarray(box, np.float64), device="cuda"), 1.0)


def _direct_rho(u, vec, weights=None, limit=1 << 26):
    """sum_j w_j exp(2 pi i n.u_j) for every row n of vec, in blocks."""
    v = vec.double()
    re = torch.zeros(v.shape[0], dtype=torch.float64, device="cuda")
    im = torch.zeros_like(re)
    step = max(1, limit // max(1, v.shape[0]))
    for j in range(0, u.shape[0], step):
        ph = v @ u[j:j + step].T
        ph = (ph - torch.round(ph)) * (2.0 * math.pi)
        c, s = torch.cos(ph), torch.sin(ph)
        if weights is not None:
            w = weights[j:j + step]
            c, s = c * w, s * w
        re += c.sum(1)
        im += s.sum(1)
    return torch.complex(re, im)


def _tiled_rho(u, vec, block=2048):
    """The same for a compact set: products of the three axes' factors, one matrix product per block."""
    lo, hi = vec.min(0).values, vec.max(0).values
    pairs, inv = torch.unique(vec[:, :2], dim=0, return_inverse=True)
    nz = int(hi[2] - lo[2]) + 1
    acc = torch.zeros((pairs.shape[0], nz), dtype=torch.complex128, device="cuda")

    def factor(col, n0, count):
        ph = col[None, :] * (torch.arange(count, device="cuda", dtype=torch.float64) + n0)[:, None]
        ph = (ph - torch.round(ph)) * (2.0 * math.pi)
        return torch.complex(torch.cos(ph), torch.sin(ph))

    for j in range(0, u.shape[0], block):
        b = u[j:j + block]
        fx = factor(b[:, 0], int(lo[0]), int(hi[0] - lo[0]) + 1)
        fy = factor(b[:, 1], int(lo[1]), int(hi[1] - lo[1]) + 1)
        fz = factor(b[:, 2], int(lo[2]), nz)
        acc += (fx[pairs[:, 0] - lo[0]] * fy[pairs[:, 1] - lo[1]]) @ fz.T
    return acc[inv, vec[:, 2] - lo[2]]


def _exact_sq(xyz, sp, nsp, box, ks):
    u = _turns(xyz, box)
    vec = torch.from_numpy(ks.vectors.astype(np.int64)).cuda()
    dense = torch.from_numpy(ks.dense.astype(bool)).cuda()
    rho = torch.zeros((nsp, vec.shape[0]), dtype=torch.complex128, device="cuda")
    tiled = int(dense.sum()) > 20000
    for a in range(nsp):
        ua = u[sp == a]
        if tiled:
            rho[a, dense] = _tiled_rho(ua, vec[dense])
            if bool((~dense).any()):
                rho[a, ~dense] = _direct_rho(ua, vec[~dense])
        else:
            rho[a] = _direct_rho(ua, vec)
    w = torch.from_numpy(ks.weights.astype(np.float64)).cuda()
    bins = torch.from_numpy(ks.bins.astype(np.int64)).cuda()
    out = torch.zeros((ks.nbins, nsp * (nsp + 1) // 2), dtype=torch.float64, device="cuda")
    row = 0
    for a in range(nsp):
        for b in range(a, nsp):
            out[:, row].index_add_(0, bins, w * (rho[a] * rho[b].conj()).real)
            row += 1
    return out


def _exact_dyn(case, seed):
    frames, sp, _ = _dyn_frames(case, seed)
    box, nbuf, sqw = _box(case), case["nbuffer"], _case_sqw(case)
    vec = torch.from_numpy(sqw.vectors.astype(np.int64)).cuda()
    bins = torch.from_numpy(sqw.bins.astype(np.int64)).cuda()
    wt = torch.tensor(BSC[:case["nsp"]], dtype=torch.float64, device="cuda")[sp.long()]
    L = torch.tensor(box.astype(np.float64), device="cuda")
    nbins, ndyn = sqw.qw.size, nbuf + 10
    fkt = torch.zeros((ndyn, nbins), dtype=torch.float64, device="cuda")
    fskt = torch.zeros_like(fkt)
    r2t = torch.zeros(ndyn, dtype=torch.float64, device="cuda")
    u = [_turns(f, box) for f in frames]
    now = u[nbuf]
    rho_t = _direct_rho(now, vec, wt)
    for b in range(nbuf):
        lag = nbuf - b
        rho_0 = _direct_rho(u[b], vec, wt)
        fkt[lag].index_add_(0, bins, (rho_0 * rho_t.conj()).real)
        fskt[lag].index_add_(0, bins, _direct_rho(now - u[b], vec).real)
        # unwrapped frame by frame, as the walk went
        d = torch.zeros_like(now)
        for f in range(b, nbuf):
            step = u[f + 1] - u[f]
            d += step - torch.round(step)
        r2t[lag] = ((d * L) ** 2).sum() / now.shape[0]
    return {"fkt": fkt, "fskt": fskt, "r2t": r2t}
