"""Memory admission of the request loop: what counts against the budget is what the plans hold, and a request whose
plans turn out too large waits, with the results of the others and its own unchanged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def workload():
    from trj_analysis_b200.serve import serving_workload
    return serving_workload(10, seed=4, n_lo=1500, n_hi=12000)


def serve(reqs, hook=None, **kw):
    from trj_analysis_b200.serve import Server
    srv = Server(slots=4, n_max=1 << 14, method="plain", **kw)
    res = {r.rid: r for r in srv.run(reqs, realtime=False, on_turn=hook)}
    return srv, res


@pytest.mark.parametrize("fuse", [0, 1 << 14])
def test_budget_counts_what_plans_hold(workload, fuse):
    seen = []

    def hook(srv, turn):
        seen.append((srv.in_use, srv.alloc.bytes_live - (srv.batch.device_bytes if srv.batch is not None else 0)))
    _, free = serve(workload, hook, fuse_max_atoms=fuse)
    used, live = max(seen)
    assert used > 0
    # the allocator also holds the plans' small tables and the layout's scratch; outputs are PyTorch's own
    assert 0.9 * live - (1 << 20) <= used <= 1.1 * live + (1 << 20)

    seen.clear()
    srv, tight = serve(workload, hook, fuse_max_atoms=fuse, hbm_budget=used // 3)
    assert srv.admission_waits > 0 and srv.in_use == 0 and not srv._sizes
    assert max(u for u, _ in seen) < used
    assert set(tight) == set(free)
    for rid, r in free.items():
        assert np.array_equal(r.hist, tight[rid].hist) and np.array_equal(r.sq_sums, tight[rid].sq_sums)
