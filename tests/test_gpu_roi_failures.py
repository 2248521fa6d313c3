"""Bounded exits of the ROI searches: a team's wait that runs out and a phase cap (ogr_debug_limits, as for the
whole-lattice search) come back as errors, in single searches and in passes with and without windows.  A pass that
stops so leaves the congestion state of exactly the paths in its store, and the next job routes as on a fresh router."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from test_gpu_failures import assert_state_matches_store

NX, NY, NZ = 70, 50, 6


def requests(n, seed):
    rng = np.random.default_rng(seed)
    out = []
    while len(out) < n:
        x0, x1 = rng.integers(0, NX, size=2)
        y0, y1 = rng.integers(0, NY, size=2)
        if 5 <= abs(int(x1) - int(x0)) + abs(int(y1) - int(y0)) < 100:
            out.append((f"N{len(out)}", int(y0) * NX + int(x0), int(y1) * NX + int(x1)))
    return out


REQS = requests(60, 9)


def router(window_slots):
    from orthoroute_gb300 import Lattice
    from orthoroute_gb300.router import PathFinderConfig, PathFinderRouter
    R = PathFinderRouter(PathFinderConfig(max_iterations=3), mode="persistent", full_engine="grid",
                         window_slots=window_slots)
    R.initialize_lattice(Lattice(NX, NY, NZ))
    return R


def paths(R):
    return {k: list(v) for k, v in R.route_multiple_nets(REQS)["paths"].items()}


@pytest.mark.parametrize("window_slots", [0, 16])
@pytest.mark.parametrize("limit,status", [((1, 0), "grid barrier timed out"), ((0, 3), "iteration limit reached")])
def test_pass_of_roi_nets_stops_with_its_state_consistent(window_slots, limit, status):
    from orthoroute_gb300 import _lib
    want = paths(router(window_slots))
    R = router(window_slots)
    try:
        _lib.debug_limits(*limit)
        with pytest.raises(RuntimeError, match=status):
            R.route_multiple_nets(REQS)
    finally:
        _lib.debug_limits(0, 0)
    assert_state_matches_store(R)
    assert paths(R) == want


@pytest.mark.parametrize("window_slots", [0, 16])
def test_later_pass_stops_with_its_state_consistent(window_slots):
    """The search that fails has its old path ripped up, as have the other members of its window."""
    from orthoroute_gb300 import _lib
    from orthoroute_gb300.device import PathStore, route_pass
    from test_gpu_windows import _table
    R = router(window_slots)
    R.store = PathStore(R.g, len(REQS), window_slots=window_slots)
    R.s.total_cost.copy_(R.g.base_costs)
    R.s.live_static.copy_(R.g.base_costs)
    R.ops.sync_rcost()
    table = _table(R.lattice, [(s, d) for _, s, d in REQS], R.g.device)
    run = lambda: route_pass(R.ops, R.store, table, np.arange(len(REQS), dtype=np.int32), fallback_quota=5,
                             max_roi_nodes=50_000, owner_weight=25.0, path_weight=25.0, history_weight=5.0, pres_fac=1.0,
                             live=True, windows=window_slots > 0)
    run()
    assert assert_state_matches_store(R) > 40
    try:
        _lib.debug_limits(0, 40)          # the short nets still get through
        with pytest.raises(RuntimeError, match="iteration limit reached"):
            run()
    finally:
        _lib.debug_limits(0, 0)
    left = assert_state_matches_store(R)
    assert 0 < left < len(REQS)
    run()
    assert assert_state_matches_store(R) > 40


def test_single_searches_stop_and_go_on():
    from orthoroute_gb300 import _lib
    from test_gpu_kernels import make
    import torch
    g, s, ops, ref = make(NX, NY, NZ)
    s.total_cost.copy_(g.base_costs)
    net = ops.net_args(0, 5 * NX + 5, 30 * NX + 40, penalty=False)
    roi = ops.extract_roi(net)
    seeds, targets = [(5 * NX + 5, 0.0), (5 * NX + 5 + ref.plane, 0.5)], [(30 * NX + 40, 0.0)]
    calls = [lambda: ops.find_path(net), lambda: ops.find_path_given_roi(net.src, net.dst, s.total_cost, roi),
             lambda: ops.find_path_multi(seeds, targets, s.total_cost, roi)]
    want = [c() for c in calls]
    assert all(want)
    for limit, status in (((1, 0), "grid barrier timed out"), ((0, 3), "iteration limit reached")):
        for c in calls:
            try:
                _lib.debug_limits(*limit)
                with pytest.raises(RuntimeError, match=status):
                    c()
            finally:
                _lib.debug_limits(0, 0)
        assert [c() for c in calls] == want
