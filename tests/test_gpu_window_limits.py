"""Passes of one path store under changing ROI limits: the windows' search slots, sized for the store's limit, serve any
smaller one, and every pass equals the one without windows (whole numbers: equal or wrong)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from test_gpu_windows import _table


def _passes(window_slots, limits, seed, scribble=False):
    from orthoroute_gb300 import Lattice
    from orthoroute_gb300.device import DeviceGraph, DeviceState, Ops, PathStore, route_pass
    lat = Lattice(60, 50, 6)
    g = DeviceGraph(lat)
    s = DeviceState(g)
    ops = Ops(g, s)
    rng = np.random.default_rng(seed)
    costs = (0.4 + rng.random(g.E) * 0.05).astype(np.float32)
    costs[rng.random(g.E) < 0.2] = np.float32("inf")
    s.total_cost.copy_(torch.from_numpy(costs))
    s.live_static.copy_(torch.from_numpy(costs))
    nets = []
    while len(nets) < 80:
        a, b = (int(v) for v in rng.integers(0, lat.plane, size=2))
        if 4 <= abs(a % lat.nx - b % lat.nx) + abs(a // lat.nx - b // lat.nx) <= 25:
            nets.append((a, b))
    store = PathStore(g, len(nets), max_roi_nodes=max(limits), window_slots=window_slots)
    if scribble and window_slots:
        # whatever lies behind a slot's node map (4 bytes a node) is scratch
        w = store.win_ws.view(window_slots, store.win_slot_bytes)[:, (4 * g.N + 255) // 256 * 256:]
        w.copy_(torch.tensor([7, 0, 0, 0, 8, 0, 0, 0], dtype=torch.uint8).repeat(w.shape[1] // 8))
    table = _table(lat, nets, g.device)
    out = []
    for limit in limits:
        status, st = route_pass(ops, store, table, np.arange(len(nets), dtype=np.int32), fallback_quota=5,
                                max_roi_nodes=limit, owner_weight=25.0, path_weight=25.0, history_weight=5.0,
                                pres_fac=1.0, live=True, windows=window_slots > 0)
        L = store.length.cpu().numpy()
        P = store.path.cpu().numpy()
        out.append((status.tolist(), st.tolist(), [P[n, :L[n]].tolist() for n in range(len(nets))]))
    return out, {k: getattr(s, k).cpu().numpy() for k in ("present", "total_cost", "path_node_use", "owner_count")}


@pytest.mark.parametrize("limits", [(50_000, 3_000, 50_000), (3_000, 700, 3_000, 18_000), (1_000, 50_000, 900, 50_000)])
@pytest.mark.parametrize("scribble", [False, True])
def test_windows_under_changing_roi_limits(limits, scribble):
    want, state = _passes(0, limits, 5)
    got, wstate = _passes(16, limits, 5, scribble)
    assert any(0 in status for status, _, _ in want)
    for k, (a, b) in enumerate(zip(want, got)):
        assert a == b, (k, limits[k])
    for k in state:
        np.testing.assert_array_equal(state[k], wstate[k], err_msg=k)
