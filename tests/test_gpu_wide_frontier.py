"""A frontier of more than 2^20 entries in one CTA: the count of places asked for in a phase shares a word with the count
of entries carried, and must not run into it."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_more_than_a_million_entries_in_one_cta():
    """Every node is a seed, at 0 where x + y is even and at 10 elsewhere, every arc costs 4.  The seeds at 0 settle at
    once; the others on the three connected layers (1.15 M, none of them local to the CTA yet) wait for the lateral hop
    of the inner layers (label 4), those of the outer one for the via below (label 8)."""
    from orthoroute_gb300 import Lattice, _lib
    from orthoroute_gb300.autotune import full_grid
    from orthoroute_gb300.device import DeviceGraph, DeviceState, Ops
    lat = Lattice(1100, 700, 4)
    g = DeviceGraph(lat)
    ops = Ops(g, DeviceState(g))
    ids = torch.arange(g.N, dtype=torch.int32, device=g.device)
    odd = ((ids % lat.plane) % lat.nx + (ids % lat.plane) // lat.nx) % 2
    connected = int((odd[: 3 * lat.plane] == 1).sum())
    assert connected > 1 << 20
    seed_cost = odd.double() * 10.0
    x, y = 501, 300
    targets = torch.tensor([lat.node_idx(x, y, 0)], dtype=torch.int32, device=g.device)
    tcost = torch.zeros(1, dtype=torch.float64, device=g.device)
    costs = torch.full((g.E,), 4.0, dtype=torch.float32, device=g.device)
    ws = ops.multi_workspace()
    n = C.c_int32(0)
    cg = g.cgraph()
    before, limit = full_grid(0)
    try:
        for share in (1, 2, limit):
            full_grid(share)
            ops.stats.zero_()
            p = lambda t: t.data_ptr()
            rc = ops.lib.ogr_find_path_multi(C.byref(cg), p(costs), p(ids), g.N, None, p(ids), p(seed_cost), g.N,
                                             p(targets), p(tcost), 1, p(ws), ops.multi_ws_bytes, p(ops.path_buf),
                                             int(ops.path_buf.numel()), C.byref(n), p(ops.stats), ops._sp())
            assert _lib.check(rc, "ogr_find_path_multi") == _lib.OGR_OK
            # of equal candidates the relaxer with the least (label, id): layer 1 before layer 2, x - 1 before x + 1
            want = [lat.node_idx(x - 1, y, 1), lat.node_idx(x, y, 1), lat.node_idx(x, y, 0)]
            assert ops.path_buf[: n.value].tolist() == want
            rows = g.indptr.cpu().numpy().astype(np.int64)
            t = int(targets[0])
            arcs, pops = ops.stats.cpu().tolist()[:2]
            assert pops == g.N and arcs == g.E - (rows[t + 1] - rows[t])
    finally:
        full_grid(before)
