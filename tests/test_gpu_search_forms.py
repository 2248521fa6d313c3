"""The form of the search follows the lattice's longest row: boards whose average row is far below it run in the form
that holds it, and a graph that does not tell (or tells too little) is searched by the next form, equal to the oracle
all the same (paths and heap statistics: whole numbers)."""
import ctypes as C

import numpy as np
import pytest
import torch

from orthoroute_gb300 import Lattice


def spans(nz, k):
    return [(a, b) for a, b in Lattice(2, 2, nz).via_pairs() if b - a <= k]


# lattice, longest row; each one's average over the inner layers is below the next smaller form's limit
BOARDS = {
    "10 layers, spans to 4": ((60, 50, 10), dict(allowed_via_spans=spans(10, 4)), 10),
    "8 layers, spans to 3, wrong way": ((40, 37, 8), dict(allowed_via_spans=spans(8, 3), wrong_way_cost_multiplier=3.0), 10),
    "12 layers, checkerboard": ((40, 33, 12), dict(min_via_center_spacing=0.5), 12),
    "6 layers, checkerboard": ((50, 41, 6), dict(min_via_center_spacing=0.5), 6),
    "4 layers": ((30, 20, 4), {}, 4),
    "20 layers": ((20, 21, 20), {}, 4),
    "24 layers, all spans": ((13, 11, 24), dict(allow_any_layer_via=True), 24),
    "narrow": ((1, 40, 6), {}, 6),
}


@pytest.mark.parametrize("name", BOARDS)
def test_longest_row_is_known(name):
    from oracle.lattice import LatticeSpec, build_csr
    dims, kw, row = BOARDS[name]
    lat = Lattice(*dims, **kw)
    ref = build_csr(LatticeSpec(*dims, **kw))
    assert lat.max_row() == int(np.diff(ref.indptr).max()) == row


def forms_left(reset=True):
    """ROI searches that left their kernel's form, and all of them."""
    from orthoroute_gb300 import _lib
    out = np.zeros(16, dtype=np.int64)
    _lib.check(_lib.load().ogr_search_profile(out.ctypes.data, int(reset)), "ogr_search_profile")
    return int(out[15]), int(out[9])


def search_all(g, s, ops, ref, costs, rng, n=3):
    """Whole-lattice, ROI and multi-source searches against the oracle; the ROI searches made."""
    from oracle.dijkstra import find_path_multisource, find_path_roi_c
    ident = np.arange(g.N, dtype=np.int32)
    dev = torch.from_numpy(costs).to(g.device)
    s.total_cost.copy_(dev)
    for _ in range(n):
        src, dst = (int(v) for v in rng.choice(ref.plane, size=2, replace=False))
        st = {}
        want = find_path_roi_c(ref.indptr, ref.indices, src, dst, costs, ident, ident, stats=st)
        ops.stats.zero_()
        assert ops.find_path(ops.net_args(7, src, dst, full_graph=True, penalty=False), engine="grid") == want
        assert ops.stats.cpu().tolist()[:2] == [st["scanned"], st["settled"]]
        ops.stats.zero_()
        assert ops.find_path_given_roi(src, dst, dev, ident) == want
        assert ops.stats.cpu().tolist()[:2] == [st["scanned"], st["settled"]]
        # (seed costs in whole ticks of 2^-30: others are a reason of their own to go over to doubles)
        seeds = [(int(v), float(c) / 64) for v, c in zip(rng.choice(g.N, size=3, replace=False), rng.integers(0, 64, size=3))]
        targets = [(int(v), float(c)) for v, c in zip(rng.choice(g.N, size=4, replace=False), rng.random(4))]
        want = find_path_multisource(ref.indptr, ref.indices, seeds, targets, costs, ident, ident, plane=ref.plane)
        want = tuple(want) if want else None
        assert ops.find_path_multi(seeds, targets, dev, ident) == want
        assert ops.find_path_full_multi(seeds, targets, ops.net_args(0, 0, 1, full_graph=True, penalty=False)) == want
    return 2 * n


@pytest.mark.gpu
@pytest.mark.parametrize("name", BOARDS)
@pytest.mark.parametrize("told", ["exactly", "not", "too little", "too much"])
def test_form_of_the_longest_row(name, told):
    from oracle.lattice import LatticeSpec, build_csr
    from orthoroute_gb300.device import DeviceGraph, DeviceState, Ops
    dims, kw, row = BOARDS[name]
    g = DeviceGraph(Lattice(*dims, **kw))
    s = DeviceState(g)
    ops = Ops(g, s)
    ref = build_csr(LatticeSpec(*dims, **kw))
    np.testing.assert_array_equal(g.indices.cpu().numpy(), ref.indices)
    assert g.max_row == row
    g.max_row = {"exactly": row, "not": 0, "too little": 3, "too much": 1000}[told]
    rng = np.random.default_rng(len(name))
    ticks = (0.125 + rng.integers(0, 3, size=g.E) * 0.125).astype(np.float32)
    ticks[rng.random(g.E) < 0.05] = np.float32("inf")
    forms_left()
    made = search_all(g, s, ops, ref, ticks, rng)
    left, all_ = forms_left()
    assert all_ == made
    if told in ("exactly", "too much"):
        assert left == 0
    if told == "too little":
        assert left == (made if row > 4 else 0)
    small = (0.001 + rng.random(g.E) * 0.004).astype(np.float32)     # off the tick grid: in doubles
    made = search_all(g, s, ops, ref, small, rng, n=1)
    assert forms_left() == (made, made)
