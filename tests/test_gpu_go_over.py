"""Searches that meet a value ticks of 2^-30 cannot hold late, in the middle or at once, and go on in doubles from there:
paths and heap statistics equal to the oracle's (whole numbers), whichever way the value comes in (a label past 2^22, an
arc's cost below 2^-7 or above 2^22, a penalty, a seed's cost), on the whole lattice and on ROIs, with few CTAs and many.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle.dijkstra import find_path_multisource, find_path_roi_c

from test_gpu_kernels import make

NX, NY, NZ = 70, 60, 6


def place(ref, N):
    ids = np.arange(N)
    return (ids % ref.plane) % ref.nx, (ids % ref.plane) // ref.nx


def inputs(kind, g, ref, rng):
    """(costs, penalty or None).  Sources lie on the left, targets on the right: `x` says when the value is met."""
    E, N = g.E, g.N
    src = ref.edge_src()
    x, _ = place(ref, N)
    costs = (0.125 + rng.integers(0, 4, size=E) * 0.125).astype(np.float32)
    pen = None
    if kind == "labels":             # pass 2^22 half way, and again and again round off
        costs = (np.float32(9.0e4) * (1 + rng.random(E))).astype(np.float32)
        costs[rng.random(E) < 0.3] = np.float32(0.3)
    elif kind == "labels at the end":
        costs[x[src] > 60] = np.float32(2.0e6) + rng.random(int((x[src] > 60).sum())).astype(np.float32) * 1.0e6
    elif kind == "huge arc":         # 2^22 and more on a few arcs, up to what float32 labels overflow by
        hit = (x[src] > 25) & (rng.random(E) < 0.15)
        costs[hit] = np.float32(5.0e6)
        costs[hit & (rng.random(E) < 0.3)] = np.float32(3.0e38)
    elif kind == "small arc":
        costs[(x[src] > 30) & (rng.random(E) < 0.05)] = np.float32(0.0031)
    elif kind == "penalty":
        pen = np.where((x > 35) & (rng.random(N) < 0.05), 0.0017, 0.0).astype(np.float32)
    elif kind == "infinite penalty":
        pen = np.where((x > 35) & (rng.random(N) < 0.02), np.inf, 0.0).astype(np.float32)
    elif kind == "huge penalty":
        # (not so huge that an arc's cost is lost in the sum: among labels that do not grow along an arc the heap's
        # order of pops, which the statistics count, is not that of (label, id))
        pen = np.where((x > 20) & (rng.random(N) < 0.1), 3.0e7, 0.5).astype(np.float32)
    costs[rng.random(E) < 0.03] = np.float32("inf")
    return costs, pen


KINDS = ["labels", "labels at the end", "huge arc", "small arc", "penalty", "infinite penalty",
         "huge penalty"]


@pytest.mark.parametrize("share", [1, 3, 0])
@pytest.mark.parametrize("kind", KINDS)
def test_searches_that_go_over_to_doubles(kind, share):
    from orthoroute_gb300.autotune import full_grid
    g, s, ops, ref = make(NX, NY, NZ)
    rng = np.random.default_rng(len(kind) + share)
    costs, pen = inputs(kind, g, ref, rng)
    dev = torch.from_numpy(costs).to(g.device)
    s.total_cost.copy_(dev)
    if pen is not None:
        s.node_history.copy_(torch.from_numpy(pen))
    ident = np.arange(g.N, dtype=np.int32)
    before, limit = full_grid(0)
    try:
        full_grid(share or limit)
        for k in range(4):
            src = int(rng.integers(0, NY)) * NX + int(rng.integers(0, 8))
            dst = int(rng.integers(0, NY)) * NX + int(rng.integers(NX - 4, NX))
            if k == 3:
                src, dst = dst, src      # the value is met at once
            for stats in (True, False):
                st = {}
                want = find_path_roi_c(ref.indptr, ref.indices, src, dst, costs, ident, ident, node_penalty=pen, stats=st)
                # (the penalty of a state is history x weight: weight 1, no owners)
                net = ops.net_args(7, src, dst, full_graph=True, hist_pen=1.0, penalty=pen is not None)
                ops.stats.zero_()
                assert ops.find_path(net, engine="grid") == want, (src, dst)
                assert ops.stats.cpu().tolist()[:2] == [st["scanned"], st["settled"]]
                roi = np.flatnonzero(rng.random(g.N) < 0.9).astype(np.int32)
                roi = np.union1d(roi, [src, dst]).astype(np.int32)
                if stats:
                    rng.shuffle(roi)
                g2r = np.full(g.N, -1, dtype=np.int32)
                g2r[roi] = np.arange(roi.size, dtype=np.int32)
                rp, st = None if pen is None else pen[roi], {}
                want = find_path_roi_c(ref.indptr, ref.indices, src, dst, costs, roi, g2r, node_penalty=rp, stats=st)
                ops.stats.zero_()
                assert ops.find_path_given_roi(src, dst, dev, roi, rp) == want, (src, dst)
                assert ops.stats.cpu().tolist()[:2] == [st["scanned"], st["settled"]]
    finally:
        full_grid(before)


@pytest.mark.parametrize("share", [1, 0])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("seed_costs", [(0.0, 0.25, 1.5), (0.0, 7.5, 2.25), (0.1, 6.0e6, 1e-9)])
def test_multi_source_searches_that_go_over(kind, share, seed_costs):
    """Seeds that wait beside the wave (some enter late, some are still waiting when it goes over)."""
    from orthoroute_gb300.autotune import full_grid
    g, s, ops, ref = make(NX, NY, NZ)
    rng = np.random.default_rng(len(kind) * 3 + share)
    costs, pen = inputs(kind, g, ref, rng)
    dev = torch.from_numpy(costs).to(g.device)
    s.total_cost.copy_(dev)
    if pen is not None:
        s.node_history.copy_(torch.from_numpy(pen))
    ident = np.arange(g.N, dtype=np.int32)
    net = ops.net_args(7, 0, 1, full_graph=True, hist_pen=1.0, penalty=pen is not None)
    x, _ = place(ref, g.N)
    left, right = np.flatnonzero(x < 8), np.flatnonzero(x > 60)
    before, limit = full_grid(0)
    try:
        full_grid(share or limit)
        for _ in range(2):
            ids = [int(rng.choice(left)), int(rng.choice(right)), int(rng.choice(left))]
            if len(set(ids)) < 3:
                continue
            seeds = list(zip(ids, seed_costs))
            tg = [int(v) for v in rng.choice(right, size=3, replace=False)] + [ids[2]]
            targets = [(t, float(c)) for t, c in zip(tg, (0.0, 0.5, 1.0e3, 5.0e6))]
            want = find_path_multisource(ref.indptr, ref.indices, seeds, targets, costs, ident, ident, node_penalty=pen,
                                         plane=ref.plane)
            want = tuple(want) if want else None
            assert ops.find_path_full_multi(seeds, targets, net) == want
            assert ops.find_path_multi(seeds, targets, dev, ident, pen) == want
    finally:
        full_grid(before)


def test_unreachable_target_past_an_overflow():
    """Every way to the target overflows float32: no path, found by the frontier running empty, not by the phase cap."""
    g, s, ops, ref = make(NX, NY, NZ)
    x, _ = place(ref, g.N)
    src_of = ref.edge_src()
    costs = np.full(g.E, 0.25, dtype=np.float32)
    costs[(x[src_of] <= 40) & (x[ref.indices] > 40)] = np.float32(3.4e38)
    pen = np.where(x > 40, 3.0e38, 0.0).astype(np.float32)
    dev = torch.from_numpy(costs).to(g.device)
    s.total_cost.copy_(dev)
    s.node_history.copy_(torch.from_numpy(pen))
    ident = np.arange(g.N, dtype=np.int32)
    src, dst = 10 * NX + 5, 20 * NX + 66
    st = {}
    want = find_path_roi_c(ref.indptr, ref.indices, src, dst, costs, ident, ident, node_penalty=pen, stats=st)
    assert want is None
    for call in (lambda: ops.find_path(ops.net_args(7, src, dst, full_graph=True, hist_pen=1.0), engine="grid"),
                 lambda: ops.find_path_given_roi(src, dst, dev, ident, pen)):
        ops.stats.zero_()
        assert call() is None
        assert ops.stats.cpu().tolist()[:2] == [st["scanned"], st["settled"]]
