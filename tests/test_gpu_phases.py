"""The phase-settled search (csrc/phases.cuh) at the edges of its forms, against the oracle's heap search, paths and
heap statistics alike (whole numbers: equal or wrong).

* rows of up to 4, 8, 16 and 32 arcs have forms of their own, longer rows the general one;
* costs, penalties and seed costs that 2^-30 ticks cannot hold (below 2^-7, 2^22 and more, labels above 2^22) are
  searched in doubles;
* one CTA (every entry local), three CTAs and every SM (surplus entries dealt out).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle.dijkstra import find_path_multisource, find_path_roi_c

from test_gpu_kernels import make

ROWS = {                      # longest row: lattice
    4: ((40, 33, 4), {}), 6: ((31, 30, 6), {}), 8: ((33, 27, 8), {}), 10: ((23, 19, 8), {"wrong_way_cost_multiplier": 3.0}),
    16: ((17, 13, 16), {}), 22: ((13, 11, 22), {"allow_any_layer_via": True}),
    40: ((9, 8, 40), {"allow_any_layer_via": True}),
}


def values(kind, E, rng):
    if kind == "ticks":
        return (0.12 + rng.random(E) * 0.05).astype(np.float32)
    if kind == "ties":        # many equal float32 keys, some arcs blocked
        c = (0.125 + rng.integers(0, 3, size=E) * 0.125).astype(np.float32)
        c[rng.random(E) < 0.05] = np.float32("inf")
        return c
    if kind == "small":       # below 2^-7: off the tick grid
        return (0.001 + rng.random(E) * 0.004).astype(np.float32)
    if kind == "some small":  # a few off-grid costs, met on the way
        c = (0.12 + rng.random(E) * 0.05).astype(np.float32)
        c[rng.random(E) < 0.002] = np.float32(0.0031)
        return c
    c = (3.0e5 + rng.random(E) * 3.0e5).astype(np.float32)      # "large": labels pass 2^22
    c[rng.random(E) < 0.01] = np.float32(5.0e6)
    return c


def check(g, s, ops, ref, costs, rng, pen_scale, n=3):
    s.total_cost.copy_(torch.from_numpy(costs))
    ident = np.arange(g.N, dtype=np.int32)
    pen = None
    if pen_scale:
        hist = np.where(rng.random(g.N) < 0.1, rng.random(g.N) * pen_scale, 0.0).astype(np.float32)
        s.node_history.copy_(torch.from_numpy(hist))
        pen = (hist * np.float32(5.0)).astype(np.float32)
    for _ in range(n):
        src, dst = (int(v) for v in rng.integers(0, ref.plane, size=2))
        st = {}
        want = find_path_roi_c(ref.indptr, ref.indices, src, dst, costs, ident, ident, node_penalty=pen, stats=st)
        ops.stats.zero_()
        got = ops.find_path(ops.net_args(7, src, dst, full_graph=True, penalty=pen is not None), engine="grid")
        assert got == want, (src, dst)
        if src != dst:
            assert ops.stats.cpu().tolist()[:2] == [st["scanned"], st["settled"]], (src, dst)


@pytest.mark.parametrize("row", sorted(ROWS))
@pytest.mark.parametrize("kind", ["ticks", "ties", "small", "some small", "large"])
def test_forms_match_oracle(row, kind):
    dims, kw = ROWS[row]
    g, s, ops, ref = make(*dims, **kw)
    assert int(np.diff(ref.indptr).max()) <= row
    rng = np.random.default_rng(row * 10 + len(kind))
    # penalties on the tick grid, then (off the grid) around 2^-7
    for pen_scale in (0.0, 2.0, 0.002):
        check(g, s, ops, ref, values(kind, g.E, rng), rng, pen_scale)


@pytest.mark.parametrize("ctas", [1, 2, 3, 0])
@pytest.mark.parametrize("kind", ["ties", "some small"])
def test_team_sizes_match_oracle(ctas, kind):
    """A frontier larger than its CTA's places and uneven shares; 0 = every SM."""
    from orthoroute_gb300.autotune import full_grid
    g, s, ops, ref = make(260, 210, 4)
    rng = np.random.default_rng(17)
    before, limit = full_grid(0)
    try:
        full_grid(ctas or limit)
        check(g, s, ops, ref, values(kind, g.E, rng), rng, 1.0, n=2)
    finally:
        full_grid(before)


@pytest.mark.parametrize("seed_costs", [(0.0, 0.25, 1.5), (0.1, 0.30000001, 1e-9), (0.0, 5.0e6, 0.5)])
@pytest.mark.parametrize("row", [6, 22, 40])
def test_seed_costs_match_oracle(seed_costs, row):
    dims, kw = ROWS[row]
    g, s, ops, ref = make(*dims, **kw)
    rng = np.random.default_rng(5)
    costs = values("ties", g.E, rng)
    s.total_cost.copy_(torch.from_numpy(costs))
    ident = np.arange(g.N, dtype=np.int32)
    net = ops.net_args(0, 0, 1, full_graph=True, penalty=False)
    for _ in range(4):
        seeds = [(int(n), c) for n, c in zip(rng.choice(g.N, size=3, replace=False), seed_costs)]
        targets = [(int(n), float(c)) for n, c in zip(rng.choice(g.N, size=4, replace=False), rng.random(4))]
        want = find_path_multisource(ref.indptr, ref.indices, seeds, targets, costs, ident, ident, plane=ref.plane)
        assert ops.find_path_full_multi(seeds, targets, net) == (tuple(want) if want else None)


@pytest.mark.parametrize("row", sorted(ROWS))
@pytest.mark.parametrize("kind", ["ties", "some small", "large"])
def test_roi_forms_match_oracle(row, kind):
    """The ROI search (a team of CTAs) in every form, on shuffled partial ROIs whose order is the tie order."""
    dims, kw = ROWS[row]
    g, s, ops, ref = make(*dims, **kw)
    rng = np.random.default_rng(row + 100)
    costs = values(kind, g.E, rng)
    dev = torch.from_numpy(costs).to(g.device)
    for case in range(4):
        roi = np.flatnonzero(rng.random(g.N) < 0.85).astype(np.int32)
        if case % 2:
            rng.shuffle(roi)
        g2r = np.full(g.N, -1, dtype=np.int32)
        g2r[roi] = np.arange(roi.size, dtype=np.int32)
        pen = (rng.integers(0, 3, size=roi.size) * 0.5).astype(np.float32) if case >= 2 else None
        src, dst = (int(v) for v in rng.choice(roi, size=2, replace=False))
        st = {}
        want = find_path_roi_c(ref.indptr, ref.indices, src, dst, costs, roi, g2r, node_penalty=pen, stats=st)
        ops.stats.zero_()
        assert ops.find_path_given_roi(src, dst, dev, roi, pen) == want
        assert ops.stats.cpu().tolist()[:3] == [st["scanned"], st["settled"], roi.size]
        seeds = [(int(n), float(c)) for n, c in zip(rng.choice(g.N, size=3, replace=False), rng.random(3))]
        targets = [(int(n), float(c)) for n, c in zip(rng.choice(g.N, size=5, replace=False), rng.random(5))]
        want = find_path_multisource(ref.indptr, ref.indices, seeds, targets, costs, roi, g2r, node_penalty=pen,
                                     plane=ref.plane)
        got = ops.find_path_multi(seeds, targets, dev, roi, pen)
        assert got == (tuple(want) if want else None)


@pytest.mark.parametrize("dims,max_nodes,depth,blocked", [
    ((150, 140, 8), 50_000, 80, False),      # the box fits and the search stays in it
    ((33, 200, 6), 50_000, 80, True),        # one axis cut off by the lattice's edge, blocked arcs
    ((260, 250, 16), 400_000, 80, False),    # the box is cut to fit and the search leaves it
    ((64, 64, 4), 900, 80, False),           # truncated, terminals swapped in
    ((90, 70, 6), 50_000, 3, False),         # the waves do not meet
    ((60, 50, 20), 50_000, 80, False),       # more than 16 layers
    ((20, 16, 36), 50_000, 80, True),        # more than 32
    ((1, 90, 6), 50_000, 80, False), ((90, 1, 6), 50_000, 80, False),
])
def test_roi_extraction_matches_oracle(dims, max_nodes, depth, blocked):
    from oracle.roi import extract_roi_bfs
    g, s, ops, ref = make(*dims)
    rng = np.random.default_rng(dims[0])
    mask = None
    if blocked:
        mask = rng.random(g.E) < 0.2
        g.blocked = torch.from_numpy(mask.astype(np.uint8)).to(g.device)
    for k in range(3):
        src, dst = (int(v) for v in rng.integers(0, ref.plane, size=2))
        if k == 2:
            dst = src
        want, _ = extract_roi_bfs(ref.indptr, ref.indices, g.N, src, dst, initial_radius=depth, blocked=mask,
                                  max_nodes=max_nodes)
        net = ops.net_args(0, src, dst, max_depth=depth, halo=2, max_roi_nodes=max_nodes)
        np.testing.assert_array_equal(ops.extract_roi(net), want)


@pytest.mark.parametrize("columns", [3, 270, 300])
def test_commit_of_many_vias_matches_oracle(columns):
    """Ownership of the nodes that overlapping via hops of one column span: 15, 1350 (listed, sorted out by every
    thread) and 1500 hops (more than the list of 1365 holds)."""
    from oracle.tallies import NodeState
    g, s, ops, ref = make(302, 302, 8)
    ns = NodeState(g.N, ref.nx, ref.plane)
    at = 300 // 2
    row = ref.indices[ref.indptr[ref.plane + at * 303]:ref.indptr[ref.plane + at * 303 + 1]]
    along_x = ref.plane + at * 303 + 1 in row
    path = []
    for c in range(1, columns + 1):
        r = at * ref.nx + c if along_x else c * ref.nx + at
        zs = [1, 4, 2, 6, 3, 5]
        path += [z * ref.plane + r for z in (zs if c % 2 else zs[::-1])]
    owner = lambda: np.where(s.owner_count.cpu().numpy() == 0, -1,
                             np.where(s.owner_count.cpu().numpy() == 1, s.owner_xor.cpu().numpy(), -2))
    ops.apply_path(path, 5, +1, 1.0, live=False)
    ns.mark_owner(5, path)
    ns.mark_use(path)
    np.testing.assert_array_equal(owner(), ns.owner)
    np.testing.assert_array_equal(s.path_node_use.cpu().numpy(), ns.path_node_use.astype(np.int32))
    ops.commit_paths([np.asarray(path)], [6])
    ns.mark_owner(6, path)
    np.testing.assert_array_equal(owner(), ns.owner)
    ops.apply_path(path, 5, -1, 1.0, live=False)
    ns.clear_owner(5, path)
    np.testing.assert_array_equal(owner(), ns.owner)
