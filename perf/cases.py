"""Workloads of the router, from one short net to whole jobs, for measuring it.

Each case is a call a routing program makes through the public entry points:
``DeviceGraph``, ``Ops``, ``route_pass`` and ``PathFinderRouter``.  Kinds:

* ``nets``: the solver seam.  Search a few nets one after another on a
  congested board (``Ops.find_path``); short nets take the ROI search, nets of
  125 steps or more (``whole``) the whole-lattice search.
* ``portals``: the portal-seeded seam.  Multi-source multi-sink search of one
  net, on its ROI (``extract_roi`` + ``find_path_multi``) or on the whole
  lattice (``find_path_full_multi``).
* ``costs``: the congestion update between two routing passes (EMA, layer
  tallies, arc costs, live rebase, history).
* ``lattice``: the CSR of a board's lattice.
* ``pass``: one routing pass over a list of nets, short and long mixed
  (``route_pass``): rip-up, search and commit of each in order.
* ``job``: a whole routing job on a lattice that stays resident, as the router
  runs it for a list of requests.

A congested board has straight H/V paths of other nets committed on it, so
that arcs are shared, nodes are occupied and via barrels are owned, and its
costs come from the router's own cost update.
"""
import math

import numpy as np
import torch

from orthoroute_gb300 import Lattice
from orthoroute_gb300.device import DeviceGraph, DeviceState, Ops, PathStore, route_pass
from orthoroute_gb300.multipin import seeded_multipin_nets, star_requests
from orthoroute_gb300.router import PathFinderConfig, PathFinderRouter

HIST_WEIGHT = 14.4 * 1.2     # what the router derives for boards of up to 10 signal layers


def listed():
    return [
        # the smallest call: one short net of the 100x100x6 board
        dict(name="net_short", kind="nets", nx=100, ny=100, nz=6, span=0, nets=1, lo=5, hi=80, whole=False,
             paths=150, pres=1.5),
        # a few local nets of the 600x400x12 board, ROIs near the 50,000-node limit
        dict(name="nets_local", kind="nets", nx=600, ny=400, nz=12, span=4, nets=4, lo=40, hi=124, whole=False,
             paths=1500, pres=4.0),
        # long nets of the 600x400x12 board: most of its routing time
        dict(name="nets_long", kind="nets", nx=600, ny=400, nz=12, span=4, nets=3, lo=200, hi=700, whole=True,
             paths=1500, pres=4.0),
        # a long net of a mid-size board with ragged dimensions, all via spans
        dict(name="net_ragged", kind="nets", nx=307, ny=199, nz=8, span=0, nets=2, lo=125, hi=450, whole=True,
             paths=500, pres=8.0),
        # the largest board: 1000x800x32 backplane, adjacent vias only
        dict(name="net_backplane", kind="nets", nx=1000, ny=800, nz=32, span=0, nets=1, lo=500, hi=1200, whole=True,
             paths=2000, pres=2.0),
        # a net with pad portals on every inner layer: on its ROI, and a long one on the whole lattice
        dict(name="portals_roi", kind="portals", nx=300, ny=200, nz=8, span=4, lo=30, hi=110, whole=False,
             paths=600, pres=3.0),
        dict(name="portals_long", kind="portals", nx=301, ny=203, nz=8, span=4, lo=150, hi=400, whole=True,
             paths=600, pres=3.0),
        # the congestion update of the 600x400x12 board, once per negotiation iteration
        dict(name="costs_board", kind="costs", nx=600, ny=400, nz=12, span=4, pres=3.3),
        # opening a board: its lattice on the device
        dict(name="lattice_board", kind="lattice", nx=600, ny=400, nz=12, span=4, ww=0.0),
        # a small job to its iteration cap: 100x100x6, 200 two-pin nets
        dict(name="job_small", kind="job", nx=100, ny=100, nz=6, span=0, nets=200, iters=10, pins="short"),
        # multi-pin nets in 50x50 boxes (star requests) on the large board, the first iterations of a job
        dict(name="job_multipin", kind="job", nx=600, ny=400, nz=12, span=4, nets=1000, iters=2, pins="multi"),
        # a routing pass of the 600x400x12 board: mostly long nets, 30% of them from two dense clusters
        dict(name="pass_board", kind="pass", nx=600, ny=400, nz=12, span=4, nets=64, paths=600, pres=2.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same kinds, board sizes spread over the range of the listed ones."""
    kind = rng.choice(["nets", "nets", "nets", "portals", "costs", "lattice", "job", "pass"])
    nx, ny, nz = _log(rng, 60, 640), _log(rng, 50, 420), rng.choice([4, 6, 8, 10, 12])
    span = rng.choice([0, 4])
    case = dict(kind=kind, nx=nx, ny=ny, nz=nz, span=span)
    far = nx + ny - 2
    if kind in ("nets", "portals"):
        whole = far >= 180 and rng.random() < 0.55
        lo = rng.randint(125, min(300, far * 2 // 3)) if whole else rng.randint(5, 60)
        case.update(lo=lo, hi=min(far - 10, lo + rng.randint(40, 250)) if whole else min(124, far - 10, lo + 64),
                    whole=whole, paths=max(10, nx * ny * nz // _log(rng, 1500, 6000)),
                    pres=round(math.exp(rng.uniform(0.0, 3.4)), 3))
        if kind == "nets":
            case["nets"] = rng.randint(1, 4)
    elif kind == "costs":
        case["pres"] = round(math.exp(rng.uniform(0.0, 4.0)), 3)
    elif kind == "lattice":
        case["ww"] = rng.choice([0.0, 0.0, 3.0])
    elif kind == "pass":
        case.update(nets=rng.randint(8, 64), paths=max(10, nx * ny * nz // _log(rng, 3000, 9000)),
                    pres=round(math.exp(rng.uniform(0.0, 2.5)), 3))
    else:
        case.update(nets=_log(rng, 20, 250), iters=rng.randint(1, 4), pins=rng.choice(["short", "multi"]))
    return case


# ------------------------------------------------------------------ boards
def _spans(case):
    if not case["span"]:
        return None
    return [(a, b) for a, b in Lattice(2, 2, case["nz"]).via_pairs() if b - a <= case["span"]]


def _lattice(case, **kw):
    return Lattice(case["nx"], case["ny"], case["nz"], allowed_via_spans=_spans(case), **kw)


def _via_chain(lat, case, x, y, a, b):
    """Nodes after (x, y, a) down to layer b in legal via hops."""
    step = 1 if lat.nz > 18 else (case["span"] or lat.nz)
    out = []
    while a != b:
        a = min(b, a + step) if b > a else max(b, a - step)
        out.append(lat.node_idx(x, y, a))
    return out


def _straight_paths(lat, case, n, rng):
    """n paths on other nets' behalf: down a via, along an H layer, via, along a V layer, back up."""
    nx, ny, nz = lat.nx, lat.ny, lat.nz
    out = []
    while len(out) < n:
        x0, x1 = (int(v) for v in rng.integers(0, nx, size=2))
        y0, y1 = (int(v) for v in rng.integers(0, ny, size=2))
        if x0 == x1 or y0 == y1:
            continue
        h = 1 + 2 * int(rng.integers(0, max(1, (nz - 1) // 2)))
        v = 2 + 2 * int(rng.integers(0, max(1, (nz - 2) // 2)))
        h, v = min(h, nz - 2 - (nz - 2 + 1) % 2), min(v, nz - 2 - (nz - 2) % 2)
        xs = np.arange(x0, x1, 1 if x1 > x0 else -1)[1:].tolist() + [x1]
        ys = np.arange(y0, y1, 1 if y1 > y0 else -1)[1:].tolist() + [y1]
        p = [lat.node_idx(x0, y0, 0)] + _via_chain(lat, case, x0, y0, 0, h)
        p += [lat.node_idx(x, y0, h) for x in xs] + _via_chain(lat, case, x1, y0, h, v)
        p += [lat.node_idx(x1, y, v) for y in ys] + _via_chain(lat, case, x1, y1, v, 0)
        out.append(np.asarray(p, dtype=np.int32))
    return out


def _terminals(lat, lo, hi, rng):
    while True:
        x0, x1 = (int(v) for v in rng.integers(0, lat.nx, size=2))
        y0, y1 = (int(v) for v in rng.integers(0, lat.ny, size=2))
        if lo <= abs(x1 - x0) + abs(y1 - y0) <= hi:
            return x0, y0, x1, y1


def _congested(case, rng):
    """A board in mid-negotiation: (lattice, graph, state, ops)."""
    lat = _lattice(case)
    g = DeviceGraph(lat)
    s = DeviceState(g)
    s.enable_rcost()
    ops = Ops(g, s)
    paths = _straight_paths(lat, case, case["paths"], rng)
    ops.commit_paths(paths, list(range(len(paths))))
    ops.present_ema(0.40)
    ops.present_ema(0.40)
    ops.update_history(0.25)
    hot = np.unique(np.concatenate([p[::7] for p in paths]))
    s.node_history[torch.from_numpy(hot).long().cuda()] = 1.0
    bias = (1.0 + 0.3 * rng.random(lat.nz)).astype(np.float32)
    ops.update_costs(case["pres"], HIST_WEIGHT, 1.0, 0.3, bias)
    ops.live_begin(case["pres"])
    return lat, g, s, ops


def _net(ops, lat, case, net_id, x0, y0, x1, y1):
    dist = abs(x1 - x0) + abs(y1 - y0)
    return ops.net_args(net_id, lat.node_idx(x0, y0, 0), lat.node_idx(x1, y1, 0), full_graph=case["whole"],
                        max_depth=min(max(60, int(0.75 * dist)), 80), halo=2, pres_fac=case["pres"])


def _requests(case, seed):
    """Requests of a job or a pass; nets go by their board net code (an integer)."""
    nx, ny, n = case["nx"], case["ny"], case["nets"]
    if case.get("pins") == "multi":
        reqs = star_requests(seeded_multipin_nets(nx, ny, n, seed, box=min(50, nx, ny)))
        return [(k, a, b) for k, (_, a, b) in enumerate(r for r in reqs if r[1] != r[2])][:n]
    rng = np.random.default_rng(seed)
    out = []
    if case.get("pins") == "short":
        while len(out) < n:
            x0, x1 = (int(v) for v in rng.integers(0, nx, size=2))
            y0, y1 = (int(v) for v in rng.integers(0, ny, size=2))
            if 5 <= abs(x1 - x0) + abs(y1 - y0) <= 80:
                out.append((len(out), y0 * nx + x0, y1 * nx + x1))
        return out
    box = min(20, nx // 3, ny // 3)
    centres = [(int(rng.integers(0, nx - box)), int(rng.integers(0, ny - box))) for _ in range(2)]
    while len(out) < n:
        x1, y1 = int(rng.integers(0, nx)), int(rng.integers(0, ny))
        if len(out) % 10 < 3:
            cx, cy = centres[len(out) % 2]
            x0, y0 = cx + int(rng.integers(0, box)), cy + int(rng.integers(0, box))
        else:
            x0, y0 = int(rng.integers(0, nx)), int(rng.integers(0, ny))
        if (x0, y0) != (x1, y1):
            out.append((len(out), y0 * nx + x0, y1 * nx + x1))
    return out


def _table(lat, requests):
    """Per-net parameters of a routing pass on the device, and which nets are long (host)."""
    ends = np.asarray([(a, b) for _, a, b in requests], dtype=np.int64)
    y, x = np.divmod(ends % lat.plane, lat.nx)
    dist = np.abs(x[:, 1] - x[:, 0]) + np.abs(y[:, 1] - y[:, 0])
    depth = np.minimum(np.maximum(60, (0.75 * dist).astype(np.int64)), 80).repeat(2)
    full = dist >= 125
    t = dict(src=ends[:, 0], dst=ends[:, 1], id=1_000_000 + np.arange(len(requests)), full=full, depth=depth,
             halo=np.full(2 * len(requests), 2))
    return {k: torch.from_numpy(v.astype(np.int32)).cuda() for k, v in t.items()}, full.astype(np.uint8)


def _lattice_params(case, seed):
    """Grid pitch and via cost of a board (they scale the arc costs)."""
    rng = np.random.default_rng(seed)
    return dict(pitch=float(np.round(0.35 + 0.1 * rng.random(), 4)), via_cost=float(np.round(0.5 + rng.random(), 4)))


def _arc_inputs(E, seed):
    """Present, EMA and history per arc: most arcs unused, some shared."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand(E, generator=gen, device="cuda")
    present = (u < 0.06).float() + (u < 0.01).float() + (u < 0.002).float()
    ema = present * 0.4 + (torch.rand(E, generator=gen, device="cuda") < 0.05).float() * 0.6
    history = torch.where(u < 0.02, torch.rand(E, generator=gen, device="cuda"), torch.zeros_like(u))
    return present, ema, history


def _bias(nz, seed):
    return (1.0 + 0.4 * np.random.default_rng(seed).random(nz)).astype(np.float32)


# ------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "lattice":
        kw = _lattice_params(case, seed)
        if case["ww"] > 0:
            kw["wrong_way_cost_multiplier"] = case["ww"]
        return dict(case=case, lat=_lattice(case, min_via_center_spacing=kw["pitch"], **kw))
    if kind == "job":
        lat = _lattice(case)
        p = lat.pitch
        router = PathFinderRouter(PathFinderConfig(max_iterations=case["iters"]))
        router.initialize_lattice(lat, (7.0, 7.0, 7.0 + (lat.nx - 1) * p, 7.0 + (lat.ny - 1) * p))
        return dict(case=case, router=router, requests=_requests(case, seed))
    if kind == "costs":
        g = DeviceGraph(_lattice(case))
        s = DeviceState(g)
        s.enable_rcost()
        ops = Ops(g, s)
        for t, v in zip((s.present, s.present_ema, s.history), _arc_inputs(g.E, seed)):
            t.copy_(v)
        s.path_node_use.copy_(torch.from_numpy((rng.random(g.N) < 0.04).astype(np.int32) +
                                               (rng.random(g.N) < 0.01).astype(np.int32)))
        return dict(case=case, g=g, s=s, ops=ops, bias=_bias(g.lattice.nz, seed))
    lat, g, s, ops = _congested(case, rng)
    if kind == "nets":
        nets = [_net(ops, lat, case, 1_000_000 + k, *_terminals(lat, case["lo"], case["hi"], rng))
                for k in range(case["nets"])]
        return dict(case=case, g=g, s=s, ops=ops, nets=nets)
    if kind == "pass":
        requests = _requests(case, seed)
        table, full = _table(lat, requests)
        return dict(case=case, g=g, s=s, ops=ops, table=table, full=full, store=PathStore(g, len(requests),
                                                                                          window_slots=32))
    x0, y0, x1, y1 = _terminals(lat, case["lo"], case["hi"], rng)
    inner = range(1, lat.nz - 1)
    return dict(case=case, g=g, s=s, ops=ops, net=_net(ops, lat, case, 1_000_000, x0, y0, x1, y1),
                seeds=[(lat.node_idx(x0, y0, z), 0.05 * z) for z in inner],
                targets=[(lat.node_idx(x1, y1, z), 0.03 * z) for z in inner])


def _nodes(path, room=8192):
    """A path's nodes in an array of fixed length."""
    out = np.full(room, -1, dtype=np.int32)
    if path is not None:
        out[:len(path)] = path
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "lattice":
        g = DeviceGraph(state["lat"])
        return dict(indptr=g.indptr, indices=g.indices, base_costs=g.base_costs, edge_layer=g.edge_layer,
                    edge_kind=g.edge_kind, edge_src=g.edge_src, rev=g.rev)
    if kind == "job":
        router = state["router"]
        router.config = PathFinderConfig(max_iterations=case["iters"])   # a job derives its own parameters
        router.initialize_state()
        res = router.route_multiple_nets(state["requests"])
        paths = [res["paths"].get(name) or [] for name, _, _ in state["requests"]]
        s = router.s
        return dict(paths=_nodes([v for p in paths for v in p], 1024 * len(paths)),
                    lengths=np.asarray([len(p) for p in paths]),
                    result=np.asarray([int(res.get(k) or 0) for k in ("success", "iterations", "barrel_conflicts",
                                                                      "overuse_sum", "overuse_edges", "failed_nets")]),
                    present=s.present, path_node_use=s.path_node_use, owner_count=s.owner_count, history=s.history)
    if kind == "costs":
        ops, s = state["ops"], state["s"]
        ops.present_ema(0.40)
        tally = ops.tally(canonical_only=True)
        ops.update_costs(case["pres"], HIST_WEIGHT, 1.0, 0.3, state["bias"])
        ops.live_begin(case["pres"])
        ops.update_history(0.25)
        return dict(total_cost=s.total_cost, live_static=s.live_static, present_ema=s.present_ema, history=s.history,
                    over=np.asarray(tally[:4]), layers=tally[4])
    ops = state["ops"]
    if kind == "pass":
        store, s = state["store"], state["s"]
        status, stats = route_pass(ops, store, state["table"], np.arange(case["nets"], dtype=np.int32),
                                   fallback_quota=5, max_roi_nodes=50_000, owner_weight=25.0 * case["pres"],
                                   path_weight=25.0 * case["pres"], history_weight=5.0, pres_fac=case["pres"], live=True,
                                   order_full=state["full"])
        used = torch.arange(store.slot_cap, device=s.present.device) < store.length[:, None]
        return dict(status=status, work=stats[:2], paths=torch.where(used, store.path, -1), present=s.present,
                    total_cost=s.total_cost, path_node_use=s.path_node_use, owner_count=s.owner_count)
    ops.stats.zero_()
    if kind == "nets":
        out = dict(("path%d" % k, _nodes(ops.find_path(net))) for k, net in enumerate(state["nets"]))
        out["work"] = ops.stats[:2]          # arcs scanned and nodes popped, as the heap search counts them
        return out
    if case["whole"]:
        got = ops.find_path_full_multi(state["seeds"], state["targets"], state["net"])
        return dict(path=_nodes(got and got[0]), work=ops.stats[:2])
    roi = ops.extract_roi(state["net"])
    got = ops.find_path_multi(state["seeds"], state["targets"], state["s"].total_cost, roi)
    return dict(path=_nodes(got and got[0]), roi=_nodes(roi, 50_000), work=ops.stats[:2])


# ------------------------------------------------------------------ work
def _num_arcs(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    lat = _lattice(case)
    ww = case.get("ww", 0.0) > 0
    E = 2 * len(lat.via_pairs()) * nx * ny
    for z in lat.lateral_layers():
        if lat.layer_dirs[z] == "h" or ww:
            E += 2 * ny * (nx - 1)
        if lat.layer_dirs[z] == "v" or ww:
            E += 2 * nx * (ny - 1)
    return E


def work(case):
    N, E = case["nx"] * case["ny"] * case["nz"], _num_arcs(case)
    kind = case["kind"]
    # a search reads each arc's head and cost and each node's row and penalty inputs once
    whole = 8 * E + 20 * N
    roi = min(1.0, 50_000 / N) * whole
    if kind == "lattice":
        return {"bytes": 4 * N + 18 * E, "flops": E}
    if kind == "costs":
        # in: base, layer, kind, present, EMA, capacity, history, node use; out: EMA, history, live and total costs
        return {"bytes": 38 * E + 4 * N, "flops": 20 * E}
    if kind == "job":
        b = case["nets"] * (1 + 0.25 * (case["iters"] - 1)) * roi + case["iters"] * 38 * E
        return {"bytes": b, "flops": b / 4}
    if kind == "pass":
        long = min(0.9, max(0.1, (case["nx"] + case["ny"] - 150) / 900.0))   # share of long nets
        b = case["nets"] * (long * whole + (1 - long) * roi)
        return {"bytes": b, "flops": b / 4}
    b = case.get("nets", 1) * (whole if case["whole"] else roi)
    return {"bytes": b, "flops": b / 4}


# ------------------------------------------------------------------ exact values
def _plain_csr(case, pitch=0.4, via_cost=0.7):
    """The lattice's arcs in 64 bits, by rows sorted on the destination."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    lat = _lattice(case)
    dev = "cuda"
    ids = torch.arange(nx * ny * nz, device=dev).view(nz, ny, nx)
    src, dst, cost, kind = [], [], [], []

    def add(a, b, c, k):
        for u, v in ((a, b), (b, a)):
            src.append(u.reshape(-1))
            dst.append(v.reshape(-1))
            cost.append(torch.full((u.numel(),), c, dtype=torch.float64, device=dev))
            kind.append(torch.full((u.numel(),), k, dtype=torch.uint8, device=dev))

    ww = case.get("ww", 0.0)
    for z in lat.lateral_layers():
        h = lat.layer_dirs[z] == "h"
        if h or ww > 0:
            add(ids[z, :, :-1], ids[z, :, 1:], pitch if h else pitch * ww, 0)
        if not h or ww > 0:
            add(ids[z, :-1, :], ids[z, 1:, :], pitch if not h else pitch * ww, 0)
    pairs = lat.via_pairs()
    adjacent = nz > 2 and all(b - a == 1 for a, b in pairs)
    for a, b in pairs:
        add(ids[a], ids[b], via_cost * 4.0 if adjacent else via_cost * (1.0 + 0.15 * (b - a - 1)), 1)
    src, dst, cost, kind = (torch.cat(t) for t in (src, dst, cost, kind))
    N = nx * ny * nz
    order = torch.argsort(src * N + dst)
    src, dst, cost, kind = src[order], dst[order], cost[order], kind[order]
    indptr = torch.zeros(N + 1, dtype=torch.int64, device=dev)
    indptr[1:] = torch.cumsum(torch.bincount(src, minlength=N), 0)
    back = torch.searchsorted(src * N + dst, dst * N + src)
    return indptr, src, dst, cost, (src // (nx * ny)).to(torch.uint8), kind, back


def exact(case, seed):
    if case["kind"] == "lattice":
        p = _lattice_params(case, seed)
        indptr, src, dst, cost, layer, kind, back = _plain_csr(case, p["pitch"], p["via_cost"])
        return dict(indptr=indptr, indices=dst, base_costs=cost, edge_layer=layer, edge_kind=kind, edge_src=src,
                    rev=back)
    if case["kind"] != "costs":
        return None                      # paths and counts: whole numbers
    _, src, dst, base, layer, kind, _ = _plain_csr(case)
    E = src.numel()
    present, ema, history = (t.double() for t in _arc_inputs(E, seed))
    bias = torch.where(kind == 0, torch.from_numpy(_bias(case["nz"], seed)).double().cuda()[layer.long()], 1.0)
    ema = 0.4 * present + 0.6 * ema
    scale = case["pres"] * bias
    over = torch.clamp(ema - 1.0, min=0.0)
    # the jitter's argument is the arc number rounded to 32 bits: that is its definition
    jitter = torch.remainder(torch.arange(E, device="cuda").float().double(), 9973.0) * 1e-6
    total = base * 0.3 * bias + scale * over + HIST_WEIGHT * history + jitter
    live = total - scale * over
    total = live + scale * torch.clamp(present, min=0.0)      # max(0, present + 1 - capacity), capacity 1
    history = history + torch.minimum(0.25 * torch.clamp(present - 1.0, min=0.0), 15.0 * base)
    return dict(total_cost=total, live_static=live, present_ema=ema, history=history, over=None, layers=None)
