"""Whole-lattice multi-source searches with many seeds and targets (entered by all threads of a CTA), and bad ones among
them, against the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle.dijkstra import find_path_multisource

from test_gpu_kernels import make


def board(seed):
    g, s, ops, ref = make(60, 50, 6)
    rng = np.random.default_rng(seed)
    costs = (0.125 + rng.integers(0, 3, size=g.E) * 0.125).astype(np.float32)
    s.total_cost.copy_(torch.from_numpy(costs))
    return g, s, ops, ref, costs, rng


@pytest.mark.parametrize("n_seeds,n_targets", [(1, 1), (511, 513), (3000, 700), (18_000, 1), (2, 18_000)])
@pytest.mark.parametrize("exact", [True, False])        # seed costs that ticks hold, and that they do not
def test_many_seeds_and_targets(n_seeds, n_targets, exact):
    g, s, ops, ref, costs, rng = board(n_seeds + n_targets)
    ident = np.arange(g.N, dtype=np.int32)
    net = ops.net_args(0, 0, 1, full_graph=True, penalty=False)
    for _ in range(2):
        sc = rng.integers(0, 16, size=n_seeds) / 8.0 + (0.0 if exact else 1e-12)
        seeds = [(int(n), float(c)) for n, c in zip(rng.choice(g.N, size=n_seeds, replace=False), sc)]
        targets = [(int(n), float(c)) for n, c in zip(rng.choice(g.N, size=n_targets, replace=False),
                                                      rng.integers(0, 16, size=n_targets) / 8.0)]
        want = find_path_multisource(ref.indptr, ref.indices, seeds, targets, costs, ident, ident, plane=ref.plane)
        assert ops.find_path_full_multi(seeds, targets, net) == (tuple(want) if want else None)


@pytest.mark.parametrize("where", [0, 1, 511, 512, 999])
@pytest.mark.parametrize("what", ["seed twice", "seed outside", "seed below 0", "seed NaN", "target twice",
                                  "target outside", "target NaN"])
def test_a_bad_seed_or_target_anywhere_is_refused(what, where):
    from orthoroute_gb300 import _lib
    g, s, ops, ref, costs, rng = board(3)
    ids = rng.choice(g.N, size=2000, replace=False).astype(np.int32)
    seeds, targets = ids[:1000].copy(), ids[1000:].copy()
    sc, tc = np.zeros(1000), np.zeros(1000)
    if what == "seed twice":
        seeds[where] = seeds[(where + 500) % 1000]
    elif what == "seed outside":
        seeds[where] = g.N
    elif what == "seed below 0":
        sc[where] = -0.5
    elif what == "seed NaN":
        sc[where] = np.nan
    elif what == "target twice":
        targets[where] = targets[(where + 500) % 1000]
    elif what == "target outside":
        targets[where] = -1
    else:
        tc[where] = np.nan
    d = [torch.from_numpy(v).to(g.device) for v in (seeds, sc, targets, tc)]
    ws = ops.full_workspace()
    cg, st, net, n = g.cgraph(), s.cstate(), ops.net_args(0, 0, 1, full_graph=True, penalty=False), C.c_int32(0)
    p = lambda t: t.data_ptr()
    call = lambda k: ops.lib.ogr_find_path_full_multi(C.byref(cg), C.byref(st), C.byref(net), p(d[0]), p(d[1]), k, p(d[2]),
                                                      p(d[3]), k, p(ws), ops.full_ws_bytes, p(ops.path_buf),
                                                      int(ops.path_buf.numel()), C.byref(n), None, ops._sp())
    assert call(1000) == _lib.OGR_ERR_ARG
    # and the marks of the good ones are gone
    good = [(int(v), 0.0) for v in ids[:3]], [(int(v), 0.0) for v in ids[1000:1003]]
    ident = np.arange(g.N, dtype=np.int32)
    want = find_path_multisource(ref.indptr, ref.indices, *good, costs, ident, ident, plane=ref.plane)
    assert ops.find_path_full_multi(*good, net) == (tuple(want) if want else None)
