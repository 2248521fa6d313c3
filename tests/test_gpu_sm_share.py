"""ROI searches keep to their host thread's share of the SMs (ogr_full_grid) and return the same at any share."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle.dijkstra import find_path_multisource, find_path_roi_c

from test_gpu_kernels import make


@pytest.mark.parametrize("share", [1, 2, 19, 75, 77, 0])
def test_roi_searches_at_any_share(share):
    from orthoroute_gb300.autotune import full_grid
    g, s, ops, ref = make(90, 70, 6)
    rng = np.random.default_rng(31)
    costs = (0.125 + rng.integers(0, 3, size=g.E) * 0.125).astype(np.float32)
    costs[rng.random(g.E) < 0.05] = np.float32("inf")
    s.total_cost.copy_(torch.from_numpy(costs))
    before, limit = full_grid(0)
    try:
        full_grid(share or limit)
        for _ in range(4):
            src, dst = (int(v) for v in rng.choice(ref.plane, size=2, replace=False))
            net = ops.net_args(0, src, dst, penalty=False)
            roi = ops.extract_roi(net)
            g2r = np.full(g.N, -1, dtype=np.int32)
            g2r[roi] = np.arange(roi.size, dtype=np.int32)
            want = find_path_roi_c(ref.indptr, ref.indices, src, dst, costs, roi, g2r)
            assert ops.find_path(net) == want
            assert ops.find_path_given_roi(src, dst, s.total_cost, roi) == want
            seeds = [(src, 0.0), (src + ref.plane, 0.25)]
            targets = [(dst, 0.0), (dst + ref.plane, 0.5)]
            want = find_path_multisource(ref.indptr, ref.indices, seeds, targets, costs, roi, g2r, plane=ref.plane)
            assert ops.find_path_multi(seeds, targets, s.total_cost, roi) == (tuple(want) if want else None)
    finally:
        full_grid(before)


def test_a_share_of_one_waits_for_no_one():
    """One CTA has no team to wait for, so a limit of no polls does not stop it; a team of two it stops."""
    from orthoroute_gb300 import _lib
    from orthoroute_gb300.autotune import full_grid
    g, s, ops, ref = make(60, 50, 6)
    s.total_cost.copy_(g.base_costs)
    net = ops.net_args(0, 5 * 60 + 5, 30 * 60 + 40, penalty=False)
    want = ops.find_path(net)
    before, _ = full_grid(0)
    try:
        _lib.debug_limits(1, 0)
        full_grid(1)
        assert want and ops.find_path(net) == want
        full_grid(2)
        with pytest.raises(RuntimeError, match="grid barrier timed out"):
            ops.find_path(net)
    finally:
        _lib.debug_limits(0, 0)
        full_grid(before)
