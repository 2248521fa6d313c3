"""ROIs whose box shared memory cannot hold (searched in global memory by the whole cluster): node for node the oracle's,
again and again on one workspace, with blocked arcs, cut to a limit, and from the pass's own extraction."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle.roi import extract_roi_bfs

from test_gpu_kernels import make


@pytest.mark.parametrize("dims,limit,blocked", [
    ((260, 250, 16), 10**6, False), ((200, 190, 32), 10**6, False), ((200, 190, 32), 150_000, True),
    ((260, 250, 16), 90_001, False), ((400, 70, 40), 10**6, True),
])
def test_large_extraction_matches_oracle(dims, limit, blocked):
    g, s, ops, ref = make(*dims)
    rng = np.random.default_rng(dims[0] + dims[2])
    mask = None
    if blocked:
        mask = rng.random(g.E) < 0.1
        g.blocked = torch.from_numpy(mask.astype(np.uint8)).to(g.device)
    nets = [tuple(int(v) for v in rng.integers(0, ref.plane, size=2)) for _ in range(3)]
    mid = (dims[1] // 2) * dims[0] + dims[0] // 2
    nets += [(mid, mid), (mid, mid + 1), (0, ref.plane - 1)]
    for src, dst in nets + nets[:2]:
        want, _ = extract_roi_bfs(ref.indptr, ref.indices, g.N, src, dst, initial_radius=80, blocked=mask, max_nodes=limit)
        net = ops.net_args(0, src, dst, max_depth=80, halo=2, max_roi_nodes=limit)
        np.testing.assert_array_equal(ops.extract_roi(net), want, err_msg=str((src, dst)))


def test_search_on_a_large_roi_matches_oracle():
    from oracle.dijkstra import find_path_roi_c
    g, s, ops, ref = make(200, 190, 32)
    rng = np.random.default_rng(6)
    costs = (0.125 + rng.integers(0, 3, size=g.E) * 0.125).astype(np.float32)
    s.total_cost.copy_(torch.from_numpy(costs))
    for src, dst in ((95 * 200 + 60, 100 * 200 + 150), (20 * 200 + 20, 60 * 200 + 70)):
        roi, g2r = extract_roi_bfs(ref.indptr, ref.indices, g.N, src, dst, initial_radius=80, max_nodes=10**6)
        st = {}
        want = find_path_roi_c(ref.indptr, ref.indices, src, dst, costs, roi, g2r, stats=st)
        net = ops.net_args(0, src, dst, max_depth=80, halo=2, max_roi_nodes=10**6, penalty=False)
        ops.stats.zero_()
        assert ops.find_path(net) == want
        assert ops.stats.cpu().tolist()[:3] == [st["scanned"], st["settled"], roi.size]
