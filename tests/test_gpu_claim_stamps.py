"""The stamps that mark a search's claimed nodes count searches; where the count runs out they begin again at 1, and no
node may still carry a stamp of the first searches."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle.dijkstra import find_path_roi_c

from test_gpu_kernels import make


def r256(v):
    return (v + 255) // 256 * 256


@pytest.mark.parametrize("left", [0, 1, 2])
def test_roi_searches_after_the_stamps_ran_out(left):
    g, s, ops, ref = make(40, 33, 6)
    rng = np.random.default_rng(4)
    costs = (0.125 + rng.integers(0, 3, size=g.E) * 0.125).astype(np.float32)
    dev = torch.from_numpy(costs).to(g.device)
    everything = np.arange(g.N, dtype=np.int32)
    few = everything[: ref.plane // 4]

    def search(roi, src, dst):
        g2r = np.full(g.N, -1, dtype=np.int32)
        g2r[roi] = np.arange(roi.size, dtype=np.int32)
        want = find_path_roi_c(ref.indptr, ref.indices, src, dst, costs, roi, g2r)
        assert ops.find_path_given_roi(src, dst, dev, roi) == want, (roi.size, src, dst)

    far = (0, ref.plane - 1)
    for _ in range(4):                       # stamps 1 to 4 on the nodes of the whole lattice
        search(everything, *far)
    # the count of searches, behind the team's 384 bytes of control words, as 2^31 searches would leave it
    at = 5 * r256(4 * g.N) + 3 * r256(16 * g.N) + 384
    sid = ops.ws[0][at: at + 4].view(torch.int32)
    assert int(sid) == 4
    sid.fill_(0x7ffffffe - left)
    for _ in range(3 + left):                # the next stamp is 4 again: that of the last search of the whole lattice
        search(few, 0, 1)
    assert int(sid) == 3
    for _ in range(4):
        search(everything, *far)


def test_whole_lattice_searches_after_the_stamps_ran_out():
    g, s, ops, ref = make(40, 33, 6)
    rng = np.random.default_rng(4)
    costs = (0.125 + rng.integers(0, 3, size=g.E) * 0.125).astype(np.float32)
    s.total_cost.copy_(torch.from_numpy(costs))
    ident = np.arange(g.N, dtype=np.int32)
    net = ops.net_args(0, 0, ref.plane - 1, full_graph=True, penalty=False)
    want = find_path_roi_c(ref.indptr, ref.indices, 0, ref.plane - 1, costs, ident, ident)
    for _ in range(3):
        assert ops.find_path(net, engine="grid") == want
    sid = ops.full_workspace()[384 + 16: 384 + 20].view(torch.int32)     # behind the team's words and the result
    assert int(sid) == 3
    sid.fill_(0x7ffffffd)
    for _ in range(6):
        assert ops.find_path(net, engine="grid") == want
    assert 0 < int(sid) < 6
