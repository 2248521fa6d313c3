"""What a job is admitted by is what it allocates."""
import pytest

from orthoroute_gb300 import Lattice
from orthoroute_gb300.serve import job_footprint


@pytest.mark.parametrize("dims,nets", [((100, 100, 6), 200), ((600, 400, 12), 2000), ((1000, 800, 32), 512)])
def test_footprint_counts_the_workspaces_as_the_library_sizes_them(dims, nets):
    """Each of them is in the sum: more window slots, nets or arcs cost what the library says they cost."""
    from orthoroute_gb300 import _lib
    lib = _lib.load()
    N, E = dims[0] * dims[1] * dims[2], 10_000_000
    f = lambda **k: job_footprint(*dims, **{**dict(num_edges=E, num_nets=nets), **k})
    assert f(window_slots=8) - f(window_slots=0) == lib.ogr_window_workspace_bytes(N, 50_000, 8) + 8 * 8192 * 4
    qcap = min(N, 1 << 18)
    assert f(bfs_slots=5) - f(bfs_slots=4) == lib.ogr_bfs_workspace_bytes(N, qcap, 1)
    more = f(num_edges=E + 1_000_000) - f()
    assert more == (18 + 28) * 1_000_000 + lib.ogr_full_workspace_bytes(N, E + 1_000_000) - lib.ogr_full_workspace_bytes(N, E)
    assert f() > lib.ogr_route_workspace_bytes(N) + lib.ogr_full_workspace_bytes(N, E) + 46 * E


@pytest.mark.gpu
@pytest.mark.parametrize("dims,slots", [((300, 200, 8), 32), ((300, 200, 8), 0), ((120, 100, 20), 16)])
def test_footprint_is_what_a_router_allocates(dims, slots):
    """At most 64 MB (its allowance for the small arrays of a job) and 2 % above, never below."""
    import gc

    import numpy as np
    import torch
    from orthoroute_gb300.router import PathFinderConfig, PathFinderRouter
    rng = np.random.default_rng(1)
    reqs = [(f"N{k}", int(a), int(b)) for k, (a, b) in enumerate(rng.integers(0, dims[0] * dims[1], size=(60, 2))) if a != b]
    gc.collect()                 # (another test's router)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    R = PathFinderRouter(PathFinderConfig(max_iterations=1), window_slots=slots)
    R.initialize_lattice(Lattice(*dims))
    R.route_multiple_nets(reqs)
    R.ops.full_workspace()
    used = torch.cuda.memory_allocated() - before
    said = job_footprint(*dims, num_edges=R.g.E, num_nets=len(reqs), window_slots=slots)
    assert used <= said <= used * 1.02 + (64 << 20), (used, said)
