"""What a cached tuning is keyed by, and that knobs the searches ignore are not told apart."""
import json
import types

import pytest

from orthoroute_gb300 import Lattice
from orthoroute_gb300 import autotune as T


@pytest.fixture
def gpu(monkeypatch):
    props = types.SimpleNamespace(name="GB300", multi_processor_count=152)
    monkeypatch.setattr(T.torch.cuda, "get_device_properties", lambda d: props)


def test_key_tells_lattices_and_engines_apart(gpu, monkeypatch):
    base = dict(nx=60, ny=50, nz=6)
    lats = [Lattice(**base), Lattice(61, 50, 6), Lattice(**base, allowed_via_spans=[(0, 1), (1, 2)]),
            Lattice(**base, wrong_way_cost_multiplier=3.0), Lattice(**base, wrong_way_cost_multiplier=4.0),
            Lattice(**base, min_via_center_spacing=0.5), Lattice(**base, min_via_center_spacing=0.9),
            Lattice(**base, allow_any_layer_via=False)]
    keys = [T.lattice_key(lat, "cuda") for lat in lats]
    assert len(set(keys)) == len(keys)
    assert T.lattice_key(Lattice(**base), "cuda") == keys[0]
    monkeypatch.setattr(T, "ENGINE", "another")
    assert T.lattice_key(lats[0], "cuda") != keys[0]


def test_a_choice_of_an_earlier_engine_is_not_found(gpu, tmp_path, monkeypatch):
    """Entries written before the engine was part of the key."""
    path = tmp_path / "tune.json"
    monkeypatch.setenv("ORTHOROUTE_GB300_TUNE_CACHE", str(path))
    old = "GB300/152sm/60x50x6/all"
    path.write_text(json.dumps({old: {"key": old, "full_engine": "cta", "full_ctas": 76}}))
    assert T.lattice_key(Lattice(60, 50, 6), "cuda") not in T._load_cache(T.cache_path())


@pytest.mark.gpu
def test_ignored_knobs_are_timed_once_and_left_alone(tmp_path, monkeypatch):
    import numpy as np
    import torch
    from test_gpu_kernels import make
    monkeypatch.setenv("ORTHOROUTE_GB300_TUNE_CACHE", str(tmp_path / "tune.json"))
    g, s, ops, ref = make(60, 50, 6)
    s.total_cost.copy_(torch.from_numpy((0.125 + np.random.default_rng(2).integers(0, 3, size=g.E) * 0.125).astype(np.float32)))
    cur, lim = T.full_grid(0)
    try:
        T.full_lanes(8)
        T.full_reuse(1)
        T.search_lanes(2)
        t = T.tune(ops, Lattice(60, 50, 6), [(0, 2999), (59, 2940)], [(3, 400), (70, 900)])
        assert (t.full_lanes, t.full_reuse, t.roi_lanes) == (8, 1, 2)
        assert (T.full_lanes(0), T.full_reuse(), T.search_lanes(0)) == (8, 1, 2)
        assert len({t.ms_per_search[f"full_lanes{k}_reuse{r}"] for k in T.FULL_LANES for r in (0, 1)}) == 1
        assert len({t.ms_per_search[f"roi_lanes{k}"] for k in T.LANES}) == 1
        assert not t.cached and T.tune(ops, Lattice(60, 50, 6), [(0, 2999)]).cached
    finally:
        T.full_tile(0)
        T.full_grid(cur)
        T.full_lanes(16)
        T.full_reuse(0)
        T.search_lanes(4)
