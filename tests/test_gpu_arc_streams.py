"""The per-arc streams (cost update, live rebase, EMA, history, reverse costs, tally) in both their forms: four arcs at
a time (aligned arrays, with a remainder) and one by one (arrays that start off a 16-byte boundary), bit for bit
against the oracle's accounting and whole-number sums."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import accounting as oacc


def at(a, off):
    """`a` on the device, starting `off` elements into an aligned buffer."""
    t = torch.zeros(a.size + off + 8, dtype=torch.from_numpy(a).dtype, device="cuda")[off:off + a.size]
    t.copy_(torch.from_numpy(a))
    return t


@pytest.mark.parametrize("E", [1, 3, 4, 7, 1030, 20_011])
@pytest.mark.parametrize("off", [0, 1])
def test_streams_match_oracle(E, off):
    from orthoroute_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(E + off)
    nz = 5
    f = np.float32
    present = rng.integers(0, 4, size=E).astype(f)
    ema = np.zeros(E, dtype=f)
    for _ in range(3):
        ema = f(0.4) * rng.integers(0, 4, size=E).astype(f) + f(0.6) * ema
    hist, base = rng.random(E).astype(f), (0.1 + rng.random(E)).astype(f)
    layer = np.sort(rng.integers(0, nz, size=E)).astype(np.uint8)
    kind = rng.integers(0, 2, size=E).astype(np.uint8)
    src, dst = rng.integers(0, 50, size=(2, E)).astype(np.int32)
    rev = rng.permutation(E).astype(np.int32)
    bias = (1.0 + rng.random(nz)).astype(f)
    use = rng.integers(0, 4, size=10 * nz).astype(np.int32)
    A = oacc.Accountant(E)
    A.present[:], A.present_ema[:], A.history[:] = present, ema, hist
    d = {k: at(v, off) for k, v in dict(present=present, ema=ema, hist=hist, base=base, cap=np.ones(E, dtype=f),
                                        total=np.zeros(E, dtype=f), live=np.zeros(E, dtype=f),
                                        rcost=np.zeros(E, dtype=f), layer=layer, kind=kind, rev=rev, src=src,
                                        dst=dst).items()}
    p = {k: t.data_ptr() for k, t in d.items()}
    db, du = at(bias, 0), at(use, 0)
    a = _lib.CostArgs(E, p["base"], p["layer"], p["kind"], p["ema"], p["cap"], p["hist"], None, db.data_ptr(), 1.5, 0.25,
                      float(f(3.7)), float(f(9.6)), 1)
    A.update_costs(base, 3.7, 9.6, via_cost_multiplier=1.5, base_cost_weight=0.25, edge_layer=layer,
                   layer_bias_per_layer=bias, edge_kind=kind)
    assert lib.ogr_costs_update(C.byref(a), p["total"], None) == 0
    np.testing.assert_array_equal(d["total"].cpu().numpy(), A.total_cost)
    A.begin_live_present_costs()
    assert lib.ogr_live_begin(C.byref(a), p["present"], p["total"], p["live"], None) == 0
    np.testing.assert_array_equal(d["total"].cpu().numpy(), A.total_cost)
    np.testing.assert_array_equal(d["live"].cpu().numpy(), A._live_static_cost)
    assert lib.ogr_reverse_costs(E, p["rev"], p["total"], p["rcost"], None) == 0
    np.testing.assert_array_equal(d["rcost"].cpu().numpy(), A.total_cost[rev])
    out = torch.zeros(5, dtype=torch.int64, device="cuda")
    units = torch.zeros(nz, dtype=torch.int64, device="cuda")
    for canonical in (0, 1):
        assert lib.ogr_tally(E, use.size, nz, p["present"], p["ema"], p["cap"], p["src"], p["dst"], p["layer"],
                             du.data_ptr(), canonical, out.data_ptr(), units.data_ptr(), None) == 0
        over = np.maximum(present - 1, 0).astype(np.int64) * ((src < dst) if canonical else 1)
        eo = np.maximum(f(0), ema - f(1)).astype(np.float64) * 2.0 ** 23
        want = np.bincount(layer, weights=eo, minlength=nz).astype(np.int64)
        want += np.maximum(use.reshape(nz, -1) - 1, 0).sum(axis=1).astype(np.int64) << 23
        assert out.cpu().tolist() == [int(over.sum()), int((over > 0).sum()), int(np.maximum(use - 1, 0).sum()),
                                      int((use > 1).sum()), 0]
        assert units.cpu().tolist() == want.tolist()
    A.update_history(0.2, base_costs=base, history_cap_multiplier=15.0, decay_factor=0.98, use_raw_present=True)
    assert lib.ogr_history_update(E, p["hist"], p["present"], p["ema"], p["cap"], p["base"], float(f(0.2)), 15.0,
                                  float(f(0.98)), 1, None) == 0
    np.testing.assert_array_equal(d["hist"].cpu().numpy(), A.history)
    A.update_present_ema(0.40)
    assert lib.ogr_present_ema(E, p["present"], p["ema"], float(f(0.4)), float(f(0.6)), None) == 0
    np.testing.assert_array_equal(d["ema"].cpu().numpy(), A.present_ema)
    # an EMA value off the 2^-23 grid is flagged
    d["ema"][E // 2] = 1.0000001
    d["cap"][E // 2] = 0.3
    assert lib.ogr_tally(E, use.size, nz, p["present"], p["ema"], p["cap"], p["src"], p["dst"], p["layer"],
                         du.data_ptr(), 1, out.data_ptr(), units.data_ptr(), None) == 0
    assert (int(out[4]) != 0) == (float(np.float64(f(f(1.0000001) - f(0.3))) * 2 ** 23) % 1 != 0)
