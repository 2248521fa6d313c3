"""Cost updates of more than 2^31 arcs (the count is 64-bit), and EMA overuse at the top of the tally's range, bit for bit
against numpy."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1])      # four arcs at a time, and one by one
def test_jitter_of_arcs_past_2_to_the_31(off):
    """Every array that is only read is one and the same (1.0 an arc): 19 GB in all."""
    from orthoroute_gb300 import _lib
    E = 2 ** 31 + 1029
    ones = torch.ones(E + 8, dtype=torch.float32, device="cuda")[off:]
    zero = torch.zeros(E + 8, dtype=torch.uint8, device="cuda")[off:]
    total = torch.zeros(E + 8, dtype=torch.float32, device="cuda")[off:]
    p, z = ones.data_ptr(), zero.data_ptr()
    a = _lib.CostArgs(E, p, z, z, p, p, p, None, None, 1.0, 1.0, 1.0, 0.0, 1)
    _lib.check(_lib.load().ogr_costs_update(C.byref(a), total.data_ptr(), None), "ogr_costs_update")
    for at in (0, 5_000_011, 2 ** 24 - 500, 2 ** 30 - 3, 2 ** 31 - 1000, 2 ** 31 - 2, E - 1000):
        n = min(1000, E - at)
        e = np.arange(at, at + n, dtype=np.int64).astype(np.float32)
        want = np.float32(1.0) + (e % np.float32(9973.0)) * np.float32(1e-6)
        np.testing.assert_array_equal(total[at:at + n].cpu().numpy(), want, err_msg=str(at))
    assert float(total[E:].sum()) == 0.0


@pytest.mark.parametrize("ema", [1.0, 2.0 ** 39, 2.0 ** 40, 2.0 ** 40 * 1.5, 2.0 ** 41 - 2.0 ** 17, 2.0 ** 41, 3.0e38, np.inf,
                                 2.0 ** -23, 2.0 ** -24, 1e-40])
@pytest.mark.parametrize("off", [0, 1])
def test_tally_takes_what_64_bits_hold(ema, off):
    """One overused arc: its units of 2^-23 are exact below 2^64, and told as inexact from there on."""
    from orthoroute_gb300 import _lib
    E, nz = 37, 3
    f = lambda v, dt=torch.float32: torch.full((E + 8,), v, dtype=dt, device="cuda")[off:off + E]
    present, em, cap, src, dst = f(0), f(0), f(0), f(0, torch.int32), f(1, torch.int32)
    layer = f(2, torch.uint8)
    em[17] = float(np.float32(ema))
    use = torch.zeros(30, dtype=torch.int32, device="cuda")
    out = torch.zeros(5, dtype=torch.int64, device="cuda")
    units = torch.zeros(nz, dtype=torch.int64, device="cuda")
    p = lambda t: t.data_ptr()
    assert _lib.load().ogr_tally(E, use.numel(), nz, p(present), p(em), p(cap), p(src), p(dst), p(layer), p(use), 1, p(out),
                                 p(units), None) == 0
    want = float(np.float32(ema)) * 2.0 ** 23
    exact = want < 2.0 ** 64 and want == np.floor(want)
    assert (int(out[4]) != 0) == (not exact)
    if exact:
        assert [int(v) & (2 ** 64 - 1) for v in units] == [0, 0, int(want)]
