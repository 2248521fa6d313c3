"""CSR builds from via-partner lists of any kind: a layer named twice (with other sites and costs), the layer itself, lists
that do not ascend, and rows far longer than a lattice's.  The oracle is the rule of the row, written out per node:
partners before the first that is not below, laterals, partners above; the reverse arc is the first of the other row."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def ok(mode, x, y):
    return mode == 0 or (mode == 1 and (x + y) % 2 == 0) or (mode > 1 and x % mode == 0 and y % mode == 0)


def rows(nx, ny, nz, axis, partners, ww):
    """[(dst, cost, via)] of every node."""
    out = []
    for z in range(nz):
        for y in range(ny):
            for x in range(nx):
                n = (z * ny + y) * nx + x
                row = []
                for zz, c, m in partners[z]:
                    if zz >= z:
                        break
                    if ok(m, x, y):
                        row.append(((zz * ny + y) * nx + x, c, 1))
                h, v = axis[z] == 1 or (axis[z] and ww > 0), axis[z] == 2 or (axis[z] and ww > 0)
                ch, cv = (0.5 if axis[z] == 1 else ww), (0.5 if axis[z] == 2 else ww)
                if v and y > 0:
                    row.append((n - nx, cv, 0))
                if h and x > 0:
                    row.append((n - 1, ch, 0))
                if h and x + 1 < nx:
                    row.append((n + 1, ch, 0))
                if v and y + 1 < ny:
                    row.append((n + nx, cv, 0))
                row += [((zz * ny + y) * nx + x, c, 1) for zz, c, m in partners[z] if zz > z and ok(m, x, y)]
                out.append(row)
    return out


def build(nx, ny, nz, axis, partners, ww, device=False):
    from orthoroute_gb300 import _lib
    flat = [p for z in range(nz) for p in partners[z]]
    a = dict(axis=np.asarray(axis, np.uint8), ptr=np.cumsum([0] + [len(partners[z]) for z in range(nz)]).astype(np.int32),
             z=np.asarray([p[0] for p in flat] or [0], np.int32), c=np.asarray([p[1] for p in flat] or [0], np.float32),
             s=np.asarray([p[2] for p in flat] or [0], np.int32))
    d = _lib.LatticeDesc(nx, ny, nz, 0.5, ww, *(a[k].ctypes.data for k in ("axis", "ptr", "z", "c", "s")))
    lib = _lib.load()
    E = C.c_int64(0)
    _lib.check(lib.ogr_csr_num_edges(C.byref(d), C.byref(E)), "edges")
    t = lambda n, dt: torch.full((max(n, 1),), 77, dtype=dt, device="cuda")
    N = nx * ny * nz
    out = [t(N + 1, torch.int32), t(E.value, torch.int32), t(E.value, torch.float32), t(E.value, torch.uint8),
           t(E.value, torch.uint8), t(E.value, torch.int32), t(E.value, torch.int32)]
    nb = int(lib.ogr_csr_workspace_bytes(C.byref(d)))
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    rc = lib.ogr_csr_build(C.byref(d), *(v.data_ptr() for v in out), ws.data_ptr(), nb,
                           torch.cuda.current_stream().cuda_stream)
    _lib.check(rc, "ogr_csr_build")
    return out if device else [v.cpu().numpy() for v in out]


def build_device(*a):
    return build(*a, device=True)[0]


F = lambda v: float(np.float32(v))
LISTS = {
    "as a lattice has it": [[(1, 1.0, 0), (2, 1.5, 0)], [(0, 1.0, 0), (2, 1.0, 0)], [(0, 1.5, 0), (1, 1.0, 0), (3, 1.0, 0)],
                            [(2, 1.0, 0)]],
    "a layer twice, sites and costs apart": [[(1, 1.0, 2), (1, 2.0, 1), (2, 3.0, 0)], [(0, 1.0, 3), (0, 2.0, 0), (2, 1.0, 1), (2, 5.0, 2)],
                                             [(0, 3.0, 0), (1, 1.0, 0), (1, 2.0, 1)], []],
    "the layer itself": [[(0, 9.0, 0), (1, 1.0, 0)], [(0, 1.0, 0), (1, 9.0, 1), (2, 1.0, 0)], [(1, 1.0, 0), (2, 9.0, 0), (3, 1.0, 0)],
                         [(2, 1.0, 0), (3, 9.0, 2)]],
    "not ascending": [[(2, 1.0, 0), (1, 2.0, 0)], [(2, 1.0, 0), (0, 2.0, 0), (3, 3.0, 1)], [(3, 1.0, 0), (1, 2.0, 0), (0, 3.0, 0)],
                      [(2, 1.0, 0), (0, 1.0, 1), (1, 1.0, 0)]],
    "one way": [[(3, 1.0, 0)], [(0, 1.0, 0)], [(0, 1.0, 1), (1, 1.0, 2)], [(1, 1.0, 0)]],
    "rows of 100": [[(1 + k % 3, F(1 + k), k % 3) for k in range(96)], [(0, 1.0, 0)], [(0, 1.0, 0)], [(0, 1.0, 0)]],
    "rows of 900": [[(1 + k % 3, F(1 + k), 0) for k in range(896)], [(0, 1.0, 0)] * 40, [(0, 1.0, 0)], []],
    "rows of 3,000": [[(1 + k % 3, F(1 + k), 0) for k in range(2996)], [(0, 1.0, 0)], [(0, 1.0, 0)], []],
}


@pytest.mark.parametrize("name", LISTS)
@pytest.mark.parametrize("dims,ww", [((13, 11), -1.0), ((7, 9), 2.0), ((1, 5), 2.0)])
def test_csr_of_partner_lists(name, dims, ww):
    nx, ny = dims
    partners, axis = LISTS[name], [0, 1, 2, 1]
    want = rows(nx, ny, 4, axis, partners, ww)
    indptr, indices, cost, lay, kind, src, rev = build(nx, ny, 4, axis, partners, ww)
    ptr = np.cumsum([0] + [len(r) for r in want])
    np.testing.assert_array_equal(indptr, ptr)
    n = int(ptr[-1])
    flat = [(u, *a) for u, r in enumerate(want) for a in r]
    np.testing.assert_array_equal(src[:n], [a[0] for a in flat])
    np.testing.assert_array_equal(indices[:n], [a[1] for a in flat])
    np.testing.assert_array_equal(cost[:n], np.asarray([a[2] for a in flat], np.float32))
    np.testing.assert_array_equal(kind[:n], [a[3] for a in flat])
    np.testing.assert_array_equal(lay[:n], [a[0] // (nx * ny) for a in flat])
    back = [next((int(ptr[v]) + j for j, b in enumerate(want[v]) if b[0] == u), -1) for u, v, _, _ in flat]
    np.testing.assert_array_equal(rev[:n], back)


def test_a_layer_of_nearly_2_to_the_31_cells():
    """Steps from tile to tile and from row to row pass 2^31 behind the last ones: one layer without arcs (8.6 GB of row
    starts, all 0)."""
    indptr = build_device(46_340, 46_341, 1, [0], [[]], -1.0)
    assert indptr.numel() == 46_340 * 46_341 + 1
    assert int(indptr.min()) == 0 and int(indptr.max()) == 0
