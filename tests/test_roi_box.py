"""The box of an ROI search in shared memory (csrc/roibox.h), on the CPU: for any depth, up to 2^31 - 1 and below 0, it
lies in the lattice, holds both terminals and every cell that the search can reach, and its marks fit.  The same header
is what the kernels compile."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CAP = 41_000                       # about the words that a CTA has for the marks


@pytest.fixture(scope="module")
def fit(tmp_path_factory):
    d = tmp_path_factory.mktemp("roibox")
    (d / "box.cpp").write_text('#include "roibox.h"\nextern "C" void fit(const int* a, long long cap, int* out) {\n'
                               "  ogr_box::Box b = ogr_box::fit(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], cap);\n"
                               "  out[0] = b.x0; out[1] = b.y0; out[2] = b.w; out[3] = b.h; out[4] = b.row; out[5] = b.words;\n}\n")
    so = str(d / "box.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ftrapv", "-shared", "-fPIC",
                    "-I", os.path.join(ROOT, "orthoroute_gb300", "csrc"), str(d / "box.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    I8, I6 = ctypes.c_int * 8, ctypes.c_int * 6

    def call(nx, ny, nz, sx, sy, dx, dy, depth, cap=CAP):
        out = I6()
        lib.fit(I8(nx, ny, nz, sx, sy, dx, dy, depth), ctypes.c_longlong(cap), out)
        return list(out)
    return call


def words(nx, ny, nz, sx, sy, dx, dy, reach):
    """Unbounded integers: the box of `reach`, as the definition has it."""
    x0, x1 = max(0, min(sx, dx) - reach), min(nx - 1, max(sx, dx) + reach)
    y0, y1 = max(0, min(sy, dy) - reach), min(ny - 1, max(sy, dy) + reach)
    w, h = x1 - x0 + 1, y1 - y0 + 1
    return [x0, y0, w, h, (w + 15) // 16, (w + 15) // 16 * h * nz]


@pytest.mark.parametrize("depth", [-2**31, -1, 0, 1, 3, 80, 81, 1000, 10**6, 2**30, 2**31 - 120, 2**31 - 1])
def test_box_of_any_depth(fit, depth):
    rng = np.random.default_rng(abs(depth) % 1000)
    boards = [(600, 400, 12), (1000, 800, 32), (30, 25, 6), (1, 90, 6), (90, 1, 6), (1, 1, 1), (60_000, 30_000, 1),
              (2_000_000, 1_000, 1)]
    for nx, ny, nz in boards:
        for _ in range(6):
            sx, dx = (int(v) for v in rng.integers(0, nx, size=2))
            sy, dy = (int(v) for v in rng.integers(0, ny, size=2))
            a = (nx, ny, nz, sx, sy, dx, dy)
            got = fit(*a, depth)
            # the deepest reach that fits, by its definition; past max(nx, ny) the box does not grow
            top = min(max(depth, 0), max(nx, ny))
            lo, hi = -1, top
            while lo < hi:                       # (the words grow with the reach)
                mid = (lo + hi + 1) // 2
                if words(*a, mid)[5] <= CAP:
                    lo = mid
                else:
                    hi = mid - 1
            if lo < 0:
                assert got[5] == 0, (a, depth)
            else:
                assert got == words(*a, lo), (a, depth)
                assert 0 <= got[0] <= min(sx, dx) and max(sx, dx) < got[0] + got[2] <= nx
                assert 0 <= got[1] <= min(sy, dy) and max(sy, dy) < got[1] + got[3] <= ny


def test_box_of_no_limit_is_not_wrapped(fit):
    """Terminals (100, 100) and (150, 120) of 600x400x12 at a depth of 2^31 - 1, where the sums of a plain expression
    leave 32 bits on one axis before the other."""
    x0, y0, w, h, row, n = fit(600, 400, 12, 100, 100, 150, 120, 2**31 - 1)
    assert 0 < n <= CAP and n == row * h * 12 and w > 50 and h > 20


@pytest.mark.gpu
@pytest.mark.parametrize("depth", [-5, 0, 54, 56, 1000, 2**31 - 1])
def test_extraction_of_any_depth_matches_oracle(depth):
    """Depths past the lattice's sides (30 + 25) bound nothing; of 0 and less, the ROI is the terminals."""
    from oracle.roi import extract_roi_bfs
    from test_gpu_kernels import make
    g, s, ops, ref = make(30, 25, 6)
    rng = np.random.default_rng(8)
    for _ in range(4):
        src, dst = (int(v) for v in rng.choice(ref.plane, size=2, replace=False))
        want, _ = extract_roi_bfs(ref.indptr, ref.indices, g.N, src, dst, initial_radius=max(0, depth))
        got = ops.extract_roi(ops.net_args(0, src, dst, max_depth=depth, halo=2))
        np.testing.assert_array_equal(got, want)
