"""The FP32 transforms: plans that run pairs of small radices as one pass of 10,
12 or 16, the two-pass kernels of the y and x axes (every length they take, and
column counts that leave part of the last block empty), and the z kernels that
read their pointwise inputs in rounds of four.  The mixed form's energy and
gradient against the FP64 form of the same state, by the built-in kernels, by
the shared-memory passes, and by orders in which no pair is fused.

Tolerance: an FP32 transform of N = Nx Ny Nz points rounds with a relative rms
of about 2^-24 sqrt(log2 N) < 3e-7 of its largest output, five times in a row
(three axes forward, three back, twice) with Phi's derivative (condition below
10 at eta = 0.3) between them: below 1.5e-5 of the largest gradient.  A wrong
index or root changes it by order one."""
import numpy as np
import pytest

from deft_gb300 import _lib

pytestmark = pytest.mark.gpu


def _state(shape, precision):
    from tests.capi import Ctx, Fmt, Grid
    rng = np.random.default_rng(17)
    lat = np.ascontiguousarray(np.diag(0.2 * np.array(shape, dtype=float)))
    ctx = Ctx(0)
    g = Grid(ctx, lat, shape)
    mask = np.ones(shape)
    mask[:, :, :2] = 0.0
    n = 0.3 * 6 / (8 * np.pi) * (1 + 0.3 * rng.random(shape)) * mask
    f = Fmt(g, R=1.0, kT=1.0, mu=1.0, terms=_lib.TERM_HS | _lib.TERM_IDEAL | _lib.TERM_MU |
            _lib.TERM_MASK, mask=mask.reshape(-1), precision=precision)
    return ctx, g, f, n.reshape(-1)


def _orders(g):
    t = np.zeros(6, dtype=np.int32)
    r = np.zeros(24, dtype=np.int32)
    _lib.check(g.L.deft_grid_get_tiles(g.h, 1, t.ctypes.data, r.ctypes.data))
    return t, r


# (x, y, z) lengths: 10, 12 and 16 alone, first, last and with every other
# radix; odd line counts (a half pair); a third pass after a fused one
@pytest.mark.parametrize("shape,plain", [
    ((10, 12, 16), ([5, 2], [3, 4], [8, 2])),
    ((12, 20, 10), ([3, 2, 2], [4, 5], [5, 2])),
    ((48, 10, 40), ([4, 3, 4], [2, 5], [8, 5])),
    ((5, 7, 48), ([5], [7], [8, 3, 2])),
    ((9, 48, 96), ([3, 3], [8, 2, 3], [4, 8, 3])),
    ((96, 5, 80), ([4, 8, 3], [5], [2, 8, 5])),
    ((3, 100, 36), ([3], [5, 4, 5], [3, 3, 4])),
    ((2, 3, 480), ([2], [3], [8, 3, 4, 5])),
])
def test_fused_passes(shape, plain, monkeypatch):
    monkeypatch.setenv("DEFT_PENCIL", "0")  # the shared-memory passes on every axis
    tol = 1.5e-5
    ctx, g, f, n = _state(shape, 0)
    try:
        E64, g64, _ = f.energy_grad(n)
    finally:
        f.close(), g.close(), ctx.close()
    ctx, g, f, n = _state(shape, 1)
    try:
        t, r = _orders(g)
        for a in range(3):
            o = [int(v) for v in r[8 * a:8 * a + 8] if v]
            assert np.prod(o) == shape[a] and max(o) <= 13  # orders stay in plain radices
        assert g.L.deft_grid_set_tiles(g.h, 1, t.ctypes.data, r.ctypes.data) == 0
        results = [f.energy_grad(n)]
        r2 = np.zeros(24, dtype=np.int32)
        for a in range(3):
            r2[8 * a:8 * a + len(plain[a])] = plain[a]
        assert g.L.deft_grid_set_tiles(g.h, 1, t.ctypes.data, r2.ctypes.data) == 0
        assert np.array_equal(_orders(g)[1], r2)
        results.append(f.energy_grad(n))
        for E, gr, _ in results:
            assert abs(E / E64 - 1) < tol
            assert np.abs(gr - g64).max() <= tol * np.abs(g64).max()
    finally:
        f.close(), g.close(), ctx.close()


@pytest.mark.parametrize("n", [32, 36, 40, 48, 50, 60, 64, 72, 80, 96, 100, 120, 128, 144, 160,
                               192, 256])
@pytest.mark.parametrize("axis", [0, 1])
def test_two_pass_lengths(n, axis):
    tol = 1.5e-5
    shape = [3, 5, 6]  # 20 or 12 columns: fewer than a block's
    shape[axis] = n
    if n == 48:
        shape[1 - axis] = 11  # 44 columns: two blocks of 32, the second part full
    out = []
    for precision in (0, 1):
        ctx, g, f, x = _state(tuple(shape), precision)
        try:
            out.append(f.energy_grad(x))
        finally:
            f.close(), g.close(), ctx.close()
    assert abs(out[1][0] / out[0][0] - 1) < tol
    assert np.abs(out[1][1] - out[0][1]).max() <= tol * np.abs(out[0][1]).max()
