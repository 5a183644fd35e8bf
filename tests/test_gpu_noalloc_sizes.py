"""The allocation-free entry point takes every grid whose arrays fit its fixed
scratch, up to the last bytes: the largest of these shapes need all but 0.3 to
7 KB of the 20 MiB with energy partials of the widest Phi tiles.

Tolerance: the two entry points add up the same FP64 terms in other orders and
transform in FP64 and double-float (2^-46 a step): 1e-11 of the largest entry."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [(32, 176, 60), (88, 64, 60), (8, 216, 200), (64, 64, 64)])
def test_largest_shapes(N):
    import torch
    from deft_gb300 import _lib
    from tests.capi import Ctx, Fmt, Grid
    L = _lib.load()
    lat = np.diag([0.2 * v for v in N])
    rng = np.random.default_rng(sum(N))
    n = 0.3 / (4 * math.pi / 3) * (1 + 0.05 * rng.standard_normal(N)).clip(0.5)
    terms = _lib.TERM_HS | _lib.TERM_IDEAL | _lib.TERM_MU
    p = _lib.FmtParams(1.0, 1.0, 0.3, terms, 0, 0)
    lat9 = np.ascontiguousarray(lat.reshape(9))
    nd = torch.tensor(n, device="cuda")
    grad = torch.empty_like(nd)
    E = ctypes.c_double()
    torch.cuda.synchronize()
    _lib.check(L.deft_fmt_energy_grad_noalloc(
        lat9.ctypes.data, *N, ctypes.byref(p), nd.data_ptr(), None, None, ctypes.addressof(E),
        grad.data_ptr(), None, None))
    ctx = Ctx(0)
    g = Grid(ctx, lat, N)
    f = Fmt(g, mu=0.3, terms=terms)
    Er, gr, _ = f.energy_grad(n)
    for c in (f, g, ctx):
        c.close()
    assert abs(E.value / Er - 1) <= 1e-11
    err = np.abs(grad.cpu().numpy().reshape(-1) - gr).max() / np.abs(gr).max()
    print(f"{N}: gradient {err:.1e}")
    assert err <= 1e-11
