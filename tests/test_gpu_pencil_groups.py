"""The double-float register transforms along x and y where the columns do not
fill the last group of 32: in place along y, forward and adjoint along x, with a
block for a column group's five fields and with one a field.

Tolerance as in test_gpu_double_float.py: 2^-42 of the largest entry and four
roundings of the oracle's logarithm."""
import ctypes
import math

import numpy as np
import pytest

from deft_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from tests.capi import Ctx
    c = Ctx(0)
    yield c
    c.close()


def _launches(L, g):
    out = {}
    for i in range(L.deft_grid_profile_count(g.h)):
        name, launches, ms = ctypes.c_char_p(), ctypes.c_longlong(), ctypes.c_double()
        _lib.check(L.deft_grid_profile_entry(g.h, i, ctypes.byref(name), ctypes.byref(launches),
                                             ctypes.byref(ms)))
        out[name.value.decode()] = launches.value
    return out


# x of 64, 128 and 256 with Ny (Nz / 2 + 1) = 19, 19, 22 and 22 mod 32, few and many
# columns; y of 64, 32 and 256 with Nx (Nz / 2 + 1) = 19, 10 and 11 mod 32
@pytest.mark.parametrize("N,split", [((64, 45, 60), True), ((128, 45, 60), True),
                                     ((128, 75, 130), False), ((256, 75, 66), False),
                                     ((45, 64, 60), None), ((150, 32, 60), None),
                                     ((33, 256, 20), None)])
def test_part_filled_groups(ctx, oracle_mod, monkeypatch, N, split):
    from tests.capi import Fmt, Grid
    O = oracle_mod
    lat = np.array([[0.2 * N[0], 0.1, 0.0], [0.0, 0.2 * N[1], 0.2], [0.3, 0.0, 0.25 * N[2]]])
    rng = np.random.default_rng(sum(N))
    n = 0.2 / (4 * math.pi / 3) * (1 + 0.2 * rng.standard_normal(N)).clip(0.1)
    got = {}
    for pencil in ("1", "0"):
        monkeypatch.setenv("DEFT_PENCIL", pencil)
        g = Grid(ctx, lat, N)
        f = Fmt(g, terms=O.HS)
        g.L.deft_grid_profile(g.h, 0)
        got[pencil] = f.energy_grad(n)
        adjoints = _launches(g.L, g)["x_conv_adj"]
        if split is not None:  # the split adjoint is two launches
            assert adjoints == (2 if split and pencil == "1" else 1)
        f.close()
        g.close()
    # another path than the shared-memory passes ran
    assert not np.array_equal(got["1"][1], got["0"][1])
    tol = 2.0 ** -42 + 4 * 2.0 ** -53 / 0.2
    Er, gr = O.Problem(lat, N, terms=O.HS).energy_grad(n)
    for k in ("1", "0"):
        E, grad, _ = got[k]
        err = np.abs(grad - gr.reshape(-1)).max() / np.abs(gr).max()
        print(f"{N} pencils {k}: |dE/E| {abs(E / Er - 1):.1e} grad {err:.1e}")
        assert abs(E / Er - 1) <= tol and err <= tol
