"""Points of the tensor and water functionals that take the FP64 formulas:
nearly empty space next to a liquid (weighted densities below 1e-9), a fluid as
dilute everywhere, and one packed to 1 - n3 = 2^-21, a trial point that a line
search may reach.

Tolerances.  Next to a liquid: 2^-42 of the largest entry, as for the liquid.
Dilute: the oracle's and these formulas' ln(1 - n3) is rounded to 2^-53 / n3 of
itself, which the association term sees whole.  Packed: n3 comes from
double-float transforms, 2^-46 of 1, and the leading terms go as (1 - n3)^-3: 3 x
2^-46 / 2^-21 = 2^-23."""
import math

import numpy as np
import pytest

from deft_gb300 import _lib

pytestmark = pytest.mark.gpu
KINDS = [_lib.HS_WB_NOTENSOR, _lib.HS_RF, _lib.HS_WB_MARK2, _lib.HS_WB_TENSOR,
         _lib.HS_TARAZONA, "water"]


@pytest.fixture(scope="module")
def ctx():
    from tests.capi import Ctx
    c = Ctx(0)
    yield c
    c.close()


def _both(ctx, O, kind, dx, N, n):
    """Energy and gradient here and by the oracle; lengths in units of R."""
    from tests.capi import Fmt, Grid
    from tests.golden.cases import WATER_KT, WATER_R, WATER_SAFT
    water = kind == "water"
    R, kT = (WATER_R, WATER_KT) if water else (1.0, 1.0)
    lat = np.diag([dx * R * v for v in N])
    n = n / R ** 3
    terms = _lib.TERM_HS | _lib.TERM_IDEAL | (_lib.TERM_SAFT if water else 0)
    g = Grid(ctx, lat, N)
    f = Fmt(g, R=R, kT=kT, terms=terms, functional=0 if water else kind)
    if water:
        sp = np.array(WATER_SAFT)
        _lib.check(f.L.deft_fmt_set_saft(f.h, sp.ctypes.data))
    P = O.Problem(lat, N, R=R, kT=kT, terms=O.HS | O.IDEAL, hs=0 if water else kind,
                  saft=WATER_SAFT if water else None)
    Er, gr = P.energy_grad(n)
    E, grad, _ = f.energy_grad(n)
    f.close()
    g.close()
    return E, grad.reshape(N), Er, gr.reshape(N)


def _report(kind, E, grad, Er, gr, where=None):
    where = np.ones(gr.shape, bool) if where is None else where
    d, s = (grad - gr)[where], gr[where]
    e, worst, norm = abs(E / Er - 1), np.abs(d).max() / np.abs(s).max(), \
        np.linalg.norm(d) / np.linalg.norm(s)
    print(f"{kind}: |dE/E| {e:.1e}, gradient {worst:.1e}, 2-norm {norm:.1e}")
    return e, worst, norm


@pytest.mark.parametrize("kind", KINDS)
def test_beside_a_liquid(ctx, oracle_mod, kind):
    """Half the box at 1e-14 of the liquid: beyond two radii from it the weighted
    densities are as small, and every point there takes the FP64 formulas."""
    N = (8, 8, 64)
    rng = np.random.default_rng(3)
    n = 0.3 / (4 * math.pi / 3) * (1 + 0.02 * rng.standard_normal(N))
    if kind == "water":
        n *= 0.35 / 0.3  # 0.0049 a molecule
    n[:, :, 20:44] *= 1e-14
    E, grad, Er, gr = _both(ctx, oracle_mod, kind, 0.4, N, n)
    liquid = np.zeros(N, bool)
    liquid[:, :, :20] = liquid[:, :, 44:] = True
    assert np.all(np.isfinite(grad))
    e, worst, _ = _report(kind, E, grad, Er, gr)
    le, lworst, lnorm = _report(f"{kind}, liquid", E, grad, Er, gr, liquid)
    tol = 2.0 ** -42
    assert e <= tol and lworst <= tol and lnorm <= tol
    # water divides by the shell density, which there is the transforms' rounding
    assert worst <= tol or kind == "water"


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n3", [3e-10, 1e-12])
def test_dilute(ctx, oracle_mod, kind, n3):
    N = (12, 10, 14)
    rng = np.random.default_rng(5)
    n = n3 / (4 * math.pi / 3) * (1 + 0.1 * rng.standard_normal(N)).clip(0.5)
    E, grad, Er, gr = _both(ctx, oracle_mod, kind, 0.3, N, n)
    e, worst, _ = _report(kind, E, grad, Er, gr)
    tol = 2.0 ** -42 + (4 * 2.0 ** -53 / n3 if kind == "water" else 0)
    assert e <= tol and worst <= tol


@pytest.mark.parametrize("kind", KINDS)
def test_packed(ctx, oracle_mod, kind):
    N = (12, 10, 14)
    n = np.full(N, (1 - 2.0 ** -21) / (4 * math.pi / 3))
    E, grad, Er, gr = _both(ctx, oracle_mod, kind, 0.3, N, n)
    e, worst, _ = _report(kind, E, grad, Er, gr)
    assert e <= 2.0 ** -23 and worst <= 2.0 ** -23


@pytest.mark.parametrize("N", [(7, 11, 13), (12, 20, 14), (16, 16, 48)])
def test_water_liquid(ctx, oracle_mod, N):
    """Around a cavity of 1e-5 of the liquid the liquid's entries are as exact as a
    liquid's alone."""
    rng = np.random.default_rng(sum(N))
    n = 0.35 / (4 * math.pi / 3) * (1 + 0.1 * rng.standard_normal(N)).clip(0.3)
    n[: N[0] // 3, : N[1] // 3] = 1e-5 * 0.35 / (4 * math.pi / 3)
    E, grad, Er, gr = _both(ctx, oracle_mod, "water", 0.2, N, n)
    liquid = np.ones(N, bool)
    liquid[: N[0] // 3, : N[1] // 3] = False
    e, worst, norm = _report("water", E, grad, Er, gr, liquid)
    assert e <= 2.0 ** -42 and worst <= 2.0 ** -42 and norm <= 2.0 ** -42
