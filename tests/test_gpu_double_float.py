"""The FP64 form's double-float kernels against the FP64 oracle where their
branches meet: Phi in every density regime (dilute fluids, the series below
n3 = 1/32 and 1/16, dense fluids, empty walls) for each hard-sphere kind, and
the x and y transforms at the lengths their register form takes and at odd
and prime-factor lengths.

Tolerances.  A double-float operation rounds at 2^-47 or better and Phi's
longest chains are some tens of them: 2^-42 of a partial's largest term.  The
oracle's own ln(1 - n3) is FP64's, whose argument is rounded to 2^-53, i.e. to
2^-53 / n3 of the logarithm; dilute cases allow four of those."""
import math

import numpy as np
import pytest

from deft_gb300 import _lib

pytestmark = pytest.mark.gpu

KINDS = [_lib.HS_WB_NOTENSOR, _lib.HS_RF, _lib.HS_WB_MARK2]


@pytest.fixture(scope="module")
def ctx():
    from tests.capi import Ctx
    c = Ctx(0)
    yield c
    c.close()


def _check(ctx, O, lat, N, n, kind, n3, R=1.0, kT=1.0):
    from tests.capi import Fmt, Grid
    g = Grid(ctx, lat, N)
    f = Fmt(g, R=R, kT=kT, terms=O.HS, functional=kind)
    E, grad, terms = f.energy_grad(n)
    P = O.Problem(lat, N, R=R, kT=kT, terms=O.HS, hs=kind)
    Er, gr = P.energy_grad(n)
    tol = 2.0 ** -42 + 4 * 2.0 ** -53 / n3
    print(f"kind {kind} N {N} n3 {n3:.3g}: |dE/E| {abs(E / Er - 1):.2e} "
          f"grad {np.abs(grad.reshape(-1) - gr.reshape(-1)).max() / np.abs(gr).max():.2e} "
          f"(allowed {tol:.2e})")
    assert abs(E / Er - 1) <= tol
    assert np.abs(grad.reshape(-1) - gr.reshape(-1)).max() <= tol * np.abs(gr).max()
    f.close()
    g.close()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n3", [1e-12, 1e-7, 1e-3, 1 / 32, 1 / 16, 0.25, 0.48])
def test_phi_regimes(ctx, oracle_mod, kind, n3):
    N, lat = (12, 10, 14), np.diag([2.4, 2.0, 2.8])
    rng = np.random.default_rng(int(1e6 * n3) + kind)
    n = n3 / (4 * math.pi / 3) * (1 + 0.1 * rng.standard_normal(N))
    _check(ctx, oracle_mod, lat, N, n.clip(0.5 * n3 / (4 * math.pi / 3)), kind, n3)


@pytest.mark.parametrize("kind", KINDS)
def test_phi_walls(ctx, oracle_mod, kind):
    """Empty walls (n = 0) beside a dense fluid, non-unit R and kT."""
    N, lat = (9, 8, 64), np.diag([1.8, 1.6, 12.8])
    rng = np.random.default_rng(5)
    n = 0.3 / (4 * math.pi / 3) / 0.8 ** 3 * (1 + 0.05 * rng.standard_normal(N))
    n[:, :, 30:] = 0.0
    _check(ctx, oracle_mod, lat, N, n, kind, 0.3, R=0.8, kT=1.7)


@pytest.mark.parametrize("N", [(32, 32, 32), (64, 32, 15), (32, 64, 9), (128, 32, 6), (32, 128, 7),
                               (256, 32, 4), (32, 256, 4), (33, 64, 10), (64, 30, 11),
                               (26, 49, 22), (143, 16, 7), (16, 77, 169)])
def test_transform_lengths(ctx, oracle_mod, N):
    """Lengths 32 to 256 along x and y (and neighbours that are not), columns
    that do not fill a group, prime factors 7, 11 and 13 on each axis."""
    lat = np.array([[0.2 * N[0], 0.1, 0.0], [0.0, 0.2 * N[1], 0.2], [0.3, 0.0, 0.25 * N[2]]])
    rng = np.random.default_rng(sum(N))
    n = 0.2 / (4 * math.pi / 3) * (1 + 0.2 * rng.standard_normal(N)).clip(0.1)
    _check(ctx, oracle_mod, lat, N, n, _lib.HS_WB_NOTENSOR, 0.2)


@pytest.mark.parametrize("kind", [_lib.HS_WB_TENSOR, _lib.HS_TARAZONA])
@pytest.mark.parametrize("N,n3", [((7, 11, 13), 0.3), ((16, 9, 25), 1 / 32), ((33, 8, 12), 1e-8),
                                  ((1, 1, 64), 0.4)])
def test_tensor_sets(ctx, oracle_mod, kind, N, n3):
    """The eleven convolutions and their adjoints on odd, prime and
    one-dimensional grids, each branch of the third term, with empty walls
    where the fluid is dense."""
    lat = np.array([[0.2 * N[0], 0.1, 0.0], [0.0, 0.2 * N[1], 0.1], [0.1, 0.0, 0.2 * N[2]]])
    rng = np.random.default_rng(N[0] + kind)
    n = n3 / (4 * math.pi / 3) * (1 + 0.1 * rng.standard_normal(N)).clip(0.5)
    if n3 > 0.1:
        n[:, :, N[2] // 2:] = 0.0
    _check(ctx, oracle_mod, lat, N, n, kind, n3)


@pytest.mark.parametrize("N", [(7, 11, 13), (16, 9, 25), (12, 20, 14)])
def test_water_sets(ctx, oracle_mod, N):
    """The water terms around a nearly empty cavity (1e-5 of the liquid): their
    energy and gradient against the oracle's.  The pass has some hundred
    double-float operations in a row and divides by the shell density, which
    falls to 1e-3 of the liquid's in the cavity: 2^-42 / 1e-3 of the largest
    entry."""
    from tests.capi import Fmt, Grid
    from tests.golden.cases import WATER_KT, WATER_N, WATER_R, WATER_SAFT
    O = oracle_mod
    lat = np.diag([0.6 * v for v in N])
    rng = np.random.default_rng(sum(N))
    n = WATER_N * (1 + 0.1 * rng.standard_normal(N)).clip(0.3)
    n[: N[0] // 3, : N[1] // 3] = 1e-5 * WATER_N
    P = O.Problem(lat, N, R=WATER_R, kT=WATER_KT, mu=0.01, terms=O.HS | O.IDEAL | O.MU,
                  saft=WATER_SAFT)
    Er, gr = P.energy_grad(n)
    g = Grid(ctx, lat, N)
    f = Fmt(g, R=WATER_R, kT=WATER_KT, mu=0.01,
            terms=_lib.TERM_HS | _lib.TERM_IDEAL | _lib.TERM_MU | _lib.TERM_SAFT)
    sp = np.array(WATER_SAFT)
    _lib.check(f.L.deft_fmt_set_saft(f.h, sp.ctypes.data))
    E, grad, _ = f.energy_grad(n)
    err = np.abs(grad.reshape(-1) - gr.reshape(-1)).max() / np.abs(gr).max()
    print(f"N {N}: |dE/E| {abs(E / Er - 1):.2e} grad {err:.2e}")
    assert abs(E / Er - 1) <= 2.0 ** -42 and err <= 2.0 ** -42 * 1e3
    f.close()
    g.close()
