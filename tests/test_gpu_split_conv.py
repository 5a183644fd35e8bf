"""The forward convolution along x with a block per tile and field (grids whose
tiles are no more than the SMs) and with all five fields in one block (larger
grids): energy and gradient of the double-float form against FP64 transforms
(DEFT_FP64_TRANSFORMS=fp64) and of the mixed form against the same.

Shapes: one tile, a part-filled last tile, tile counts around the 148 to 160 SMs
of the device (16 columns a tile).  Tolerances: double-float transforms carry
2^-46 a step, below 1e-11 of the largest gradient after some 60 steps and Phi's
condition (below 10); FP32 as in test_gpu_fused_radix.py."""
import numpy as np
import pytest

from deft_gb300 import _lib

pytestmark = pytest.mark.gpu


def _run(shape, precision):
    from tests.capi import Ctx, Fmt, Grid
    rng = np.random.default_rng(23)
    lat = np.ascontiguousarray(np.diag(0.2 * np.array(shape, dtype=float)))
    ctx = Ctx(0)
    g = Grid(ctx, lat, shape)
    n = 0.3 * 6 / (8 * np.pi) * (1 + 0.3 * rng.random(shape))
    f = Fmt(g, R=1.0, kT=1.0, mu=1.0, terms=_lib.TERM_HS | _lib.TERM_IDEAL | _lib.TERM_MU,
            precision=precision)
    try:
        E, gr, _ = f.energy_grad(n.reshape(-1))
        return E, np.array(gr)
    finally:
        f.close(), g.close(), ctx.close()


@pytest.mark.parametrize("shape", [
    (6, 3, 4),      # 9 columns, one tile
    (14, 10, 12),   # 70 columns, a part-filled tile
    (22, 64, 72),   # 2368 columns: 148 tiles
    (22, 65, 72),   # 2405 columns: 151
    (22, 66, 72),   # 2442 columns: 153
    (22, 70, 72),   # 2590 columns: 162
    (7, 128, 44),   # 2944 columns: 184
])
def test_split_forward_convolution(shape, monkeypatch):
    E, gr = _run(shape, 0)
    Em, grm = _run(shape, 1)
    monkeypatch.setenv("DEFT_FP64_TRANSFORMS", "fp64")
    E64, g64 = _run(shape, 0)
    top = np.abs(g64).max()
    assert abs(E / E64 - 1) < 1e-11
    assert np.abs(gr - g64).max() <= 1e-11 * top
    assert abs(Em / E64 - 1) < 1.5e-5
    assert np.abs(grm - g64).max() <= 1.5e-5 * top
