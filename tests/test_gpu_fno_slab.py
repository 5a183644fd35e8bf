"""The network's slab kernels (z and y transforms of an N x N slab in one block,
the inference layer fused with both) where their loops end: N = 4 and 0 mod 8,
lines that do not fill a warp, every register tile of modes, several lines a
block pass and one, and N = 152, which takes the kernels without slabs.

Tolerances: FP32 sums of at most 152 products an axis, three axes and a few
layers: sqrt(3 layers 152) 2^-24 of the field's scale is 2e-6; 2e-5 allowed, ten
times that for the gradient (sums over the points on top)."""
import numpy as np
import pytest

from . import fno_reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,C,m,L", [(4, 4, 1, 1), (12, 8, 5, 2), (24, 4, 3, 2), (36, 8, 16, 1),
                                     (40, 16, 9, 2), (60, 4, 12, 2), (68, 16, 4, 1),
                                     (152, 4, 3, 1)])
def test_forward_and_gradient(N, C, m, L):
    from deft_gb300.warmstart import FourierOperator
    net = FourierOperator(N=N, channels=C, modes=m, layers=L, seed=5)
    try:
        rng = np.random.default_rng(N + m)
        p = (net.get_params() + 0.05 * rng.standard_normal(net.nparam)).astype(np.float32)
        net.set_params(p)
        mask = (rng.random(N ** 3) > 0.3).astype(np.float32)
        target = (mask * (1 + 0.3 * rng.standard_normal(N ** 3))).astype(np.float32)
        y0, _, _ = net.eval(mask, 0.31)
        y, loss, grad = net.eval(mask, 0.31, target, want_grad=True)
        loss_r, y_r, grad_r = ref.loss_and_grad(p, mask, 0.31, target, N, C, m, L)
        sy, sg = np.abs(y_r).max(), np.abs(grad_r).max()
        print(f"N {N} C {C} m {m}: inference {np.abs(y0 - y_r).max() / sy:.1e} training "
              f"{np.abs(y - y_r).max() / sy:.1e} grad {np.abs(grad - grad_r).max() / sg:.1e}")
        assert np.abs(y0 - y_r).max() <= 2e-5 * sy
        assert np.abs(y - y_r).max() <= 2e-5 * sy
        assert abs(loss / loss_r - 1) <= 2e-5
        assert np.abs(grad - grad_r).max() <= 2e-4 * sg
    finally:
        net.close()
