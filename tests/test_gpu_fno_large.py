"""Networks beyond the slab kernels' shared memory (which ends between N = 136 and
160, by the modes): the z and y transforms as kernels of their own, and the layer
kernel that takes the z synthesis alone.  One size of each register tile of modes
whose last tile of lines is not full; launches a forward pass tell which kernels
ran.

Tolerances as in test_gpu_fno_slab.py: FP32 sums of at most 164 products an axis,
2e-5 of the field's scale and ten times that for the gradient."""
import numpy as np
import pytest

from . import fno_reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,m,slab", [(164, 3, False), (156, 7, False), (148, 12, False),
                                      (140, 16, False), (144, 12, True)])
def test_forward_and_gradient(N, m, slab):
    from deft_gb300.warmstart import FourierOperator
    C, L = 4, 1
    net = FourierOperator(N=N, channels=C, modes=m, layers=L, seed=5)
    try:
        rng = np.random.default_rng(N + m)
        p = (net.get_params() + 0.05 * rng.standard_normal(net.nparam)).astype(np.float32)
        net.set_params(p)
        mask = (rng.random(N ** 3) > 0.3).astype(np.float32)
        target = (mask * (1 + 0.3 * rng.standard_normal(N ** 3))).astype(np.float32)
        before = net.L.deft_fno_launches(net.h)
        y0, _, _ = net.eval(mask, 0.31)
        # lift, projection and, a layer, analysis (1 or 2), x, mixing, x, synthesis (1 or 2)
        assert net.L.deft_fno_launches(net.h) - before == (2 + 5 if slab else 2 + 7)
        y, loss, grad = net.eval(mask, 0.31, target, want_grad=True)
        loss_r, y_r, grad_r = ref.loss_and_grad(p, mask, 0.31, target, N, C, m, L)
        sy, sg = np.abs(y_r).max(), np.abs(grad_r).max()
        print(f"N {N} m {m}: inference {np.abs(y0 - y_r).max() / sy:.1e} training "
              f"{np.abs(y - y_r).max() / sy:.1e} grad {np.abs(grad - grad_r).max() / sg:.1e}")
        assert np.abs(y0 - y_r).max() <= 2e-5 * sy
        assert np.abs(y - y_r).max() <= 2e-5 * sy
        assert abs(loss / loss_r - 1) <= 2e-5
        assert np.abs(grad - grad_r).max() <= 2e-4 * sg
    finally:
        net.close()
