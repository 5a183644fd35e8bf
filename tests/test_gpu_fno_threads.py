"""Networks of different sizes share their kernels' functions, not each other's
launch settings: each gives the bits it gives alone, with the other created
after it and with both at work in two threads."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _net(N, C, m, L):
    from deft_gb300.warmstart import FourierOperator
    rng = np.random.default_rng(N)
    net = FourierOperator(N=N, channels=C, modes=m, layers=L, seed=N)
    mask = (rng.random(N ** 3) > 0.3).astype(np.float32)
    target = (mask * (1 + 0.3 * rng.standard_normal(N ** 3))).astype(np.float32)
    return net, mask, target


# kernels that need different amounts of shared memory above a block's 48 KB, or one
# above and one below, with the slab kernels and (N > 148) without
@pytest.mark.parametrize("big,small", [((24, 16, 12, 4), (40, 16, 11, 4)),
                                       ((192, 4, 8, 1), (152, 4, 7, 1))])
def test_two_sizes(big, small):
    nets, ref = [], []
    try:
        for size in (big, small):
            nets.append(_net(*size))
        for net, mask, target in nets:
            y, loss, grad = net.eval(mask, 0.3, target, want_grad=True)
            ref.append((net.eval(mask, 0.3)[0].copy(), y.copy(), loss, grad.copy()))
        bad = []

        def work(i):
            net, mask, target = nets[i]
            try:
                for k in range(400):
                    y0 = net.eval(mask, 0.3)[0]
                    if not np.array_equal(y0, ref[i][0]):
                        bad.append("network %d: another inference" % i)
                    if k % 40 or bad:
                        continue
                    y, loss, grad = net.eval(mask, 0.3, target, want_grad=True)
                    if not (np.array_equal(y, ref[i][1]) and loss == ref[i][2]
                            and np.array_equal(grad, ref[i][3])):
                        bad.append("network %d: other values" % i)
            except Exception as e:  # noqa: BLE001
                bad.append("network %d: %s" % (i, e))

        threads = [threading.Thread(target=work, args=(i,)) for i in (0, 1)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad, bad[:3]
    finally:
        for net, _, _ in nets:
            net.close()
