"""A batch's device memory comes from a pool of the call: more problems than
workers over several grid sizes give the same profiles whatever the number of
workers, also from two threads at once, and the memory is given back.

The solves are deterministic (fixed-order sums), so a worker's neighbours may
not change a bit of its result."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(probs, workers, precision=1):
    from tests.capi import batch_solve
    code, st, outs = batch_solve(probs, precision=precision, workers=workers)
    assert code == 0 and all(s.converged for s in st)
    return [np.array(o) for o in outs]


@pytest.mark.parametrize("precision", [0, 1])
def test_workers_do_not_change_results(precision):
    from deft_gb300.workloads import batch_sweep
    probs = batch_sweep(count=9, seed=11, sizes=(32, 48, 36))
    ref = _solve(probs, 1, precision)
    for workers in (3, 9):
        for a, b in zip(ref, _solve(probs, workers, precision)):
            assert np.array_equal(a, b)


def test_two_batches_at_once_and_memory_is_given_back():
    import torch
    from deft_gb300.workloads import batch_sweep
    probs = batch_sweep(count=6, seed=13, sizes=(32, 48))
    ref = _solve(probs, 2)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    got = [None, None]

    def run(i):
        got[i] = _solve(probs, 3)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for outs in got:
        for a, b in zip(ref, outs):
            assert np.array_equal(a, b)
    torch.cuda.synchronize()
    # the driver's own per-thread and per-module state may grow; one 48^3 problem
    # of these batches holds more than 20 MB
    assert torch.cuda.mem_get_info()[0] > free - (16 << 20)
