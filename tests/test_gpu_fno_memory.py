"""A network on a slab grid holds no coefficients between its z and y axes (the
slab kernels keep them on the chip): its device memory is that of its
parameters, tables and fields.

16 MiB are left for the allocator's pages and the library's kernels; the
coefficients would be 30 MiB."""
import pytest

pytestmark = pytest.mark.gpu


def test_slab_grid_memory():
    import torch
    from deft_gb300.warmstart import FourierOperator
    N, C, m, L = 144, 16, 12, 1
    FourierOperator(N=N, channels=C, modes=m, layers=L, seed=1).close()  # kernels loaded
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    net = FourierOperator(N=N, channels=C, modes=m, layers=L, seed=1)
    try:
        used = free - torch.cuda.mem_get_info()[0]
        field, K = 4 * N ** 3, 4 * m ** 3
        arrays = [4 * net.nparam] * 4 + [2 * net.nparam]
        arrays += [C * field] * (2 * L + 1 + 4) + [field] * 4  # h, z, zq, hb0, hb1, zb; y ..
        arrays += [8 * C * N * 2 * m * m] + [8 * C * K] * (L + 2)
        page = 2 << 20
        need = sum((a + page - 1) // page * page for a in arrays)
        print(f"used {used / 2 ** 20:.1f} MiB, arrays {need / 2 ** 20:.1f}")
        assert used <= need + (16 << 20)
    finally:
        net.close()
