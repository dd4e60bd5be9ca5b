"""The lexicographic sweep call on a grid whose 27 N stored coefficients would take more than half of the free
device memory: it forms them row by row instead, and leaves the memory to others."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

USED_MEM_HIGH = 8  # CU_MEMPOOL_ATTR_USED_MEM_HIGH


def test_lex_sweep_leaves_half_of_the_free_memory(cuda):
    """A fixed point of the sweep (b = H x) stays where it is, to the rounding of 54 updates by 27-term sums of
    FP64 values (1e-12), and with b = 0 every projection with w = 1.5 shortens x."""
    import torch
    from h3d import ops

    cu = C.CDLL("libcuda.so.1")
    pool, high = C.c_void_p(), C.c_uint64(0)
    torch.cuda.synchronize()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), torch.cuda.current_device()) == 0

    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    # 27 x 16 bytes a point: 0.55 of what is free, with as few hyperplanes i + 3j + 9k as such a grid can have
    c = int((0.55 * free / (27 * 16) / 27) ** (1 / 3)) + 1
    n, h, npml = (9 * c, 3 * c, c), (20.0, 20.0, 20.0), 8
    N = n[0] * n[1] * n[2]
    gen = torch.Generator(device=cuda).manual_seed(0)
    wn = torch.rand(N, dtype=torch.float64, device=cuda, generator=gen).mul_(1e-4).add_(1e-4)
    x = torch.view_as_complex(torch.randn(N, 2, dtype=torch.float64, device=cuda, generator=gen))
    b = ops.mvp((n, h, npml), wn, x)
    assert cu.cuMemPoolSetAttribute(pool, USED_MEM_HIGH, C.byref(high)) == 0
    y = ops.kacz_sweep((n, h, npml), wn, 1.5, x, b, 1, order=0)
    z = ops.kacz_sweep((n, h, npml), wn, 1.5, x, None, 1, order=0)
    torch.cuda.synchronize()
    assert cu.cuMemPoolGetAttribute(pool, USED_MEM_HIGH, C.byref(high)) == 0
    assert high.value < free // 4, high.value
    nx = float(torch.linalg.norm(x))
    assert float(torch.linalg.norm(y - x)) <= 1e-12 * nx
    assert float(torch.linalg.norm(z)) < nx
    del x, b, y, z, wn
    torch.cuda.empty_cache()
