"""h3d_residual_noalloc with many right-hand sides, where one partial sum per 128-point tile of a plane
overruns the fixed scratch and one per 32 x 8 columns does not."""
import ctypes as C

import numpy as np
import pytest


def _size_check(n, nrhs):
    """True when the call gets past the scratch check (data pointers NULL: nothing is launched)."""
    from h3d import _lib as L

    lib = L.load()
    grid = L.make_grid(n, (10.0, 10.0, 10.0), 1)
    rc = lib.h3d_residual_noalloc(C.byref(grid), None, None, None, None, None, None, None, nrhs, L.FORWARD, None)
    assert rc == L.ERR_BAD_ARG
    return b"scratch" not in lib.h3d_last_error()


# One chunk in z (nz < 32: the split chosen without a GPU).  The tables take 6 sum_a (n_a + 2) doubles,
# rounded up to 32, a partial sum two; the scratch holds 4 MiB / 8 of them.
@pytest.mark.parametrize("n", [(64, 64, 20), (96, 96, 30), (201, 201, 30), (33, 9, 5)])
def test_scratch_takes_one_sum_per_column_block(n):
    tab = (6 * sum(m + 2 for m in n) + 31) // 32 * 32
    tiles = min(-(-n[0] // 32) * -(-n[1] // 8), -(-(n[0] * n[1]) // 128))
    most = min(((4 << 20) // 8 - tab) // (2 * tiles), 65535)
    assert _size_check(n, most)
    if most < 65535:
        assert not _size_check(n, most + 1)


@pytest.mark.gpu
def test_many_columns_match_allocating_entry_point(cuda):
    """9000 columns on 64 x 64 x 3: 16 sums a column fit, 32 do not.  Both entry points form r and the sums
    in FP64, by different kernels: 27-term rows and 12288-term sums, 1e-13 relative."""
    import torch
    from h3d import _lib as L
    from h3d import ops

    n, h, P, npml = (64, 64, 3), (25.0, 20.0, 22.0), 9000, (6, 5, 4, 7, 1, 1)
    N = int(np.prod(n))
    gen = torch.Generator(device=cuda).manual_seed(4)
    wn = (2 * np.pi * 4.0) ** 2 / (1500 + 2000 * torch.rand(N, dtype=torch.float64, device=cuda, generator=gen)) ** 2
    x = torch.randn(P, N, dtype=torch.complex128, device=cuda, generator=gen)
    b = torch.randn(P, N, dtype=torch.complex128, device=cuda, generator=gen)
    grid, lib = L.make_grid(n, h, npml), L.load()
    for mode in (1, 2):
        r0, rr0, bb0 = ops.residual(grid, wn, b, x, mode)
        r, rr, bb = torch.empty_like(b), torch.empty_like(rr0), torch.empty_like(bb0)
        rc = lib.h3d_residual_noalloc(C.byref(grid), wn.data_ptr(), None, b.data_ptr(), x.data_ptr(), r.data_ptr(),
                                      rr.data_ptr(), bb.data_ptr(), P, mode, torch.cuda.current_stream().cuda_stream)
        assert rc == 0, lib.h3d_last_error()
        assert float((r - r0).abs().max()) <= 1e-13 * float(r0.abs().max())
        assert float(((rr - rr0).abs() / rr0).max()) <= 1e-13
        assert float(((bb - bb0).abs() / bb0).max()) <= 1e-13
