"""A smoother that has stopped costs launches that return at once, not matvecs."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve_seconds(levels, R, P, b, precision, k, smooth_tol):
    """Fastest of three solves of two outer steps, from the solve's own clock."""
    import torch
    from h3d import _lib as L
    from h3d import multigrid as MG

    lib = L.load()
    lv, Rs, Ps = MG._level_structs(levels, R, P)
    o = L.MLOpts()
    lib.h3d_ml_default_opts(C.byref(o))
    o.tol, o.maxit, o.maxinnerit, o.smooth_tol, o.precision = 1e-12, 1, 2, smooth_tol, precision
    for i in range(4):
        o.k[i] = k[i]
    best = 1e30
    for _ in range(4):
        u, info = torch.zeros_like(b), L.MLInfo()
        rc = lib.h3d_mlgmres_solve(lv, len(levels), Rs, Ps, b.data_ptr(), u.data_ptr(), L.FORWARD, C.byref(o), None, 0,
                                   C.byref(info), torch.cuda.current_stream().cuda_stream)
        assert rc == 0, lib.h3d_last_error()
        best = min(best, info.seconds)
    return best, u


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_stopped_smoother_runs_no_matvecs(cuda, precision):
    """smooth_tol = 1: the smoothers stop before their first step (FGMRES.m:88, hst = 1).  Up to three
    cycles of 16 steps are then enqueued for one of one step: 100 matvecs more per V-cycle, on 3.3 million points
    (0.7 ms each in complex128, 40 us in complex64) beside a few milliseconds of outer and coarse work.  The
    solve takes three times as long or more where they run, a third longer where they return at once."""
    import torch
    from h3d import _lib as L
    from h3d import multigrid as MG

    n = (161, 161, 81)
    z = np.arange(n[2]) / (n[2] - 1.0)
    v = np.broadcast_to(1500 + 1500 * z, n).copy()
    lv, R, P = MG.build_levels(v, (20.0,) * 3, 10, 5.0, "m/s", device=cuda)
    nx, ny, nz = lv[0].nt
    b = torch.zeros(nx * ny * nz, dtype=torch.complex128, device=cuda)
    b[nx // 2 + nx * (ny // 2 + ny * (nz // 2))] = 1.0
    p = L.PREC_FP64 if precision == "fp64" else L.PREC_MIXED
    many, u1 = _solve_seconds(lv, R, P, b, p, (3, 16, 1, 1), 1.0)
    one, u0 = _solve_seconds(lv, R, P, b, p, (1, 1, 1, 1), 1.0)
    assert torch.equal(u0, u1)  # nothing was smoothed in either
    assert many <= 2.0 * one, (many, one)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("smooth_tol", [0.7, 0.3])
def test_loose_smoother_gives_the_same_solution(cuda, precision, smooth_tol):
    """Smoothers that stop in the middle of a cycle: the outer iteration still converges to its tolerance."""
    import torch
    from h3d import _lib as L
    from h3d import multigrid as MG

    n = (37, 33, 29)
    v = np.full(n, 2000.0)
    lv, R, P = MG.build_levels(v, (25.0,) * 3, 6, 4.0, "m/s", device=cuda)
    b = torch.zeros(int(np.prod(lv[0].nt)), dtype=torch.complex128, device=cuda)
    b[b.numel() // 2 + lv[0].nt[0] // 2] = 1.0
    lib = L.load()
    s = MG._level_structs(lv, R, P)
    o = L.MLOpts()
    lib.h3d_ml_default_opts(C.byref(o))
    o.tol, o.maxit, o.smooth_tol = 1e-8, 200, smooth_tol
    o.precision = L.PREC_FP64 if precision == "fp64" else L.PREC_MIXED
    u, info = torch.zeros_like(b), L.MLInfo()
    rc = lib.h3d_mlgmres_solve(s[0], len(lv), s[1], s[2], b.data_ptr(), u.data_ptr(), L.FORWARD, C.byref(o), None, 0,
                               C.byref(info), torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and info.converged == 1
    assert torch.linalg.norm(b - lv[0].A(u, 1)) <= 1.01e-8 * torch.linalg.norm(b)
