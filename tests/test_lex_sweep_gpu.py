"""The lexicographic sweep on stored coefficients (a warp per row, planes chained): grids down to one
point on an axis, planes of more than four rows per line, several right-hand sides, both modes
and precisions, real and complex wavenumbers, against the oracle's sequential sweep.

Tolerance: complex128 rows have errors of a few 1e-16, 27 updates per point and pass: 1e-12 leaves
three digits; complex64 the same with 6e-8: 1e-5.
"""
import numpy as np
import pytest

from oracle import h3d_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,npml", [((1, 1, 9), 0), ((9, 1, 1), 0), ((1, 11, 3), 0), ((4, 3, 2), 1), ((7, 6, 5), 2),
                                    ((31, 9, 8), 2), ((5, 40, 6), 1), ((6, 17, 33), 2)])
@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("wnc", [False, True])
def test_lex_stored_matches_sequential(cuda, n, npml, mode, wnc):
    import torch
    from h3d import ops

    rng = np.random.default_rng(sum(n) + mode)
    h, N = (25.0, 22.0, 20.0), int(np.prod(n))
    g = O.make_grid(n, h, npml)
    wn = (2 * np.pi * 5.0) ** 2 / (1500.0 + 1500.0 * rng.random(N)) ** 2
    wn = wn * (1 + 0.03j) if wnc else wn
    for nrhs in (1, 3):
        X = rng.standard_normal((N, nrhs)) + 1j * rng.standard_normal((N, nrhs))
        B = rng.standard_normal((N, nrhs)) + 1j * rng.standard_normal((N, nrhs))
        for dt, tol in ((torch.complex128, 1e-12), (torch.complex64, 1e-5)):
            for b in (B, None):
                ref = O.sweep(g, wn, 1.5, X, b, adj=(mode == 2), order=O.ORDER_LEX, nthreads=2)
                t = lambda a: torch.as_tensor(np.ascontiguousarray(a.T), device=cuda).to(dt)
                w = torch.as_tensor(wn, device=cuda)
                w = w.to(dt) if wnc else w.to(torch.float64 if dt == torch.complex128 else torch.float32)
                y = ops.kacz_sweep((n, h, npml), w, 1.5, t(X), t(b) if b is not None else None, mode, order=0)
                err = np.linalg.norm(y.cpu().numpy().T - ref) / np.linalg.norm(ref)
                assert err <= tol, (nrhs, dt, b is None, err)
