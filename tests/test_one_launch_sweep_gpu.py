"""The complex128 BLOCK8 sweep in one launch, taken where a parity has more blocks than the GPU has SMs (and
four times as many at most): grids on both sides of that line, uneven and partial blocks, flat and long
grids (blocks with few neighbours), several columns, both modes, a complex wavenumber, and a batch with
columns that stop at different iterations.

Tolerance: the order of dependent updates is the same as in the oracle, so the two differ by FP64 roundings:
54 updates of a point by 27-term sums, some 1e-14 of the field's size.
"""
import numpy as np
import pytest

from oracle import h3d_oracle as O

pytestmark = pytest.mark.gpu


def _problem(n, npml, seed, wnc, nrhs):
    rng = np.random.default_rng(seed)
    h = (25.0, 20.0, 22.0)
    N = int(np.prod(n))
    wn = (2 * np.pi * 5.0) ** 2 / (1500.0 + 1500.0 * rng.random(N)) ** 2
    wn = wn * (1.0 + 0.03j) if wnc else wn
    X = rng.standard_normal((N, nrhs)) + 1j * rng.standard_normal((N, nrhs))
    B = wn.real.mean() * (rng.standard_normal((N, nrhs)) + 1j * rng.standard_normal((N, nrhs)))
    return h, O.make_grid(n, h, npml), wn, X, B


@pytest.mark.parametrize("n,npml,nrhs", [((145, 61, 110), 10, 2), ((61, 58, 50), 5, 14), ((300, 13, 11), 4, 13),
                                         ((170, 166, 14), 8, 3), ((12, 12, 12), 3, 160), ((13, 180, 181), 6, 1),
                                         ((37, 38, 60), 4, 30)])
@pytest.mark.parametrize("mode,wnc", [(1, False), (2, False), (1, True)])
def test_one_launch_sweep_matches_oracle(cuda, n, npml, nrhs, mode, wnc):
    import torch
    from h3d import ops

    h, g, wn, X, B = _problem(n, npml, 3, wnc, nrhs)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda)
    for b in (B, None):
        ref = O.sweep(g, wn, 1.5, X, b, adj=(mode == 2), order=O.ORDER_BLOCK8, blk=(12, 12, 12), nthreads=8)
        y = ops.kacz_sweep((n, h, npml), t(wn), 1.5, t(X.T), t(B.T) if b is not None else None, mode, order=3)
        err = np.linalg.norm(y.cpu().numpy().T - ref) / np.linalg.norm(ref)
        assert err <= 1e-13, err


def test_batch_of_uneven_problems_matches_single_solves(cuda):
    """Four problems, 17 columns, one of them zero: each column as its own solve gives it."""
    import torch
    from h3d import solver

    probs, rng = [], np.random.default_rng(0)
    for q, (n, nrhs) in enumerate((((61, 58, 50), 6), ((30, 49, 37), 5), ((25, 26, 61), 4), ((60, 40, 40), 2))):
        h, _, wn, _, _ = _problem(n, 5, q, False, 1)
        b = torch.zeros(nrhs, wn.size, dtype=torch.complex128, device=cuda)
        for s in range(nrhs):
            if (q, s) != (1, 2):
                b[s, n[0] // 2 + n[0] * (8 + s + n[1] * int(rng.integers(8, n[2] - 8)))] = 1.0
        probs.append(solver.Problem((n, h, 5), torch.as_tensor(wn, device=cuda), b, 1 + q % 2))
    opts = solver.make_opts(tol=1e-9, maxit=4000, precision="fp64")
    us = solver.solve_batch(probs, opts)[0]
    for p, u in zip(probs, us):
        for s in range(0, p.b.shape[0], 2):
            one = solver.solve(p.grid, p.wn, p.b[s:s + 1], p.mode, opts)[0]
            # both meet a preconditioned residual of 1e-9; in CGMN's metric that bounds the difference to
            # the operator's condition times as much
            assert float((u[s] - one[0]).norm()) <= 1e-5 * max(float(one.norm()), 1e-300)
