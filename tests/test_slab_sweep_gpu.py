"""The complex64 BLOCK8 sweep (one warp per z slab, windows in registers) where it can go wrong:
block remainders of 1, 2 and 11 points on every axis, a single block, PML everywhere and nowhere
inside a block, one, two and three right-hand sides (a full and a half-filled group), both modes,
real and complex wavenumbers, and how far a NaN spreads.  (Problems of several kinds in one batch are in
test_solver_gpu.py.)

Tolerance: a row projection in complex64 has a relative error of a few FP32 roundings (6e-8 each,
27-term sums); a point is updated by at most 27 rows per pass and two passes, so errors stay
below 54 x a few roundings ~ 1e-5 of the field's size.
"""
import numpy as np
import pytest

from oracle import h3d_oracle as O

pytestmark = pytest.mark.gpu


def _problem(n, npml, seed, wnc, nrhs):
    rng = np.random.default_rng(seed)
    h = (25.0, 20.0, 22.0)
    N = int(np.prod(n))
    wn = ((2 * np.pi * 5.0) ** 2 / (1500.0 + 1500.0 * rng.random(N)) ** 2).astype(np.float32)
    wn = wn * np.complex64(1.0 + 0.03j) if wnc else wn
    X = (rng.standard_normal((N, nrhs)) + 1j * rng.standard_normal((N, nrhs))).astype(np.complex64)
    B = (wn.real.mean() * (rng.standard_normal((N, nrhs)) + 1j * rng.standard_normal((N, nrhs)))).astype(np.complex64)
    return h, O.make_grid(n, h, npml), wn, X, B


@pytest.mark.parametrize("n,npml", [((12, 12, 12), 3), ((13, 25, 36), 4), ((26, 13, 11), 2), ((49, 37, 38), 5),
                                    ((3, 30, 14), 1), ((24, 5, 47), 0)])
@pytest.mark.parametrize("wnc", [False, True])
@pytest.mark.parametrize("mode", [1, 2])
def test_slab_sweep_block_remainders(cuda, n, npml, wnc, mode):
    import torch
    from h3d import ops

    for nrhs in (1, 2, 3):
        h, g, wn, X, B = _problem(n, npml, 11 + nrhs, wnc, nrhs)
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda)
        for b in (B, None):
            ref = O.sweep(g, wn.astype(np.complex128 if wnc else np.float64), 1.5, X, b, adj=(mode == 2),
                          order=O.ORDER_BLOCK8, blk=(12, 12, 12), nthreads=2)
            y = ops.kacz_sweep((n, h, npml), t(wn), 1.5, t(X.T), t(B.T) if b is not None else None, mode, order=3)
            err = np.linalg.norm(y.cpu().numpy().T - ref) / np.linalg.norm(ref)
            assert err <= 1e-5, (nrhs, b is None, err)


def test_slab_sweep_keeps_nan_and_inactive_columns(cuda):
    """A NaN in x spreads only where the sweep carries it (every block here), and a batched solve with
    a zero right-hand side leaves that column exactly zero beside a converging one."""
    import torch
    from h3d import ops, solver

    n, npml = (26, 25, 27), 4
    h, g, wn, X, _ = _problem(n, npml, 5, False, 1)
    x = torch.as_tensor(X.T.copy(), device=cuda)
    x[0, 0] = float("nan")
    y = ops.kacz_sweep((n, h, npml), torch.as_tensor(wn, device=cuda), 1.5, x, None, 1, order=3)
    assert bool(torch.isnan(y).any())
    b = torch.zeros(2, X.shape[0], dtype=torch.complex128, device=cuda)
    b[1, X.shape[0] // 2] = 1.0
    u, info = solver.solve((n, h, npml), torch.as_tensor(wn.astype(np.float64), device=cuda), b, precision="mixed")
    assert bool((u[0] == 0).all()) and info["rel_res_true"] <= 1e-6


@pytest.mark.parametrize("n,npml,at", [((300, 13, 14), 4, (0, 0, 0)), ((14, 290, 13), 5, (7, 150, 6)),
                                       ((11, 12, 280), 3, (10, 11, 279)), ((130, 140, 13), 6, (60, 70, 12))])
@pytest.mark.parametrize("mode,wnc", [(1, False), (2, False), (1, True)])
def test_nan_spreads_as_far_as_in_the_oracle(cuda, n, npml, at, mode, wnc):
    """One NaN in x, on a face, in the interior or in a corner of a grid that is long enough for the sweep not
    to carry it everywhere: the same points turn NaN as in the sequential sweep, no others."""
    import torch
    from h3d import ops

    h, g, wn, X, _ = _problem(n, npml, 7, wnc, 1)
    X[at[0] + n[0] * (at[1] + n[1] * at[2]), 0] = np.nan
    ref = O.sweep(g, wn.astype(np.complex128 if wnc else np.float64), 1.5, X, None, adj=(mode == 2),
                  order=O.ORDER_BLOCK8, blk=(12, 12, 12), nthreads=2)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda)
    y = ops.kacz_sweep((n, h, npml), t(wn), 1.5, t(X.T), None, mode, order=3).cpu().numpy().T
    assert 0 < np.isnan(ref).sum() < ref.size
    np.testing.assert_array_equal(np.isnan(y), np.isnan(ref))
