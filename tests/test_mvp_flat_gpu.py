"""The complex128 matvec over flattened planes where it can go wrong: planes of fewer points than a
CTA and of a multiple of it, axes of one and two points, rows that straddle warps, PML on all
of an axis and on none of it, every variant, two columns of an odd grid (the second starts off a
16-byte boundary), an input that does, the residual, and a row too long for it (the tiled kernel).

Tolerance: 27-term sums of FP64 products, a few 1e-16 of the field's size each: 1e-14.
"""
import numpy as np
import pytest

from oracle import h3d_oracle as O

pytestmark = pytest.mark.gpu


def _case(n, seed, wnc):
    rng = np.random.default_rng(seed)
    N = int(np.prod(n))
    wn = (2 * np.pi * 5.0) ** 2 / (1500.0 + 1500.0 * rng.random(N)) ** 2
    X = rng.standard_normal((N, 2)) + 1j * rng.standard_normal((N, 2))
    return wn * (1 + 0.03j) if wnc else wn, X


@pytest.mark.parametrize("n,npml", [((16, 8, 9), 2), ((17, 15, 13), (3, 2, 1, 4, 2, 3)), ((1, 1, 40), 0), ((2, 70, 3), 1),
                                    ((64, 4, 6), 0), ((33, 31, 2), 1), ((129, 3, 5), (20, 20, 1, 1, 1, 1)),
                                    ((45, 40, 37), 5), ((3001, 2, 2), 1)])
@pytest.mark.parametrize("wnc", [False, True])
@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("deriv", [False, True])
def test_flat_matvec(cuda, n, npml, wnc, mode, deriv):
    import torch
    from h3d import ops

    h = (25.0, 20.0, 22.0)
    g = O.make_grid(n, h, npml)
    wn, X = _case(n, 7 + sum(n), wnc)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda)
    ref = O.mvp(g, wn, X, adj=(mode == 2), deriv=deriv, nthreads=2).T
    N = X.shape[0]
    y = ops.mvp((n, h, npml), t(wn), t(X.T), mode, deriv).cpu().numpy()
    assert np.linalg.norm(y - ref) / np.linalg.norm(ref) <= 1e-14
    # a wavenumber 8 bytes off a 16-byte boundary
    off = torch.empty(N + 1, dtype=torch.complex128 if wnc else torch.float64, device=cuda)[1:]
    off.copy_(t(wn))
    y = ops.mvp((n, h, npml), off, t(X.T), mode, deriv).cpu().numpy()
    assert np.linalg.norm(y - ref) / np.linalg.norm(ref) <= 1e-14
    if not deriv:
        b = t(X.T.conj().copy())
        r, rr, bb = ops.residual((n, h, npml), t(wn), b, t(X.T), mode)
        want = X.T.conj() - ref
        assert np.linalg.norm(r.cpu().numpy() - want) / np.linalg.norm(want) <= 1e-14
        np.testing.assert_allclose(rr.cpu().numpy(), (abs(want) ** 2).sum(1), rtol=1e-12)
        np.testing.assert_allclose(bb.cpu().numpy(), (abs(X.T) ** 2).sum(1), rtol=1e-12)


def test_nonfinite_values_stay_local(cuda):
    """A NaN in x reaches its 27 neighbours and nothing else, across row ends and plane faces too."""
    import torch
    from h3d import ops

    n, h = (13, 11, 7), (20.0, 20.0, 20.0)
    wn, X = _case(n, 3, False)
    for at in ((0, 5, 3), (12, 10, 6), (6, 0, 0)):
        x = torch.as_tensor(X[:, 0].copy(), device=cuda)
        x[at[0] + n[0] * (at[1] + n[1] * at[2])] = float("nan")
        y = ops.mvp((n, h, 2), torch.as_tensor(wn, device=cuda), x, 1)
        bad = torch.isnan(y.real).cpu().numpy().reshape(n, order="F")
        want = np.zeros(n, bool)
        want[tuple(slice(max(a - 1, 0), a + 2) for a in at)] = True
        assert (bad == want).all(), at
