"""The BLOCK8 tuner's choice is kept per batch shape and kind of wavenumber: a complex one has other
records and other kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_complex_wavenumber_is_tuned_by_itself(cuda, precision, capfd):
    import torch
    from h3d import solver

    n, h, npml = (27, 31, 23), (20.0, 20.0, 20.0), 5
    N = int(np.prod(n))
    wn = torch.full((N,), (2 * np.pi * 5.0 / 2000.0) ** 2, dtype=torch.float64, device=cuda)
    b = torch.zeros(3, N, dtype=torch.complex128, device=cuda)
    for s in range(3):
        b[s, N // 2 + s] = 1.0
    opts = solver.make_opts(tol=1e-6, precision=precision, verbose=True)

    def tuned(w):
        capfd.readouterr()
        solver.solve((n, h, npml), w, b, 1, opts)
        return capfd.readouterr().err.count("tune batched BLOCK8")

    assert tuned(wn) > 0
    assert tuned(wn * 1.01) == 0           # the same shape again
    assert tuned(wn * (1 + 0.02j)) > 0
    assert tuned(wn * (1 + 0.03j)) == 0
