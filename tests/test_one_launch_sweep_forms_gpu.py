"""The complex128 BLOCK8 sweep in one launch, in each of its compiled forms (right-hand sides per CTA and per
thread, by H3D_BLOCK8_CONFIG), on grids whose blocks miss neighbours, with as many columns as take a parity
past the GPU's SMs and the last group half filled; and its wait for the blocks around, made to run out.

Tolerance: the order of dependent updates is the oracle's; 54 updates of a point by 27-term FP64 sums differ
by some 1e-14 of the field's size.
"""
import numpy as np
import pytest

from oracle import h3d_oracle as O

pytestmark = pytest.mark.gpu

R_OF_CONFIG = (1, 2, 2)


def _blocks(n):
    """Blocks of the parity that has the most: the even-indexed ones."""
    return int(np.prod([(-(-m // 12) + 1) // 2 for m in n]))


def _sweep_matches_oracle(cuda, n, npml, nrhs, mode, wnc, seed=3):
    import torch
    from h3d import ops

    rng = np.random.default_rng(seed)
    h, N = (25.0, 20.0, 22.0), int(np.prod(n))
    g = O.make_grid(n, h, npml)
    wn = (2 * np.pi * 5.0) ** 2 / (1500.0 + 1500.0 * rng.random(N)) ** 2
    wn = wn * (1.0 + 0.03j) if wnc else wn
    X = rng.standard_normal((N, nrhs)) + 1j * rng.standard_normal((N, nrhs))
    B = wn.real.mean() * (rng.standard_normal((N, nrhs)) + 1j * rng.standard_normal((N, nrhs)))
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda)
    for b in (B, None):
        ref = O.sweep(g, wn, 1.5, X, b, adj=(mode == 2), order=O.ORDER_BLOCK8, blk=(12, 12, 12), nthreads=8)
        y = ops.kacz_sweep((n, h, npml), t(wn), 1.5, t(X.T), t(B.T) if b is not None else None, mode, order=3)
        err = np.linalg.norm(y.cpu().numpy().T - ref) / np.linalg.norm(ref)
        assert err <= 1e-13, err


@pytest.mark.parametrize("cfg", range(3))
@pytest.mark.parametrize("n,npml,mode,wnc", [((145, 61, 110), 10, 1, False),   # most neighbours there
                                             ((300, 13, 11), 4, 2, False),     # long: two blocks by one
                                             ((170, 166, 14), 8, 1, True),     # flat
                                             ((12, 12, 12), 3, 2, True),       # one block: no neighbour at all
                                             ((13, 61, 62), 6, 2, False),
                                             ((25, 24, 37), 4, 1, False)])
def test_each_form_matches_oracle(cuda, cfg, n, npml, mode, wnc, monkeypatch):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nb, r = _blocks(n), R_OF_CONFIG[cfg]
    groups = sms // nb + 1
    nrhs = r * groups - (r - 1)
    assert sms < nb * groups <= 4 * sms  # the rule that takes one launch
    monkeypatch.setenv("H3D_BLOCK8_CONFIG", str(cfg))
    _sweep_matches_oracle(cuda, n, npml, nrhs, mode, wnc)


@pytest.mark.parametrize("mode", [1, 2])
def test_one_column_matches_oracle(cuda, mode):
    """A single column on a grid that takes one launch by its own size: no configuration fixed."""
    import torch

    n = (161, 161, 81)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert sms < _blocks(n) <= 4 * sms
    _sweep_matches_oracle(cuda, n, 15, 1, mode, False)


def test_wait_for_the_blocks_around_expires_with_a_status(cuda):
    """Both bounded waits give up after 3 ms (the whole sweep's blocks take less than one), and a sweep right
    after, in one launch, matches the oracle."""
    from h3d import _lib as L

    lib = L.load()
    assert lib.h3d_check_wait_timeout(3.0) == L.ERR_TIMEOUT
    status = str(L.ERR_TIMEOUT).encode()
    assert b"blocks around in one launch (status " + status + b")" in lib.h3d_last_error()
    _sweep_matches_oracle(cuda, (61, 58, 50), 5, 14, 1, False)
