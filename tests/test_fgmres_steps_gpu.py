"""The FGMRES cycle's kernels at every number of basis vectors they are instantiated for (1 to 5, up
to 8, up to 16) and on a field whose inner products go through clusters, against
GMRES(m) written out in torch; and the complex64 cycle at several smoother and coarse-solver settings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _levels(n, cuda, npml=6, f=4.0, seed=0):
    from h3d import multigrid as MG

    rng = np.random.default_rng(seed)
    h = 25.0
    z = np.arange(n[2]) * h
    v = np.broadcast_to(1500 + 1000 * z / z[-1], n).copy() * (1 + 0.05 * rng.standard_normal(n))
    return MG.build_levels(v, (h, h, h), npml, f, "m/s", device=cuda)


def _gmres(A, b, x, m, cycles):
    """GMRES(m), modified Gram-Schmidt twice over and an explicit least-squares solve."""
    import torch

    hst, r0 = [1.0], None
    for _ in range(cycles):
        r = b - A(x)
        beta = torch.linalg.norm(r)
        r0 = beta if r0 is None else r0
        V, H = [r / beta], torch.zeros(m + 1, m, dtype=torch.complex128)
        for j in range(m):
            w = A(V[j])
            for _ in range(2):
                for i in range(j + 1):
                    c = torch.vdot(V[i], w)
                    H[i, j] += c.cpu()
                    w = w - c * V[i]
            nw = torch.linalg.norm(w)
            H[j + 1, j] = nw.cpu()
            V.append(w / nw)
            e = torch.zeros(j + 2, 1, dtype=torch.complex128)
            e[0] = beta.cpu()
            y = torch.linalg.lstsq(H[: j + 2, : j + 1], e).solution
            hst.append(float(torch.linalg.norm(e - H[: j + 2, : j + 1] @ y) / r0.cpu()))
        x = x + sum(V[i] * y[i, 0].to(b.device) for i in range(m))
    return x, hst


# 2 x 16 steps of a restarted method whose quasi-residual falls by less than a factor of ten, classical
# Gram-Schmidt in FP64: the basis loses orthogonality as the Krylov matrix's condition times 1e-16, and
# scipy's GMRES(m) is held to the same bounds in the multigrid tests.
@pytest.mark.parametrize("n,m", [((17, 15, 13), m) for m in (1, 2, 3, 4, 5, 6, 8, 9, 16)]
                         + [((70, 66, 64), 5), ((70, 66, 64), 7)])
def test_cycles_match_gmres_written_out(cuda, n, m):
    import torch
    from h3d import multigrid as MG

    lv, R, P = _levels(n, cuda)
    g = torch.Generator().manual_seed(3)
    b = torch.randn(int(np.prod(lv[0].nt)), dtype=torch.complex128, generator=g).to(cuda)
    x0 = torch.zeros_like(b)
    x, hst = _gmres(lv[0].A, b, x0, m, 2)
    # FGMRES.m's step counter starts at one: GMRES(1) counts its first cycle as two
    u, info = MG.solve(lv, R, P, b, tol=1e-13, maxit=2 if m > 1 else 3, maxinnerit=m, precond="none")
    assert info["iters"] == 2 * m
    np.testing.assert_allclose(info["hst"], hst, rtol=1e-8)
    assert torch.linalg.norm(u - x) <= 1e-8 * torch.linalg.norm(x)


@pytest.mark.parametrize("n,k", [((17, 15, 13), (3, 5, 3, 5)), ((17, 15, 13), (2, 3, 1, 6)),
                                 ((17, 15, 13), (6, 4, 2, 10)), ((70, 66, 64), (2, 5, 2, 4))])
@pytest.mark.parametrize("mode", [1, 2])
def test_complex64_cycle_solves_to_the_tolerance(cuda, n, k, mode):
    import torch
    from h3d import multigrid as MG

    lv, R, P = _levels(n, cuda)
    nx, ny, nz = lv[0].nt
    b = torch.zeros(nx * ny * nz, dtype=torch.complex128, device=cuda)
    b[nx // 2 + nx * (ny // 2 + ny * (nz // 2))] = 1.0
    u, info = MG.solve(lv, R, P, b, tol=1e-8, mode=mode, precision="mixed", k=k)
    ref, full = MG.solve(lv, R, P, b, tol=1e-8, mode=mode, precision="fp64", k=k)
    assert info["converged"] == 1 and full["converged"] == 1
    # a cycle in complex64 differs from the complex128 one by some 1e-6 of its result: at most a step more
    assert info["iters"] <= full["iters"] + 1
    for s in (u, ref):
        # the quasi-residual meets 1e-8; the true one follows it to the complex128 basis' rounding
        assert torch.linalg.norm(b - lv[0].A(s, mode)) <= 1.01e-8 * torch.linalg.norm(b)
