"""Performance cases of the Helmholtz framework: what a user's program has it compute.

Each case goes through a public entry point of ``h3d`` on inputs made from a seed:

  mvp      ``ops.mvp``            H x, H^H x and the derivative operator (Born sources)
  sweep    ``ops.kacz_sweep``     one Kaczmarz double sweep (LEX: the drop-in row order; BLOCK8)
  cgmn     ``solver.solve``       CGMN with the Kaczmarz preconditioner
  batch    ``solver.solve_batch`` the same for several problems of uneven size at once
  mg       ``multigrid.solve``    FGMRES + ML_GMRES, the default solver of the 3D applications
  fwi      ``fwi.fwi_objective``  misfit and adjoint-state gradient

Sizes are those of ``h3d.models`` (61^3, 201 x 201 x 101, 161 x 161 x 81, 64-192 uneven) and of
the multigrid levels under them.  A mixed-precision solve iterates in complex64 under FP64
refinement, so two correct builds agree on the solution only as far as it is solved: these
cases ask for a tight tolerance (a reference wavefield, a gradient test), which takes more of
the same iterations.
"""
import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "slim-release-apps_gb300"))
from h3d import _lib as L  # noqa: E402
from h3d import fwi, multigrid, ops, solver  # noqa: E402

DEV = "cuda"
DTYPES = {"c64": torch.complex64, "c128": torch.complex128}
H = 20.0  # grid spacing (m)


def listed():
    return [
        # the smallest call: the matvec on the coarsest multigrid level of the 201 x 201 x 101
        # problem, where the call's own cost counts
        {"name": "mvp coarse level c64", "kind": "mvp", "nx": 51, "ny": 51, "nz": 26, "pml": 5, "rhs": 1,
         "mode": 1, "deriv": False, "cwn": False, "dtype": "c64", "ppw": 6.0},
        # the ordinary matvec in the working precision of the mixed solvers
        {"name": "mvp 201x201x101 c64", "kind": "mvp", "nx": 201, "ny": 201, "nz": 101, "pml": 20, "rhs": 1,
         "mode": 1, "deriv": False, "cwn": False, "dtype": "c64", "ppw": 12.5},
        # the adjoint in FP64 on several right-hand sides (residuals, adjoint checks)
        {"name": "mvp adjoint c128 4 rhs", "kind": "mvp", "nx": 161, "ny": 161, "nz": 81, "pml": 15, "rhs": 4,
         "mode": 2, "deriv": False, "cwn": False, "dtype": "c128", "ppw": 12.5},
        # the drop-in sweep in the reference's row order, FP64 with a right-hand side
        {"name": "sweep lex 61^3 c128", "kind": "sweep", "order": "lex", "nx": 61, "ny": 61, "nz": 61, "pml": 10,
         "rhs": 1, "mode": 1, "dtype": "c128", "ppw": 15.0},
        # the library's row order, one column and a group of sources
        {"name": "sweep block8 c64", "kind": "sweep", "order": "block8", "nx": 201, "ny": 201, "nz": 101, "pml": 20,
         "rhs": 1, "mode": 1, "dtype": "c64", "ppw": 12.5},
        {"name": "sweep block8 adjoint c64 8 rhs", "kind": "sweep", "order": "block8", "nx": 161, "ny": 161,
         "nz": 81, "pml": 15, "rhs": 8, "mode": 2, "dtype": "c64", "ppw": 12.5},
        # a whole mixed-precision CGMN solve of the 61^3 problem
        {"name": "cgmn mixed 61^3", "kind": "cgmn", "nx": 61, "ny": 61, "nz": 61, "pml": 10, "rhs": 1, "mode": 1,
         "precision": "mixed", "tol": 1e-11, "maxit": 10000, "ppw": 15.0},
        # an inexact FP64 solve: a fixed number of CGMN iterations on the FWI grid, adjoint
        {"name": "cgmn fp64 20 iterations", "kind": "cgmn", "nx": 161, "ny": 161, "nz": 81, "pml": 15, "rhs": 1,
         "mode": 2, "precision": "fp64", "tol": 1e-12, "maxit": 20, "ppw": 12.5},
        # problems of uneven size, several sources each, in one batched solve
        {"name": "batch mixed uneven", "kind": "batch", "problems": 4, "lo": 40, "hi": 96, "layout": 4, "most_rhs": 4,
         "pml": 10, "tol": 1e-11, "ppw": 6.0},
        # the applications' default solve at the size of the benchmark problem
        {"name": "mg mixed 201x201x101", "kind": "mg", "nx": 201, "ny": 201, "nz": 101, "pml": 20, "mode": 1,
         "precision": "mixed", "tol": 1e-10, "ppw": 12.5},
        # the same in FP64 with the library's default settings, adjoint, small
        {"name": "mg fp64 adjoint 61^3", "kind": "mg", "nx": 61, "ny": 61, "nz": 61, "pml": 10, "mode": 2,
         "precision": "fp64", "tol": 1e-6, "ppw": 15.0},
        # misfit and gradient of one frequency by the multigrid solver
        {"name": "fwi gradient 2 sources", "kind": "fwi", "nx": 81, "ny": 71, "nz": 51, "pml": 10, "sources": 2,
         "receivers": 100, "tol": 1e-10, "ppw": 12.5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
    # one length for all axes, each axis off by up to a third, so that odd and ragged sizes turn up
    n = _log_int(rng, lo, hi)
    return {k: max(24, min(hi, int(round(n * rng.uniform(0.67, 1.2))))) for k in ("nx", "ny", "nz")}


def draw(rng):
    kind = rng.choice(["mvp", "mvp", "sweep lex", "sweep block8", "sweep block8", "cgmn mixed", "cgmn fp64", "batch",
                       "mg mixed", "mg mixed", "mg fp64", "fwi"])
    ppw = rng.uniform(6.0, 15.0)
    mode = rng.choice([1, 2])
    if kind == "mvp":
        c = _dims(rng, 26, 170)
        return dict(c, kind="mvp", pml=rng.choice([5, 10, 15]) if min(c.values()) > 36 else 5,
                    rhs=rng.choice([1, 1, 2, 3, 8]), mode=mode, deriv=rng.random() < 0.25, cwn=rng.random() < 0.15,
                    dtype=rng.choice(["c64", "c128"]), ppw=ppw)
    if kind == "sweep lex":
        return dict(_dims(rng, 30, 80), kind="sweep", order="lex", pml=8, rhs=rng.choice([1, 1, 3]), mode=mode,
                    dtype=rng.choice(["c128", "c128", "c64"]), ppw=ppw)
    if kind == "sweep block8":
        return dict(_dims(rng, 30, 160), kind="sweep", order="block8", pml=10, rhs=rng.choice([1, 2, 5, 8]),
                    mode=mode, dtype=rng.choice(["c64", "c64", "c128"]), ppw=ppw)
    if kind == "cgmn mixed":
        return dict(_dims(rng, 32, 64), kind="cgmn", pml=10, rhs=rng.choice([1, 1, 3]), mode=mode, precision="mixed",
                    tol=1e-11, maxit=10000, ppw=rng.uniform(6.0, 12.0))
    if kind == "cgmn fp64":
        return dict(_dims(rng, 40, 150), kind="cgmn", pml=10, rhs=rng.choice([1, 2]), mode=mode, precision="fp64",
                    tol=1e-12, maxit=rng.choice([10, 20]), ppw=ppw)
    if kind == "batch":
        return {"kind": "batch", "problems": rng.choice([2, 3, 4]), "lo": 32, "hi": rng.randint(48, 88),
                "layout": rng.randrange(1000), "most_rhs": rng.choice([1, 3]), "pml": 10, "tol": 1e-11,
                "ppw": rng.uniform(6.0, 10.0)}
    if kind == "mg mixed":
        return dict(_dims(rng, 40, 160), kind="mg", pml=10, mode=mode, precision="mixed", tol=1e-10, ppw=ppw)
    if kind == "mg fp64":
        return dict(_dims(rng, 40, 80), kind="mg", pml=10, mode=mode, precision="fp64", tol=1e-6, ppw=ppw)
    return dict(_dims(rng, 44, 90), kind="fwi", pml=10, sources=rng.choice([1, 2]), receivers=rng.randint(20, 200),
                tol=1e-10, ppw=ppw)


# ---- inputs ---------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _velocity(n_phys, gen):
    """1500 -> 3500 m/s with depth, times 1 + 0.1 g with g a smooth random field in [-1, 1];
    indexed (x, y, z)."""
    nx, ny, nz = n_phys
    coarse = [max(2, -(-s // 6)) for s in (nz, ny, nx)]
    g = torch.randn((1, 1, *coarse), generator=gen, device=DEV, dtype=torch.float64)
    g = torch.nn.functional.interpolate(g, size=(nz, ny, nx), mode="trilinear", align_corners=True)[0, 0]
    z = torch.linspace(0.0, 1.0, nz, device=DEV, dtype=torch.float64)[:, None, None]
    v = (1500.0 + 2000.0 * z) * (1.0 + 0.1 * g.clamp(-1.0, 1.0))
    return v.permute(2, 1, 0).clamp(min=1350.0)


def _freq(ppw):
    return 1500.0 / (ppw * H)  # ppw points per wavelength at 1500 m/s


def _wavenumber(v, pml, freq):
    """(2 pi f)^2 / v^2 with the edge values replicated into the PML, x fastest."""
    t = v.permute(2, 1, 0)[None, None]
    t = torch.nn.functional.pad(t, (pml,) * 6, mode="replicate")[0, 0]
    return ((2.0 * math.pi * freq) ** 2 / t ** 2).reshape(-1).contiguous()


def _n(case):
    return case["nx"], case["ny"], case["nz"]


def _grid(n, pml):
    return (tuple(n), (H, H, H), pml)


def _field(shape, dtype, gen):
    real = torch.float32 if dtype == torch.complex64 else torch.float64
    return torch.view_as_complex(torch.randn((*shape, 2), generator=gen, device=DEV, dtype=real))


def _point_sources(n, pml, rhs, rng):
    """Unit impulses two cells below the top of the physical grid."""
    b = torch.zeros(rhs, n[0] * n[1] * n[2], dtype=torch.complex128, device=DEV)
    for s in range(rhs):
        i, j = rng.randrange(pml, n[0] - pml), rng.randrange(pml, n[1] - pml)
        b[s, i + n[0] * (j + n[1] * (pml + 2))] = 1.0
    return b


def _operator(n, pml, ppw, gen):
    return _wavenumber(_velocity([s - 2 * pml for s in n], gen), pml, _freq(ppw))


def _layout(case):
    """Sizes and source counts of a batch."""
    rng = random.Random(case["layout"])
    return [([_log_int(rng, case["lo"], case["hi"]) for _ in range(3)], rng.randint(1, case["most_rhs"]))
            for _ in range(case["problems"])]


def _mvp_inputs(case, seed):
    gen, n = _gen(seed), _n(case)
    dt = DTYPES[case["dtype"]]
    wn = _operator(n, case["pml"], case["ppw"], gen)
    if case["cwn"]:  # an attenuating medium: wn (1 + i/Q)
        wn = wn * (1.0 + 0.02j)
    wn = wn.to(dt if case["cwn"] else (torch.float32 if dt == torch.complex64 else torch.float64))
    return wn, _field((case["rhs"], n[0] * n[1] * n[2]), dt, gen)


def _sweep_inputs(case, seed):
    gen, n = _gen(seed), _n(case)
    dt = DTYPES[case["dtype"]]
    wn = _operator(n, case["pml"], case["ppw"], gen).to(torch.float32 if dt == torch.complex64 else torch.float64)
    N = n[0] * n[1] * n[2]
    # a right-hand side of the size of A x
    b = _field((case["rhs"], N), dt, gen) * float(wn.mean())
    return wn, _field((case["rhs"], N), dt, gen), b


def _cgmn_inputs(case, seed):
    gen, n, rng = _gen(seed), _n(case), random.Random(seed)
    return _operator(n, case["pml"], case["ppw"], gen), _point_sources(n, case["pml"], case["rhs"], rng)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mvp":
        wn, x = _mvp_inputs(case, seed)
        return {"kind": kind, "grid": _grid(_n(case), case["pml"]), "wn": wn, "x": x, "mode": case["mode"],
                "deriv": case["deriv"]}
    if kind == "sweep":
        wn, x, b = _sweep_inputs(case, seed)
        return {"kind": kind, "grid": _grid(_n(case), case["pml"]), "wn": wn, "x": x, "b": b, "mode": case["mode"],
                "order": L.ORDER_LEX if case["order"] == "lex" else L.ORDER_BLOCK8}
    if kind == "cgmn":
        wn, b = _cgmn_inputs(case, seed)
        opts = solver.make_opts(tol=case["tol"], maxit=case["maxit"], precision=case["precision"])
        return {"kind": kind, "grid": _grid(_n(case), case["pml"]), "wn": wn, "b": b, "mode": case["mode"],
                "opts": opts}
    if kind == "batch":
        gen, rng, probs = _gen(seed), random.Random(seed), []
        for q, (n, rhs) in enumerate(_layout(case)):
            probs.append(solver.Problem(_grid(n, case["pml"]), _operator(n, case["pml"], case["ppw"], gen),
                                        _point_sources(n, case["pml"], rhs, rng), 1 + q % 2))
        return {"kind": kind, "probs": probs, "opts": solver.make_opts(tol=case["tol"], precision="mixed")}
    gen, rng = _gen(seed), random.Random(seed)
    n, pml = _n(case), case["pml"]
    v = _velocity([s - 2 * pml for s in n], gen)
    if kind == "mg":
        lv, R, P = multigrid.build_levels(v.cpu().numpy(), (H, H, H), pml, _freq(case["ppw"]), "m/s", device=DEV)
        return {"kind": kind, "levels": (lv, R, P), "b": _point_sources(n, pml, 1, rng)[0], "mode": case["mode"],
                "precision": case["precision"], "tol": case["tol"]}
    # fwi: sources and receivers off the grid near the surface; the observed data are those of
    # the direct wave in a constant medium, h^3 exp(i k r) / (4 pi r)
    ext = [(s - 2 * pml - 1) * H for s in n]
    src = [[rng.uniform(0.1, 0.9) * ext[0], rng.uniform(0.1, 0.9) * ext[1], 2 * H] for _ in range(case["sources"])]
    rec = [[rng.uniform(0.05, 0.95) * ext[0], rng.uniform(0.05, 0.95) * ext[1], H] for _ in range(case["receivers"])]
    f = _freq(case["ppw"])
    geom = fwi.Geometry(o=(0.0, 0.0, 0.0), d=(H, H, H), n=tuple(s - 2 * pml for s in n), npml6=(pml,) * 6,
                        src_xyz=src, rec_xyz=rec, freqs=[f], f0=8.0, unit="s2/m2")
    prob = fwi.FWIProblem(geom, fwi.FWIConfig(tol=case["tol"], precision="mixed", solver="mlgmres"))
    s, r = (torch.tensor(t, dtype=torch.float64, device=DEV) for t in (src, rec))
    dist = torch.cdist(r, s).clamp(min=H)
    dobs = torch.polar(H ** 3 / (4 * math.pi * dist), 2 * math.pi * f / 2000.0 * dist)
    return {"kind": kind, "prob": prob, "m": v ** -2, "dobs": dobs * f ** 2 * math.exp(-(f / 8.0) ** 2)}


def run(state):
    kind = state["kind"]
    if kind == "mvp":
        return ops.mvp(state["grid"], state["wn"], state["x"], state["mode"], state["deriv"])
    if kind == "sweep":
        return ops.kacz_sweep(state["grid"], state["wn"], 1.5, state["x"], state["b"], state["mode"], state["order"])
    if kind == "cgmn":
        return solver.solve(state["grid"], state["wn"], state["b"], state["mode"], state["opts"],
                            raise_not_converged=False)[0]
    if kind == "batch":
        return solver.solve_batch(state["probs"], state["opts"])[0]
    if kind == "mg":
        lv, R, P = state["levels"]
        return multigrid.solve(lv, R, P, state["b"], tol=state["tol"], mode=state["mode"],
                               precision=state["precision"])[0]
    m = state["m"].detach().requires_grad_(True)
    f = fwi.fwi_objective(m, state["prob"], state["dobs"])
    f.backward()
    return f.detach(), m.grad


# ---- work -----------------------------------------------------------------------------------------
def _pass_bytes(N, rhs, sc):
    # one pass over the operator: x read, y written, the wavenumber read
    return N * (2.0 * sc * rhs + sc / 2)


def work(case):
    """Bytes: every input read and every output written once per pass over the operator.  Flops:
    27 products of a complex value with a real coefficient per row and pass (a row projection
    twice that).  An iterative solve takes the passes of a nominal number of iterations."""
    kind = case["kind"]
    if kind == "batch":
        its = [0.6 * sum(n) * -math.log10(case["tol"]) for n, _ in _layout(case)]
        pts = [n[0] * n[1] * n[2] for n, _ in _layout(case)]
        rhs = [r for _, r in _layout(case)]
        return {"bytes": sum(i * 2 * _pass_bytes(N, r, 8) for i, N, r in zip(its, pts, rhs)),
                "flops": sum(i * 2 * 216.0 * N * r for i, N, r in zip(its, pts, rhs))}
    N = case["nx"] * case["ny"] * case["nz"]
    if kind == "mvp":
        sc = 8 if case["dtype"] == "c64" else 16
        return {"bytes": _pass_bytes(N, case["rhs"], sc) + (N * sc / 2 if case["cwn"] else 0),
                "flops": 108.0 * N * case["rhs"]}
    if kind == "sweep":
        sc = 8 if case["dtype"] == "c64" else 16
        return {"bytes": 2 * _pass_bytes(N, case["rhs"], sc) + N * sc * case["rhs"],
                "flops": 2 * 216.0 * N * case["rhs"]}
    if kind == "cgmn":
        sc = 8 if case["precision"] == "mixed" else 16
        its = min(case["maxit"], 0.6 * sum(_n(case)) * -math.log10(case["tol"])) + 1
        return {"bytes": its * 2 * _pass_bytes(N, case["rhs"], sc), "flops": its * 2 * 216.0 * N * case["rhs"]}
    # multigrid: an outer iteration gains about a digit and takes one FP64 matvec and, on the finest
    # level, 37 matvecs of the V-cycle (two smoothers of 15 steps with 3 true residuals each, and
    # the residual), 30 of them with an orthogonalisation against 1 to 5 basis vectors
    solves = 1 if kind == "mg" else 2 * case["sources"]
    sc = 8 if kind == "fwi" or case["precision"] == "mixed" else 16
    its = -math.log10(case["tol"]) + 2
    return {"bytes": solves * its * (_pass_bytes(N, 1, 16) + 37 * _pass_bytes(N, 1, sc) + 30 * 5 * N * sc),
            "flops": solves * its * N * (38 * 108.0 + 30 * 6 * 8.0)}


# ---- exact results in 64 bits -----------------------------------------------------------------------
# The 27-point operator from its definition: the weights of the four stencils (w1, w2, w3) and of
# the mass lumping (wm1..wm4), the PML functions xi per axis, one coefficient field per offset.
W1, W2, W3 = 1.8395262e-5, 0.296692333333333, 0.02747615
WM1, WM2, WM3, WM4 = 0.49649658, 0.07516875, 0.004373916666667, 5.690375e-07
OFFSETS = [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]


def _xi(n, p):
    """xi_lower and xi_upper of one axis at the points -1 .. n (width p on both sides)."""
    def lo(x):
        return math.cos(math.pi * (x - 1) * n / (2 * (n + 1) * p))

    def hi(x):
        return math.cos(math.pi * (1 - (x - 1) / (n + 1)) * n / (2 * p))

    def gamma(x):
        return lo(x) if x <= p else hi(x) if x > n + 2 - p else 0.0

    low, up = [], []
    for x in range(0, n + 2):
        g0, g1, g2 = (gamma(x + d) for d in (0, 1, 2))
        low.append(2.0 / (2.0 - g1 * (g1 + g0) + 1j * (3.0 * g1 + g0)))
        up.append(2.0 / (2.0 - g1 * (g1 + g2) + 1j * (3.0 * g1 + g2)))
    return [torch.tensor(t, dtype=torch.complex128, device=DEV) for t in (low, up)]


def _coefs(n, pml, wn, adjoint, deriv=False):
    """Coefficient fields (z, y, x) of the 27 offsets, one after another; wn complex128, x fastest.
    Forward coefficients of neighbours outside the grid are zero."""
    h2 = H * H
    w3a = W3 * 3 / (4 * 3 * h2)
    wn_c = -(W1 + 3 * W2 + 16 * w3a * 3 * h2 / 3 + WM1 - 1)
    centre = W1 / h2 + W2 / h2 + W2 / (2 * h2) * 2 + 8 * w3a
    edge = W2 / (2 * 2 * h2)
    shape = (n[2], n[1], n[0])
    w = wn.reshape(shape)
    wp = torch.nn.functional.pad(torch.view_as_real(w), (0, 0, 1, 1, 1, 1, 1, 1))
    wp = torch.view_as_complex(wp.contiguous())
    A, S = [], []
    for a in range(3):  # x, y, z: A[a][-1], A[a][+1] and the sum at the row
        low, up = _xi(n[a], pml)
        m = n[a]
        view = [1, 1, 1]
        view[2 - a] = m
        low_c, up_c = low[1:m + 1], up[1:m + 1]
        if adjoint:
            A.append({-1: up[0:m].reshape(view), 1: low[2:m + 2].reshape(view)})
        else:
            A.append({-1: low_c.reshape(view), 1: up_c.reshape(view)})
        S.append((low_c + up_c).reshape(view))
    inside = torch.nn.functional.pad(torch.ones(shape, device=DEV, dtype=torch.float64), (1,) * 6)
    for d in OFFSETS:
        on = [a for a in range(3) if d[a]]
        off = [a for a in range(3) if not d[a]]
        sl = tuple(slice(1 + d[a], 1 + d[a] + n[a]) for a in (2, 1, 0))
        wv = w if adjoint else wp[sl]
        c = (wn_c if not on else -(0.0, WM2, WM3, WM4)[len(on)]) * wv
        if not deriv:
            if not on:
                p = centre * (S[0] + S[1] + S[2])
            elif len(on) == 1:
                p = -centre * A[on[0]][d[on[0]]] + edge * (S[off[0]] + S[off[1]])
            elif len(on) == 2:
                p = -edge * (A[on[0]][d[on[0]]] + A[on[1]][d[on[1]]]) + 2 * w3a * S[off[0]]
            else:
                p = -2 * w3a * (A[0][d[0]] + A[1][d[1]] + A[2][d[2]])
            c = c + p
        c = c.expand(shape)
        yield c.conj() if adjoint else c * inside[sl]


def _padded(x, n):
    xr = torch.view_as_real(x.reshape(-1, n[2], n[1], n[0]))
    return torch.view_as_complex(torch.nn.functional.pad(xr, (0, 0, 1, 1, 1, 1, 1, 1)).contiguous())


def _exact_mvp(case, wn, x):
    n = _n(case)
    xp = _padded(x.to(torch.complex128), n)
    y = torch.zeros((x.shape[0], n[2], n[1], n[0]), dtype=torch.complex128, device=DEV)
    for d, c in zip(OFFSETS, _coefs(n, case["pml"], wn.to(torch.complex128), case["mode"] == 2, case["deriv"])):
        sl = (slice(None), *(slice(1 + d[a], 1 + d[a] + n[a]) for a in (2, 1, 0)))
        y += c * xp[sl]
    return y.reshape(x.shape)


class _ExactSweep:
    """Kaczmarz double sweeps in 64 bits: sets of independent rows one after another."""

    def __init__(self, n, pml, wn, mode, order):
        self.n = n
        self.coef = torch.stack([c.reshape(-1) for c in _coefs(n, pml, wn.to(torch.complex128), mode == 2)], 1)
        self.norm = (self.coef.real ** 2 + self.coef.imag ** 2).sum(1)
        N = self.norm.numel()
        q = torch.arange(N, device=DEV)
        i, j, k = q % n[0], (q // n[0]) % n[1], q // (n[0] * n[1])
        if order == "lex":
            key = i + 3 * j + 9 * k
        else:  # parity of the 12^3 block, then the colour inside it
            par = (i // 12) % 2 + 2 * ((j // 12) % 2) + 4 * ((k // 12) % 2)
            key = 27 * par + i % 3 + 3 * (j % 3) + 9 * (k % 3)
        rows = torch.argsort(key, stable=True)
        count = torch.bincount(key)
        self.sets = [s for s in torch.split(rows, count.tolist()) if s.numel()]
        px, pxy = n[0] + 2, (n[0] + 2) * (n[1] + 2)
        self.base = (i + 1) + px * (j + 1) + pxy * (k + 1)
        self.off = torch.tensor([dx + px * dy + pxy * dz for dx, dy, dz in OFFSETS], device=DEV)
        self.inside = _padded(torch.ones(1, N, dtype=torch.complex128, device=DEV), n).real.reshape(-1)

    def __call__(self, x, b, w=1.5):
        n = self.n
        xp = _padded(x.to(torch.complex128), n).reshape(x.shape[0], -1)
        for rows in self.sets + self.sets[::-1]:
            nbr = self.base[rows][:, None] + self.off
            c = self.coef[rows]
            xv = xp[:, nbr]
            d = -(c * xv).sum(2)
            if b is not None:
                d = d + b[:, rows]
            d = w * d / self.norm[rows]
            xp[:, nbr] = xv + d[:, :, None] * (c.conj() * self.inside[nbr])
        xp = xp.reshape(x.shape[0], n[2] + 2, n[1] + 2, n[0] + 2)
        return xp[:, 1:-1, 1:-1, 1:-1].reshape(x.shape)


def _exact_cgmn(case, wn, b):
    """The given number of CGMN iterations on (I - Q) x = DSWP(0, b), per column."""
    sweep = _ExactSweep(_n(case), case["pml"], wn, case["mode"], "block8")
    x = torch.zeros_like(b)
    r = sweep(x, b)
    p, rr = r.clone(), (r.real ** 2 + r.imag ** 2).sum(1)
    for _ in range(case["maxit"]):
        ap = p - sweep(p, None)
        alpha = rr / (p.conj() * ap).sum(1)
        x += alpha[:, None] * p
        r -= alpha[:, None] * ap
        new = (r.real ** 2 + r.imag ** 2).sum(1)
        p = r + (new / rr)[:, None] * p
        rr = new
    return x


def exact(case, seed):
    if case["kind"] == "mvp":
        return _exact_mvp(case, *_mvp_inputs(case, seed))
    if case["kind"] == "sweep":
        wn, x, b = _sweep_inputs(case, seed)
        return _ExactSweep(_n(case), case["pml"], wn, case["mode"], case["order"])(x, b.to(torch.complex128))
    if case["kind"] == "cgmn" and case["precision"] == "fp64":
        return _exact_cgmn(case, *_cgmn_inputs(case, seed))
    return None  # thousands of iterations: minutes in plain torch
