"""Timed cases of the collocation-BEM path: what a user of the framework has it
do, through the calls of multifebe_gb300.bem (the mirror of the reference's
builder / solver interface) and, where the caller owns device memory, the
C-ABI itself.

Families (the "kind" of a case):
  static     one static solve of an uploaded mesh (solve_staela)
  deck       a whole static job: deck -> mesh preparation and upload -> solve
             -> nodal u, t -> release
  sweep      a harmonic sweep of an uploaded box (sweep_harela)
  patch      a harmonic solve of an open free-surface patch
  batch      harmonic sweeps of several uneven cubes in one call
  assemble   one harmonic system of a plate built into device buffers
             (mfbem_assemble_harela with MFBEM_DEVICE_PTRS)
  dropin     the reference's own sequence on host arrays: build_lse_harela,
             then solve_lse
  lse        solve_lse on a given host system, with its options
  internal   internal points of a harmonic solution
  bm         a Burton & Miller (dual_bm_same) sweep
  footing    a static half-space footing (complementary kernel)
"""
import ctypes
import math

import numpy as np
import torch

from multifebe_gb300 import _abi, bem, meshgen

# ----------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------


def listed():
    return [
        # the smallest static job, deck to nodal solution: host preparation,
        # upload and launch latency (492 unknowns)
        {"name": "deck_static_cube3", "kind": "deck", "nx": 3, "ny": 3, "nz": 3, "precision": "plain"},
        # the static cube of the benchmark definition (870 unknowns)
        {"name": "static_cube4", "kind": "static", "nx": 4, "ny": 4, "nz": 4, "precision": "plain"},
        # a footing on a half-space: Mindlin's complementary kernel (675 unknowns)
        {"name": "footing8", "kind": "footing", "n": 8, "precision": "plain"},
        # one frequency of an odd box on host arrays, the reference's call
        # sequence (LAPACK semantics, complex128 throughout)
        {"name": "dropin_box5x4x6", "kind": "dropin", "nx": 5, "ny": 4, "nz": 6},
        # the drop-in's solver alone: a real system with equilibration and
        # iterative refinement, odd order, three right-hand sides
        {"name": "lse_r1999_refine", "kind": "lse", "n": 1999, "nrhs": 3, "cplx": False, "options": True},
        # the FP64 harmonic sweep (plain method) of the 8x8 cube, 4 frequencies
        {"name": "sweep_cube8x4_plain", "kind": "sweep", "nx": 8, "ny": 8, "nz": 8, "nf": 4, "precision": "plain"},
        # the benchmark sweep: 8x8 cube, 20 frequencies, mixed precision
        {"name": "sweep_cube8x20_mixed", "kind": "sweep", "nx": 8, "ny": 8, "nz": 8, "nf": 20, "precision": "mixed"},
        # the precision workload: 40x40 surface patch (14883 unknowns)
        {"name": "patch40_mixed", "kind": "patch", "n": 40, "nf": 1, "precision": "mixed"},
        # 48 uneven problems: cubes 4..10, 8 frequencies each
        {"name": "batch_cubes4_10", "kind": "batch", "sizes": "4,5,6,7,8,10", "nf": 8},
        # one FP64 system of a thin plate into the caller's device buffers
        # (quasi-singular pairs across the thickness)
        {"name": "assemble_slab16", "kind": "assemble", "n": 16, "nz": 1, "thickness": 0.02},
        # displacement and stress at 300 points from a harmonic solution
        {"name": "internal_cube6", "kind": "internal", "n": 6, "points": 300},
        # Burton & Miller collocation, 2 frequencies
        {"name": "bm_cube5x2", "kind": "bm", "n": 5, "nf": 2},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["static", "deck", "footing", "dropin", "lse", "sweep", "sweep", "sweep", "patch", "batch",
                       "assemble", "internal", "bm"])
    if kind in ("static", "deck"):
        return {"kind": kind, "nx": rng.randint(2, 7), "ny": rng.randint(2, 7), "nz": rng.randint(2, 7),
                "precision": rng.choice(["plain", "mixed"])}
    if kind == "footing":
        return {"kind": kind, "n": rng.randint(3, 12), "precision": rng.choice(["plain", "mixed"])}
    if kind == "dropin":
        return {"kind": kind, "nx": rng.randint(2, 6), "ny": rng.randint(2, 6), "nz": rng.randint(2, 6)}
    if kind == "lse":
        c = rng.random() < 0.5
        return {"kind": kind, "n": log_int(150, 1800 if c else 2600), "nrhs": rng.randint(1, 4), "cplx": c,
                "options": rng.random() < 0.5}
    if kind == "sweep":
        nx, ny, nz = rng.randint(2, 9), rng.randint(2, 9), rng.randint(2, 9)
        el = 2 * (nx * ny + ny * nz + nx * nz)
        p = rng.choice(["plain", "mixed", "mixed"])
        most = max(1, int((8 if p == "plain" else 20) * (384 / el) ** 2))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "nf": log_int(1, min(20, most)), "precision": p}
    if kind == "patch":
        p = rng.choice(["mixed", "mixed", "plain"])
        return {"kind": kind, "n": rng.randint(9, 24 if p == "plain" else 39), "nf": 1, "precision": p}
    if kind == "batch":
        k = rng.randint(2, 5)
        return {"kind": kind, "sizes": ",".join(str(rng.randint(2, 9)) for _ in range(k)), "nf": rng.randint(1, 8)}
    if kind == "assemble":
        return {"kind": kind, "n": rng.randint(4, 15), "nz": rng.randint(1, 2),
                "thickness": round(math.exp(rng.uniform(math.log(0.02), math.log(0.3))), 4)}
    if kind == "internal":
        return {"kind": kind, "n": rng.randint(2, 7), "points": log_int(10, 400)}
    return {"kind": "bm", "n": rng.randint(2, 5), "nf": rng.randint(1, 3)}


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------


def _material(rng, nu=0.25, xi=0.05):
    """The viscoelastic region of the benchmark definition, its constants moved a little."""
    return meshgen.viscoelastic(1.0, nu + 0.05 * (rng.random() - 0.5), 1.0, xi * (0.8 + 0.4 * rng.random()))


def _load(rng):
    return (0.3 * (rng.random() - 0.5), 0.3 * (rng.random() - 0.5), -1.0 - 0.2 * rng.random())


def _box(c, rng):
    """Box clamped at its bottom, loaded at its top, dimensions near 1."""
    dims = 0.9 + 0.2 * rng.random(3)
    d = meshgen.box(dims, (c["nx"], c["ny"], c["nz"]))
    z = d.nodes[:, 2]
    d.cvalue[np.abs(z - dims[2]) <= 1e-12] = np.asarray(_load(rng), dtype=np.complex128)
    bottom = np.abs(z) <= 1e-12
    d.ctype[bottom] = 0
    d.cvalue[bottom] = 0.0
    return d


def _cube(n, rng):
    return _box({"nx": n, "ny": n, "nz": n}, rng)


def _omegas(nf, mat, rng, lo=0.1, hi=2.0):
    a0 = np.array([1.0]) if nf == 1 else np.linspace(lo, hi, nf)
    return meshgen.omega_from_a0(a0 * (0.95 + 0.1 * rng.random()), mat)


def _lse_system(c, seed):
    """A second-kind system like a BEM one: a dominant diagonal (the free
    terms) and an off-diagonal kernel that falls with the distance, rows of
    different scale (mixed displacement and traction unknowns)."""
    n, rng = c["n"], np.random.default_rng(seed)
    A = rng.standard_normal((n, n))
    if c["cplx"]:
        A = A + 1j * rng.standard_normal((n, n))
    x = rng.random(n)
    A *= 0.3 / (1.0 + 0.2 * n * np.abs(x[:, None] - x[None, :]))
    A[np.arange(n), np.arange(n)] += 2.0
    if c["options"]:
        A *= np.exp(2.0 * rng.standard_normal(n))[:, None]
    b = rng.standard_normal((n, c["nrhs"]))
    if c["cplx"]:
        b = b + 1j * rng.standard_normal((n, c["nrhs"]))
    return np.asfortranarray(A), np.asfortranarray(b)


def _internal_inputs(c, seed):
    rng = np.random.default_rng(seed)
    d = _cube(c["n"], rng)
    mat = _material(rng)
    om = float(_omegas(1, mat, rng)[0])
    X = d.nodes
    k = 1.0 + rng.random((2, 3))
    ph = 2.0 * np.pi * rng.random((2, 3))
    # smooth nodal fields, as a solution has them
    u = np.exp(1j * (X @ k.T[:, :1] + ph[0])) * (0.5 + rng.random(3))
    t = np.exp(1j * (X @ k.T[:, 1:] + ph[1])) * (0.5 + rng.random(3))
    lo, hi = X.min(0), X.max(0)
    xip = lo + (hi - lo) * (0.15 + 0.7 * rng.random((c["points"], 3)))
    return d, mat, om, np.ascontiguousarray(xip), np.ascontiguousarray(u), np.ascontiguousarray(t)


def prepare(case, seed):
    c, rng = case, np.random.default_rng(seed)
    kind = c["kind"]
    if kind in ("static", "deck"):
        d = _box(c, rng)
        m = meshgen.elastic(1.0, 0.25 + 0.05 * (rng.random() - 0.5))
        return {"c": c, "deck": d, "m": m, "R": bem.BemRegion(d) if kind == "static" else None}
    if kind == "footing":
        a = 0.8 + 0.4 * rng.random()
        R = bem.BemRegion(meshgen.halfspace_footing(a, c["n"], 1.0 + rng.random()))
        R.set_halfspace(-3, 0.0, 1)
        return {"c": c, "R": R, "m": meshgen.elastic(1.0, 0.3 + 0.05 * (rng.random() - 0.5))}
    if kind == "dropin":
        mat = _material(rng)
        return {"c": c, "R": bem.BemRegion(_box(c, rng)), "m": mat, "om": float(_omegas(1, mat, rng)[0])}
    if kind == "lse":
        A, b = _lse_system(c, seed)
        return {"c": c, "A": A, "b": b}
    if kind == "sweep":
        mat = _material(rng)
        return {"c": c, "R": bem.BemRegion(_box(c, rng)), "m": mat, "om": _omegas(c["nf"], mat, rng)}
    if kind == "patch":
        mat = _material(rng, 0.33)
        half = 9.0 + 2.0 * rng.random()
        d = meshgen.surface_patch(half, c["n"], max(1.0, half / c["n"] * 2.0), _load(rng))
        om = meshgen.omega_from_a0([0.5 * (0.9 + 0.2 * rng.random())], mat)
        return {"c": c, "R": bem.BemRegion(d), "m": mat, "om": om}
    if kind == "batch":
        mat = _material(rng)
        om = _omegas(c["nf"], mat, rng, 0.2, 1.6)
        Rs = [bem.BemRegion(_cube(int(n), rng)) for n in c["sizes"].split(",")]
        return {"c": c, "R": Rs, "m": mat, "om": [om] * len(Rs)}
    if kind == "assemble":
        mat = _material(rng, 0.3, 0.02)
        d = meshgen.slab(c["n"], c["nz"], (0.9 + 0.2 * rng.random(), 0.9 + 0.2 * rng.random(), c["thickness"]),
                         _load(rng))
        R = bem.BemRegion(d)
        A = torch.empty((R.n, R.n), dtype=torch.complex128, device="cuda")  # column-major for the library
        b = torch.empty(R.n, dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        return {"c": c, "R": R, "m": mat, "om": float(_omegas(1, mat, rng)[0]), "A": A, "b": b}
    if kind == "internal":
        d, mat, om, xip, u, t = _internal_inputs(c, seed)
        return {"c": c, "R": bem.BemRegion(d), "m": mat, "om": om, "xip": xip, "u": u, "t": t}
    if kind == "bm":
        mat = _material(rng)
        R = bem.BemRegion(_cube(c["n"], rng), formulation="dual_bm", alpha=1.0)
        return {"c": c, "R": R, "m": mat, "om": _omegas(c["nf"], mat, rng, 0.5, 2.0)}
    raise ValueError(kind)


# ----------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------


def run(state):
    s, c = state, state["c"]
    kind = c["kind"]
    if kind in ("static", "footing"):
        return s["R"].solve_staela(s["m"]["mu"], s["m"]["nu"], c["precision"])
    if kind == "deck":
        R = bem.BemRegion(s["deck"])
        u, t = R.solution(R.solve_staela(s["m"]["mu"], s["m"]["nu"], c["precision"]))
        R.close()
        return u, t
    if kind in ("sweep", "patch"):
        return s["R"].sweep_harela(s["m"], s["om"], c["precision"])
    if kind == "bm":
        return s["R"].sweep_harela(s["m"], s["om"], "mixed")
    if kind == "batch":
        return bem.sweep_harela_batch(s["R"], s["m"], s["om"])[0]
    if kind == "dropin":
        A, b = s["R"].build_lse_harela(s["m"], s["om"])
        x, _ = bem.solve_lse(A, b)
        return x
    if kind == "lse":
        # the solver overwrites its system, which a user's program has just built
        A, b = s["A"].copy(order="F"), s["b"].copy(order="F")
        if c["options"]:
            x, ipiv = bem.solve_lse(A, b, scaling=True, refine=True, state=bem.LseState())
        else:
            x, ipiv = bem.solve_lse(A, b)
        return x, A, ipiv  # the solution, the LU factors in place of A and the pivots, as LAPACK leaves them
    if kind == "assemble":
        m = s["m"]
        dp = ctypes.POINTER(ctypes.c_double)
        lam, mu, nu = (np.array([complex(m[k]).real, complex(m[k]).imag]) for k in ("lambda", "mu", "nu"))
        _abi.check(_abi.load().mfbem_assemble_harela(
            s["R"]._h, lam.ctypes.data_as(dp), mu.ctypes.data_as(dp), float(m["rho"]), nu.ctypes.data_as(dp), s["om"],
            ctypes.cast(s["A"].data_ptr(), dp), s["R"].n, ctypes.cast(s["b"].data_ptr(), dp),
            _abi.MFBEM_DEVICE_PTRS | _abi.MFBEM_OVERWRITE))
        return s["A"], s["b"]
    if kind == "internal":
        return s["R"].internal_points(s["xip"], s["u"], s["t"], mat=s["m"], omega=s["om"])
    raise ValueError(kind)


# ----------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------


def _box_sizes(nx, ny, nz):
    e = 2 * (nx * ny + ny * nz + nx * nz)
    return e, 3 * e + 2


def _assembly(ne, nn, cplx, dual=1):
    """(bytes, flops) of integrating every (point, element) pair at the
    smallest precalculated rule (2 x 2 points): 15 kernel components (u*
    symmetric) weighted by 8 shape functions; kernels at 60 (real) or 300
    (complex) operations a point."""
    per = 4 * ((2 * 15 * 8) * (2 if cplx else 1) + (300 if cplx else 60))
    return 8 * (3 * nn + 3 * nn) + 32 * ne, float(per) * ne * nn * dual


def _lu(n, cplx):
    return (8.0 / 3.0 if cplx else 2.0 / 3.0) * float(n) ** 3


def work(case):
    c = case
    kind = c["kind"]
    if kind in ("static", "deck"):
        ne, nn = _box_sizes(c["nx"], c["ny"], c["nz"])
        by, fl = _assembly(ne, nn, False)
        return {"bytes": by + 24 * nn, "flops": fl + _lu(3 * nn, False)}
    if kind == "footing":
        n = c["n"]
        ne, nn = n * n, 3 * n * n + 4 * n + 1
        by, fl = _assembly(ne, nn, False, 2)
        return {"bytes": by + 24 * nn, "flops": fl + _lu(3 * nn, False)}
    if kind in ("dropin", "sweep"):
        nf = c.get("nf", 1)
        ne, nn = _box_sizes(c["nx"], c["ny"], c["nz"])
        by, fl = _assembly(ne, nn, True)
        host = 3 * 16 * (3 * nn) ** 2 if kind == "dropin" else 0  # A out of the builder, into and out of the solver
        return {"bytes": by + 48 * nn * nf + host, "flops": nf * (fl + _lu(3 * nn, True))}
    if kind == "patch":
        n = c["n"]
        ne, nn = n * n, 3 * n * n + 4 * n + 1
        by, fl = _assembly(ne, nn, True)
        return {"bytes": by + 48 * nn, "flops": fl + _lu(3 * nn, True)}
    if kind == "batch":
        b = f = 0
        for n in c["sizes"].split(","):
            ne, nn = _box_sizes(int(n), int(n), int(n))
            by, fl = _assembly(ne, nn, True)
            b += by + 48 * nn * c["nf"]
            f += c["nf"] * (fl + _lu(3 * nn, True))
        return {"bytes": b, "flops": f}
    if kind == "bm":
        ne, nn = _box_sizes(c["n"], c["n"], c["n"])
        by, fl = _assembly(ne, 8 * ne, True, 2)  # a point per element node, SBIE and HBIE
        return {"bytes": by + 48 * nn * c["nf"], "flops": c["nf"] * (fl + _lu(3 * nn, True))}
    if kind == "assemble":
        ne, nn = _box_sizes(c["n"], c["n"], c["nz"])
        by, fl = _assembly(ne, nn, True)
        return {"bytes": by + 16 * (3 * nn) ** 2, "flops": fl}
    if kind == "lse":
        n, k = c["n"], 16 if c["cplx"] else 8
        return {"bytes": 2 * k * (n * n + n * c["nrhs"]), "flops": _lu(n, c["cplx"])}
    ne, nn = _box_sizes(c["n"], c["n"], c["n"])
    # u*, t* and, for the stresses, d*, s* contracted with the nodal values
    return {"bytes": 24 * nn + 96 * nn + 216 * c["points"], "flops": 4.0 * 2500 * ne * c["points"]}


# ----------------------------------------------------------------------------
# the same in 64 bits without the framework, where that is a matter of seconds
# ----------------------------------------------------------------------------


def _stokes(r, k1, k2):
    """psi, chi and their derivatives of u* = (psi I - chi r,l r,k) / (4 pi mu)."""
    def wave(k):
        a = torch.exp(-1j * k * r) / r
        s = 1j * k + 1.0 / r
        a1 = -s * a
        a2 = (s * s + 1.0 / r ** 2) * a
        a3 = -(s ** 3 + 3.0 * s / r ** 2 + 2.0 / r ** 3) * a
        return a, a1, a2, a3
    p, q = wave(k1), wave(k2)
    d = [y - x for x, y in zip(p, q)]
    psi = q[0] + d[1] / r / k2 ** 2
    psi1 = q[1] + (d[2] / r - d[1] / r ** 2) / k2 ** 2
    chi = -(d[2] - d[1] / r) / k2 ** 2
    chi1 = -(d[3] - d[2] / r + d[1] / r ** 2) / k2 ** 2
    return psi, chi, psi1, chi1


def _internal_u(case, seed):
    """u at the points by 16 x 16 Gauss points on every (flat) element."""
    d, mat, om, xip, u, t = _internal_inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    g, w = np.polynomial.legendre.leggauss(16)
    x1, x2 = (a.ravel() for a in np.meshgrid(g, g, indexing="ij"))
    w = np.outer(w, w).ravel()
    corners = [(-1, -1), (1, -1), (1, 1), (-1, 1)]
    phi = [0.25 * (1 + a * x1) * (1 + b * x2) * (a * x1 + b * x2 - 1) for a, b in corners]
    phi += [0.5 * (1 - x1 ** 2) * (1 - x2), 0.5 * (1 + x1) * (1 - x2 ** 2), 0.5 * (1 - x1 ** 2) * (1 + x2),
            0.5 * (1 - x1) * (1 - x2 ** 2)]
    phi = np.array(phi)  # [8][256]
    X = d.nodes[d.conn]  # [ne][8][3]
    e1, e2 = (X[:, 1] - X[:, 0]) / 2, (X[:, 3] - X[:, 0]) / 2
    nv = np.cross(e1, e2)
    jac = np.linalg.norm(nv, axis=1)
    nrm = T(np.repeat(nv / jac[:, None], len(w), 0))
    pts = T(np.einsum("kp,ekc->epc", phi, X).reshape(-1, 3))
    W = T((jac[:, None] * w[None, :]).ravel())
    uq = T(np.einsum("kp,ekc->epc", phi, u[d.conn]).reshape(-1, 3))
    tq = T(np.einsum("kp,ekc->epc", phi, t[d.conn]).reshape(-1, 3))
    mu, lam, rho = complex(mat["mu"]), complex(mat["lambda"]), mat["rho"]
    k1, k2 = om / np.sqrt((lam + 2 * mu) / rho), om / np.sqrt(mu / rho)
    out = []
    for x in T(xip):
        rv = pts - x
        r = rv.norm(dim=1)
        dr = rv / r[:, None]
        psi, chi, psi1, chi1 = _stokes(r, k1, k2)
        rn = (dr * nrm).sum(1)
        dt, du, un = (dr * tq).sum(1), (dr * uq).sum(1), (nrm * uq).sum(1)
        c = lambda v: v[:, None]  # noqa: E731
        g = (c(psi) * tq - c(chi * dt) * dr) / (4 * math.pi * mu)
        a = psi1 - chi / r
        h = c(a * rn) * uq + c(a * du) * nrm  # (psi' - chi/r) (delta r,n + r,k n_l)
        h = h - c(2 * chi / r) * (c(un) * dr - c(2 * du * rn) * dr)
        h = h - c(2 * chi1 * du * rn) * dr + c((lam / mu) * (psi1 - chi1 - 2 * chi / r) * un) * dr
        out.append(((g - h / (4 * math.pi)) * c(W)).sum(0))
    return torch.stack(out).cpu().numpy()


def exact(case, seed):
    """Solver outputs and the displacements of internal points. The other
    outputs are defined by the reference's own quadrature (which rule, how
    many subdivisions a pair takes), so their 64-bit values are another
    implementation of the whole method: None."""
    if case["kind"] == "lse":
        A, b = _lse_system(case, seed)
        x = np.linalg.solve(A, b)
        for _ in range(2):
            x = x + np.linalg.solve(A, b - A @ x)
        return x, None, None
    if case["kind"] == "internal":
        return _internal_u(case, seed), None
    return None
