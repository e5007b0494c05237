"""Sizes at which the kernels of the solve, the mixed updates, the assembly and
the internal points change tile, path or remainder."""
import ctypes

import numpy as np
import pytest

from multifebe_gb300 import BemRegion, MfbemError, _abi, solve_lse
from multifebe_gb300 import meshgen as M

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


# panel widths 16 and 32, outer blocks of 64 and 128, 16-CTA panels (above 1200
# complex, 2400 real), the split block TRSM (4096 real columns to the right)
@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 33, 127, 128, 129, 257, 1199, 1201, 2305, 2403])
def test_lu_and_solve(n, cplx):
    """Backward errors of the factorisation and of the solve. Each entry of
    L U sums n products, each operation within 2 eps (4 eps complex): n times
    that of max(|L| |U|), and the same for each of the two triangular solves."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if cplx else 0)
    b = rng.standard_normal((n, 3)) + (1j * rng.standard_normal((n, 3)) if cplx else 0)
    F, x = np.array(A, order="F", copy=True), np.array(b, order="F", copy=True)
    _, ipiv = solve_lse(F, x)
    L, U = np.tril(F, -1) + np.eye(n), np.triu(F)
    p = np.arange(n)
    for k in range(n):
        j = ipiv[k] - 1
        assert k <= j < n
        p[[k, j]] = p[[j, k]]
    u = (4 if cplx else 2) * EPS
    size = np.abs(L) @ np.abs(U)
    assert np.abs(A[p] - L @ U).max() <= n * u * size.max()
    # multipliers of the |re| + |im| pivot
    assert np.abs(L).max() <= (np.sqrt(2) if cplx else 1.0) * (1 + 8 * EPS)
    assert (np.abs(A @ x - b) <= 3 * n * u * (size @ np.abs(x)).max(0)).all()


@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
def test_pivot_reciprocal_is_rounded_once(cplx):
    """The multiplier of an entry 1 is the pivot's reciprocal: each of its parts
    within half a unit in the last place, 2^-53 of |1 / d| in all."""
    rng = np.random.default_rng(11)
    for k in range(300):
        d = (1.0 + rng.random()) * 2.0 ** rng.integers(1, 30)
        if cplx:
            d = d * np.exp(2j * np.pi * rng.random())
        F = np.array([[d, 0.5], [1.0, 1.0]], dtype=np.complex128 if cplx else np.float64, order="F")
        solve_lse(F, np.ones((2, 1), dtype=F.dtype, order="F"))
        dl = np.clongdouble(d)
        exact = dl.conjugate() / (dl.real * dl.real + dl.imag * dl.imag)
        assert F[0, 0] == d and abs(np.clongdouble(F[1, 0]) - exact) <= 1.001 * EPS * abs(exact)


@pytest.mark.parametrize("cplx", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("e", [-980, 900])
def test_solve_of_tiny_and_huge_entries(e, cplx):
    """A and b times 2^e, large enough for updates on the tensor cores: the
    backward error of the solve as above (subnormal parts of an entry are 2^-90
    of the largest)."""
    n, s = 1100, 2.0 ** e
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if cplx else 0)
    b = rng.standard_normal((n, 2)) + (1j * rng.standard_normal((n, 2)) if cplx else 0)
    F, x = np.array(A * s, order="F", copy=True), np.array(b * s, order="F", copy=True)
    solve_lse(F, x)
    size = np.abs(np.tril(F, -1) + np.eye(n)) @ np.abs(np.triu(F) / s)
    u = (4 if cplx else 2) * EPS
    assert (np.abs(A @ x - b) <= 3 * n * u * (size @ np.abs(x)).max(0)).all()


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (63, 127, 15), (65, 129, 17), (130, 257, 33), (200, 300, 128)])
def test_binary16_split_of_uneven_rows_and_columns(m, n, k):
    """Rows of A and columns of B scaled over 2^+-20, one row and one column
    zero, entries down to 2^-24 of their row's largest. Split: each factor to
    2^-22 of itself and 2^-39 of its row's largest, lo lo left out (2^-22); FP32
    sums: three passes over ceil(2 k / 16) steps, each within 2^-22 of the sum
    of moduli; the last subtraction 2^-23 of C and the sum."""
    rng = np.random.default_rng(m + n + k)

    def cplx(r, c):
        x = rng.standard_normal((r, c)) + 1j * rng.standard_normal((r, c))
        return x * 2.0 ** rng.integers(-24, 1, size=(r, c))
    A = cplx(m, k) * 2.0 ** rng.integers(-20, 21, size=(m, 1))
    B = cplx(k, n) * 2.0 ** rng.integers(-20, 21, size=(1, n))
    A[m // 2], B[:, n // 2] = 0, 0
    if m == n == 1:
        A[0, 0], B[0, 0] = 3.0 + 1j, 2.0 - 5j
    C = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    A, B, C = (np.asfortranarray(v, dtype=np.complex64) for v in (A, B, C))
    L = _abi.load()
    L.mfbem_internal_tc_cgemm.argtypes = [ctypes.c_int32] * 3 + [ctypes.c_void_p] * 3 + [ctypes.c_int32]
    G = C.copy(order="F")
    _abi.check(L.mfbem_internal_tc_cgemm(m, n, k, A.ctypes.data, B.ctypes.data, G.ctypes.data, 0))
    A, B, C, G = (v.astype(np.complex128) for v in (A, B, C, G))
    a1, b1 = np.abs(A.real) + np.abs(A.imag), np.abs(B.real) + np.abs(B.imag)
    S = a1 @ b1
    top = a1.max(1)[:, None] * b1.max(0)[None, :]
    tol = (3 * 2.0 ** -22 + 3 * -(-2 * k // 16) * 2.0 ** -22) * S + 4 * k * 2.0 ** -39 * top + 2.0 ** -23 * (np.abs(C) + S)
    assert (np.abs(G - (C - A @ B)) <= tol).all()


@pytest.mark.parametrize("divs", [(1, 1, 1), (2, 1, 1), (3, 2, 1), (5, 3, 2), (7, 5, 3), (9, 6, 4)])
def test_mixed_solve_of_odd_sizes(divs):
    """Unpivoted panels, their remainders and the outer blocks: the mixed
    solution against the binary64 one (the bound of the mixed solves: 1e-9)."""
    d = M.box((1.0, 0.8, 0.6), divs)
    z = d.nodes[:, 2]
    d.ctype[z < 1e-9] = 0
    d.cvalue[z > 0.6 - 1e-9] = (0.0, 0.3, -1.0)
    R = BemRegion(d)
    xp = R.solve_staela(1.0, 0.25, precision="plain")
    xm = R.solve_staela(1.0, 0.25, precision="mixed")
    R.close()
    assert rel(xm, xp) < 1e-9


# 2220 unknowns: 172 columns beyond a multiple of 512, 44 of 128
@pytest.mark.parametrize("harmonic", [False, True], ids=["static", "harmonic"])
@pytest.mark.parametrize("width", [64, 128, 256, 512])
def test_mixed_solve_at_each_outer_block_width(width, harmonic, monkeypatch):
    """Outer blocks of one to four 128-column blocks, with interchanges and
    without: the mixed solution against the binary64 one (the bound of the mixed
    solves: 1e-9)."""
    monkeypatch.setenv("MFBEM_AUTOTUNE", str(width))
    d = M.cube_clamped_top_traction(6)
    mat = M.viscoelastic(1.0, 0.3, 1.0, 0.05)
    om = M.omega_from_a0([0.4, 1.1], mat)
    R = BemRegion(d)

    def run(precision):
        return R.sweep_harela(mat, om, precision=precision) if harmonic else \
            R.solve_staela(1.0, 0.25, precision=precision)
    xp = run("plain")
    for pivot in ("none", "partial"):
        monkeypatch.setenv("MFBEM_PIVOT", pivot)
        assert rel(run("mixed"), xp) < 1e-9
        assert R.last_stats["refactorizations"] == 0 and R.last_stats["gmres_iterations"] == 0
    R.close()


@pytest.mark.parametrize("harmonic", [False, True], ids=["static", "harmonic"])
def test_mixed_solves_repeat_bitwise(harmonic):
    """The unpivoted panel's diagonal block is read by up to 28 CTAs and written
    back by one of them (3462 rows): the same solve gives the same bits."""
    d = M.cube_clamped_top_traction(8)
    mat = M.viscoelastic(1.0, 0.3, 1.0, 0.05)
    R = BemRegion(d)
    x = [R.sweep_harela(mat, M.omega_from_a0([0.4, 1.1], mat), precision="mixed") if harmonic else
         R.solve_staela(1.0, 0.25, precision="mixed") for _ in range(4)]
    refactorizations = R.last_stats["refactorizations"]
    R.close()
    assert refactorizations == 0
    assert all((v == x[0]).all() for v in x[1:])


@pytest.mark.parametrize("m,n,k", [(1, 2, 1), (63, 127, 31), (65, 129, 33), (130, 300, 128), (200, 257, 300)])
def test_binary16_split_of_factors_in_units(m, n, k):
    """The factors of an LU with equations in units: index l carries 2^p_l in A
    and 2^-p_l in B (p over +-40), so their products are of one size. Split and
    sums as in the test above, top of the factors without the units (a power of
    two per l moves between A and B, and the split's choice of it differs from
    p by the spread of B's row maxima, 2^3 at most here)."""
    rng = np.random.default_rng(m + n + k)
    A, B = (rng.standard_normal(v) + 1j * rng.standard_normal(v) for v in ((m, k), (k, n)))
    C = rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    top = np.abs(A).max() * np.abs(B).max()
    u = 2.0 ** rng.integers(-40, 41, size=k)
    A, B, C = (np.asfortranarray(v, dtype=np.complex64) for v in (A * u, B / u[:, None], C))
    L = _abi.load()
    L.mfbem_internal_tc_cgemm.argtypes = [ctypes.c_int32] * 3 + [ctypes.c_void_p] * 3 + [ctypes.c_int32]
    G = C.copy(order="F")
    _abi.check(L.mfbem_internal_tc_cgemm(m, n, k, A.ctypes.data, B.ctypes.data, G.ctypes.data, 0))
    A, B, C, G = (v.astype(np.complex128) for v in (A, B, C, G))
    S = (np.abs(A.real) + np.abs(A.imag)) @ (np.abs(B.real) + np.abs(B.imag))
    tol = (3 * 2.0 ** -22 + 3 * -(-2 * k // 16) * 2.0 ** -22) * S + 8 * 4 * k * 2.0 ** -39 * top + \
        2.0 ** -23 * (np.abs(C) + S)
    assert (np.abs(G - (C - A @ B)) <= tol).all()


def scaled_solution(A, b):
    """x of A x = b: rows and columns scaled by powers of two to maxima near 1,
    refined with residuals in extended precision (the equations mix units, and
    a plain solution loses as many digits as they differ)."""
    p2 = lambda v: 2.0 ** -np.frexp(v)[1].astype(float)
    r = p2(np.abs(A).max(1))
    c = p2(np.abs(A * r[:, None]).max(0))
    S, sb = A * r[:, None] * c, b * r
    inv = np.linalg.inv(S)
    x = np.zeros(len(b), np.clongdouble)
    for _ in range(6):
        x = x + inv @ (sb - S.astype(np.clongdouble) @ x).astype(complex)
    return x.astype(complex) * c


@pytest.mark.parametrize("E", [1.0, 1e6, 8e10])
@pytest.mark.parametrize("region", ["crack", "codes"])
def test_mixed_sweep_of_sbie_and_hbie_rows_in_real_units(region, E):
    """SBIE and HBIE rows of one region differ by the shear modulus: the mixed
    sweep takes as many corrections in Pa as with a modulus of 1, and reaches
    the system's solution to the bound of the mixed sweeps (1e-8)."""
    if region == "crack":
        d, crack = M.penny_crack_in_box(1.0, 2, 1, 2.0, 2)
        R = BemRegion(d, crack=crack)
    else:
        d = M.cube_clamped_top_traction(4)
        f = np.full(d.n_nodes, 2, dtype=np.int32)
        f[d.nodes[:, 2] > 0.99] = 1
        f[d.nodes[:, 1] < 0.01] = 3
        f[d.nodes[:, 0] < 0.01] = 0
        R = BemRegion(d, formulation=f)
    mat = M.viscoelastic(E, 0.25, 1.0, 0.05)
    om = [float(M.omega_from_a0(a, mat)) for a in (0.4, 0.9)]
    X = R.sweep_harela(mat, om, precision="mixed")
    st = R.last_stats
    ref = [scaled_solution(*R.build_lse_harela(mat, w)) for w in om]
    R.close()
    # the counter is of all systems together, which go in step
    assert st["refactorizations"] == 0 and st["gmres_iterations"] == 0 and st["refinement_iterations"] <= 3, st
    for x, xr in zip(X, ref):
        assert rel(x, xr) < 1e-8


@pytest.mark.parametrize("E", [1e6, 1e9, 8e10])
@pytest.mark.parametrize("region", ["codes", "halves"])
def test_refinement_accepts_no_diverged_solution(region, E, monkeypatch):
    """FP32 factors with partial pivoting of SBIE / HBIE rows in Pa are no good
    preconditioner: whatever the refinement returns is a solution (its estimate
    of the error is below 1e-2, and a diverged x is off by its own size)."""
    monkeypatch.setenv("MFBEM_PIVOT", "partial")
    d = M.cube_clamped_top_traction(4)
    f = np.full(d.n_nodes, 2, dtype=np.int32)
    f[d.nodes[:, 2] > 0.99] = 1
    f[d.nodes[:, 1] < 0.01] = 3
    f[d.nodes[:, 0] < 0.01] = 0
    if region == "halves":
        f = (d.nodes[:, 0] > 0.4).astype(np.int32)
    R = BemRegion(d, formulation=f)
    mat = M.viscoelastic(E, 0.25, 1.0, 0.05)
    om = float(M.omega_from_a0(0.7, mat))
    ref = scaled_solution(*R.build_lse_harela(mat, om))
    try:
        x = R.sweep_harela(mat, [om], precision="mixed")[0]
    except MfbemError:
        x = None
    R.close()
    assert x is None or rel(x, ref) < 0.1


# 20, 56, 884 and 1154 nodes: 8 slices of a node's points, 3, and none (from 912)
@pytest.mark.parametrize("n", [1, 2, 7, 8])
def test_slices_of_a_nodes_points(oracle, n):
    d = M.cube_clamped_top_traction(n)
    R = BemRegion(d)
    A, b = R.build_lse_staela(1.0, 0.25)
    Ao, bo = oracle.Problem(d).assemble_staela(1.0, 0.25)
    R.close()
    assert rel(A, Ao) < 1e-11 and rel(b, bo) < 1e-11


# element groups of 32: 6, 24, 54 and 96 elements; 1 point, and so many that a
# warp takes several groups
@pytest.mark.parametrize("n,nip", [(1, 1), (2, 7), (3, 33), (4, 5000)])
def test_groups_of_elements_at_internal_points(oracle, n, nip):
    d = M.cube_confined_kat(n)
    rng = np.random.default_rng(nip)
    P = oracle.Problem(d)
    X = 0.4 + 0.2 * rng.random((nip, 3))
    A, b = P.assemble_staela(0.4, 0.25)
    u, t = P.solution(oracle.lu_solve(A, b))
    R = BemRegion(d)
    ui, si = R.internal_points(X, u, t, mu=0.4, nu=0.25)
    uo, so = P.internal_points(X, u, t, mu=0.4, nu=0.25)
    R.close()
    assert rel(ui, uo) < 1e-11 and rel(si, so) < 1e-11
