"""Internal points on the device (mfbem_internal_points_{staela,harela}) against
the oracle's restatement of calculate_internal_points_mechanics_bem_* and the
closed forms of docs/examples/ME-ST-EL-002 and ME-TH-EL-001. Both sides get
the same nodal solution, so the comparison isolates the internal-point step.

Tolerances (max-norm relative to the largest value): displacement and stress
<= 1e-11 against the oracle (FP64 on both sides; FMA contraction and the
device's transcendental functions); <= 1e-9 where quasi-singular subdivision
dominates (thin slab)."""
import ctypes

import numpy as np
import pytest

from multifebe_gb300 import MfbemError, BemRegion, meshgen as M, _abi
from test_oracle_kat import INTERIOR, _p_wave_column

pytestmark = pytest.mark.gpu


def _loads(name):
    try:
        return bool(ctypes.CDLL(name))
    except OSError:
        return False


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def test_static_internal_points(oracle):
    d = M.cube_confined_kat(2)
    mat = M.elastic(1.0, 0.25)
    P = oracle.Problem(d, qsi_re=1e-10)
    A, b = P.assemble_staela(mat["mu"], mat["nu"])
    u, t = P.solution(oracle.lu_solve(A, b))
    R = BemRegion(d, qsi_relative_error=1e-10)
    ui, si = R.internal_points(INTERIOR, u, t, mu=mat["mu"], nu=mat["nu"])
    uo, so = P.internal_points(INTERIOR, u, t, mu=mat["mu"], nu=mat["nu"])
    R.close()
    assert rel(ui, uo) < 1e-11 and rel(si, so) < 1e-11, (rel(ui, uo), rel(si, so))
    assert np.abs(ui[:, 0] - (1.25 * 0.5 / 0.75) * INTERIOR[:, 0]).max() < 1e-9
    assert np.abs(si - np.diag([1.0, 1.0 / 3.0, 1.0 / 3.0])).max() < 5e-8


@pytest.mark.parametrize("om", [2.0, 5.0])
def test_harmonic_internal_points(oracle, om):
    d = M.cube_confined_kat(4)
    mat = M.viscoelastic(2.4, 0.2, 1.0, 0.02)
    P = oracle.Problem(d)
    A, b = P.assemble_harela(mat, om)
    u, t = P.solution(oracle.lu_solve(A, b))
    R = BemRegion(d)
    ui, si = R.internal_points(INTERIOR, u, t, mat=mat, omega=om)
    uo, so = P.internal_points(INTERIOR, u, t, mat=mat, omega=om)
    R.close()
    assert rel(ui, uo) < 1e-11 and rel(si, so) < 1e-11, (rel(ui, uo), rel(si, so))
    ue = _p_wave_column(mat, om, INTERIOR[:, 0])
    assert np.abs(ui[:, 0] - ue).max() / np.abs(ue).max() < (3e-3 if om > 3 else 1e-4)


def test_thin_slab_quasi_singular_internal_points(oracle):
    """Points inside a slab 0.02 thick: every pair with the nearby faces is
    quasi-singular (subdivision trees for both the SBIE and the HBIE)."""
    d = M.slab(4, 1)
    mat = M.viscoelastic(1.0, 0.3, 1.0, 0.02)
    om = float(M.omega_from_a0([0.5], mat)[0])
    P = oracle.Problem(d)
    A, b = P.assemble_harela(mat, om)
    u, t = P.solution(oracle.lu_solve(A, b))
    rng = np.random.default_rng(4)
    xy = rng.uniform(0.1, 0.9, (12, 2))
    z = np.array([0.01, 0.004, 0.016] * 4)
    xip = np.column_stack([xy, z])
    R = BemRegion(d)
    ui, si = R.internal_points(xip, u, t, mat=mat, omega=om)
    uo, so = P.internal_points(xip, u, t, mat=mat, omega=om)
    R.close()
    assert rel(ui, uo) < 1e-9 and rel(si, so) < 1e-9, (rel(ui, uo), rel(si, so))


def test_internal_points_at_nodes_and_on_elements():
    d = M.cube_confined_kat(2)
    mat = M.elastic(1.0, 0.25)
    R = BemRegion(d)
    rng = np.random.default_rng(1)
    u = rng.normal(size=(d.n_nodes, 3))
    t = rng.normal(size=(d.n_nodes, 3))
    for s in (7, 20):
        ui, si = R.internal_points(d.nodes[s:s + 1], u, t, mu=mat["mu"], nu=mat["nu"])
        last = np.flatnonzero(np.linalg.norm(d.nodes - d.nodes[s], axis=1) < 1e-12).max()
        assert np.array_equal(ui[0], u[last]) and np.all(si == 0)
    e = d.conn[0]
    xm = 0.25 * (d.nodes[e[0]] + d.nodes[e[4]]) + 0.25 * (d.nodes[e[4]] + d.nodes[e[6]])
    with pytest.raises(MfbemError) as ex:
        R.internal_points(np.vstack([INTERIOR[:1], xm[None, :]]), u, t, mu=mat["mu"], nu=mat["nu"])
    assert ex.value.code == _abi.MFBEM_EUNSUPPORTED
    R.close()


def test_points_of_a_mesh_in_several_launches(oracle):
    """Sixteen precalculated rules up to the largest (9944 points an element): the
    294 elements of a harmonic region go through in launches of 256 and 38, the
    second adding to the sums of the first."""
    gl = tuple(range(17, 33))
    d = M.cube_clamped_top_traction(7)
    mat = M.viscoelastic(1.0, 0.25, 1.0, 0.05)
    om = float(M.omega_from_a0(0.7, mat))
    rng = np.random.default_rng(6)
    X = 0.1 + 0.8 * rng.random((40, 3))
    X[0] = d.nodes[3]
    u, t = (rng.standard_normal((d.n_nodes, 3)) + 1j * rng.standard_normal((d.n_nodes, 3)) for _ in range(2))
    P = oracle.Problem(d, ps_gln=gl)
    R = BemRegion(d, precalset_gln=gl)
    ui, si = R.internal_points(X, u, t, mat=mat, omega=om)
    uo, so = P.internal_points(X, u, t, mat=mat, omega=om)
    R.close()
    assert rel(ui, uo) < 1e-11 and rel(si, so) < 1e-11


def test_work_buffers_go_back_after_the_call():
    """Points x elements decide the work space of a call; once it is over,
    mfbem_trim_device_cache gives all of the large buffers back."""
    L = _abi.load()
    rt = next(ctypes.CDLL(n) for n in ("libcudart.so.13", "libcudart.so") if _loads(n))
    d = M.cube_clamped_top_traction(5)
    n = d.n_nodes
    X = np.random.default_rng(1).random((40000, 3)) * 0.2 + 0.4
    R = BemRegion(d)
    R.internal_points(X[:10], np.zeros((n, 3)), np.ones((n, 3)), mu=0.4, nu=0.25)

    def free():
        assert L.mfbem_trim_device_cache() == 0
        fr, tot = ctypes.c_size_t(), ctypes.c_size_t()
        assert rt.cudaMemGetInfo(ctypes.byref(fr), ctypes.byref(tot)) == 0
        return fr.value
    before = free()
    R.internal_points(X, np.zeros((n, 3)), np.ones((n, 3)), mu=0.4, nu=0.25)
    left = before - free()
    R.close()
    # classes alone take 12 MB; buffers below 1 MB may stay with the handle
    assert left <= 8 << 20, left
