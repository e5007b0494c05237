"""Radial tables of the harmonic kernels: the tabulated functions against 40
digits, and the assembly on both sides of the rule that chooses the table."""
import ctypes

import numpy as np
import pytest

from multifebe_gb300 import BemRegion, _abi
from multifebe_gb300 import meshgen as M

pytestmark = pytest.mark.gpu


def _exact(mp, q, r):
    """psi, chi, TT1..TT3 without their constants, from the waves e^-ikr / r (bem_harela3d.f90:118-134, 654-688)."""
    I, one = mp.mpc(0, 1), mp.mpf(1)
    lam, mu, rho, om = mp.mpc(q[0], q[1]), mp.mpc(q[2], q[3]), mp.mpf(q[4]), mp.mpf(q[5])
    c1, c2 = mp.sqrt((lam + 2 * mu) / rho), mp.sqrt(mu / rho)
    k1, k2 = om / c1, om / c2
    g = c2 ** 2 / c1 ** 2

    def wave(k):  # e^-ikr / r and its first four derivatives in r
        a, s = mp.exp(-I * k * r) / r, -I * k
        p = [one, s - 1 / r, s ** 2 - 2 * s / r + 2 / r ** 2,
             s ** 3 - 3 * s ** 2 / r + 6 * s / r ** 2 - 6 / r ** 3,
             s ** 4 - 4 * s ** 3 / r + 12 * s ** 2 / r ** 2 - 24 * s / r ** 3 + 24 / r ** 4]
        return [a * x for x in p]

    a, b = wave(k1), wave(k2)
    d = [y - x for x, y in zip(a, b)]
    psi = [b[0] + d[1] / r / k2 ** 2, b[1] + (d[2] / r - d[1] / r ** 2) / k2 ** 2,
           b[2] + (d[3] / r - 2 * d[2] / r ** 2 + 2 * d[1] / r ** 3) / k2 ** 2]
    chi = [-(d[2] - d[1] / r) / k2 ** 2, -(d[3] - d[2] / r + d[1] / r ** 2) / k2 ** 2,
           -(d[4] - d[3] / r + 2 * d[2] / r ** 2 - 2 * d[1] / r ** 3) / k2 ** 2]
    # t*: TT1 r,l r,k r,n + TT2 (delta r,n + n_l r,k) + TT3 r,l n_k
    z = 1 / g - 2  # lambda / mu
    t1 = -2 * chi[1] + 4 * chi[0] / r
    t2 = psi[1] - chi[0] / r
    t3 = z * (psi[1] - chi[1] - 2 * chi[0] / r) - 2 * chi[0] / r
    return psi[0], chi[0], t1, t2, t3


@pytest.mark.parametrize("nu,xi,om", [(0.25, 0.05, 1.2), (0.33, 0.05, 0.3), (0.49, 0.0, 2.0), (0.0, 0.1, 30.0),
                                      (0.25, 0.02, 1e-3)])
def test_radial_functions(nu, xi, om):
    """Error relative to r^-p + |k|^p (p = 1 for psi and chi, 2 for TT1..TT3),
    the size of the singular and the entire part. Binary64: the terms of an
    entire part sum to up to 4.5 |k|^p for each of the two wavenumbers, each
    good to about 2 eps, and the Chebyshev conversion can double it: 40 eps.
    Double-float: eight operations of 2^-47. The direct evaluation sums the same
    terms: the table may be at most twice as far off in the worst sample."""
    mp = pytest.importorskip("mpmath")
    mp.mp.dps = 50
    L = _abi.load()
    L.mfbem_internal_radial.argtypes = [ctypes.c_void_p, ctypes.c_double, ctypes.c_int32] + [ctypes.c_void_p] * 4
    m = M.viscoelastic(1.0, nu, 1.0, xi)
    q = np.array([m["lambda"].real, m["lambda"].imag, m["mu"].real, m["mu"].imag, 1.0, om])
    k2 = om / m["c_s"]
    rng = np.random.default_rng(11)
    # distances over the mesh, interval ends and both neighbours among them
    rmax = 3.0
    h = min(0.125 / abs(om / np.sqrt(m["mu"])), rmax)
    r = np.concatenate([10.0 ** rng.uniform(-4, np.log10(rmax), 120), h * np.arange(1, 9), h * np.arange(1, 9) * (1 - 1e-15),
                        [rmax]])
    r = np.minimum(r, rmax)
    n = len(r)
    tab, tabf, dr = np.zeros((n, 10, 2)), np.zeros((n, 5, 2)), np.zeros((n, 10, 2))
    _abi.check(L.mfbem_internal_radial(q.ctypes.data, rmax, n, r.ctypes.data, tab.ctypes.data, tabf.ctypes.data,
                                       dr.ctypes.data))
    tab, tabf, dr = (v[..., 0] + 1j * v[..., 1] for v in (tab, tabf, dr))
    eps = 2.0 ** -53
    worst = np.zeros((3, 5))
    for i in range(n):
        e = _exact(mp, q, mp.mpf(float(r[i])))
        cu, ct = 1 / (4 * mp.pi * mp.mpc(q[2], q[3])), 1 / (4 * mp.pi)
        for j in range(5):
            x = complex(e[j] * (cu if j < 2 else ct))
            p = 1 if j < 2 else 2
            size = (r[i] ** -p + k2 ** p) * abs(complex(cu if j < 2 else ct))
            for w, v in enumerate((tab, tabf, dr)):
                worst[w, j] = max(worst[w, j], abs(v[i, j] - x) / size)
    print("error / eps: table", worst[0] / eps, "double-float", worst[1] / eps, "direct", worst[2] / eps)
    assert worst[0].max() <= 40 * eps, worst[0] / eps
    assert worst[1].max() <= 8 * 2.0 ** -47, worst[1]
    assert (worst[0] <= 2 * np.maximum(worst[2], 8 * eps)).all(), worst / eps
    # S1..S5 against the direct evaluation: just above |z| = 1 its E_6 = e^z -
    # sum z^k / k! (about 1/720, from six subtractions) enters with 60 / k^2 for
    # both wavenumbers, 60 x 3 eps x 2 of k^3, and E_5, E_4 with as much again
    s = np.abs(r[:, None] ** -3 + k2 ** 3) * abs(q[2] + 1j * q[3]) / (4 * np.pi)
    assert (np.abs(tab[:, 5:] - dr[:, 5:]) <= 2000 * eps * s).all(), (np.abs(tab[:, 5:] - dr[:, 5:]) / s).max() / eps


@pytest.mark.parametrize("side", [0.97, 1.03])
def test_both_sides_of_the_table_rule(oracle, side):
    """65536 intervals per frequency at most: the assembly just below (table)
    and above (direct evaluation), against the oracle."""
    d = M.cube_clamped_top_traction(1)
    m = M.viscoelastic(1.0, 0.25, 1.0, 0.0)
    # extent of the bounding box of the elements' balls (3 times the nodes' distance from their mean)
    X = d.nodes[d.conn]
    c = X.mean(1)
    R = np.sqrt(((X - c[:, None]) ** 2).sum(2)).max(1)[:, None]
    ext = np.linalg.norm((c + 3 * R).max(0) - (c - 3 * R).min(0))
    om = side * 65536 * 0.125 / ext * m["c_s"]
    R_ = BemRegion(d)
    A, b = R_.build_lse_harela(m, om)
    Ao, bo = oracle.Problem(d).assemble_harela(m, om)
    R_.close()
    # phases |k| r of up to 8000 radians are known to |k| r eps
    assert np.abs(A - Ao).max() <= 1e-11 * np.abs(Ao).max() * 10
    assert np.abs(b - bo).max() <= 1e-11 * max(1.0, np.abs(bo).max()) * 10
