"""Constitutive relations by integer powers (van Genuchten and Mualem of one
m) over their range, at its ends and beyond it, where the FP64 formulas take
over: the saturation and its derivative against extended precision (the FP64
formula of the oracle underflows, or rounds -m - 1 before a power of 1e60, at
the far ends), the residual and Jacobian against the oracle.

Tolerances: C = rho phi S V is S to a few roundings (each power and product
within 1 ulp on either side: 16 eps); dC/dP multiplies about ten of them, with
arguments rounded before each power (64 eps).  The residual and Jacobian take
the bars of the parity tests, 1e-12 and 1e-10 of the terms' magnitudes."""
import numpy as np
import pytest

import tdycore_gb300 as T
from tdycore_gb300 import workloads as W
from oracle import Oracle

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def handle(m, alpha, mm):
    T.options_clear()
    t = W.box_column(8, 8, 8, density=T.WATER_DENSITY_CONSTANT, bc_type=T.NEUMANN_BC)
    t.set_vangenuchten_values(m, alpha)
    t.set_mualem_values(mm)
    t.setup()
    return t


# m, and x = alpha Pc: the ordinary range; n up to 33 and m down to 1/300 (both
# sides of the limits); x far from 1, where x^n leaves the integer powers' range
@pytest.mark.parametrize("m_range,log_x", [((0.1, 0.9), (-8, 1)), ((0.9, 0.97), (-8, 0.5)),
                                           ((1 / 300, 0.02), (-12, 8)), ((0.5, 0.9), (-25, 25))])
def test_saturation_and_derivative(m_range, log_x):
    r = np.random.default_rng(5)
    n = 512
    m, alpha = r.uniform(*m_range, n), 10.0 ** r.uniform(-6, -3, n)
    x = 10.0 ** r.uniform(*log_x, n)
    U = 101325.0 - x / alpha
    U[:8] = 101325.0 + np.array([0.0, 1e-11, -1e-11, 1e-9, -1e-9, 1.0, -1.0, 5e4])
    t = handle(m, alpha, m)
    C, dC = t.transient_variable(U, with_derivative=True)
    L = np.longdouble
    mass = L(998.0) * L(0.115) * t.cell_volumes().astype(L)  # rho phi V
    Pc, ml = (101325.0 - U).astype(L), m.astype(L)
    xe = np.where(Pc > 0, ((101325.0 - U) * alpha).astype(L), 1)
    nl, S1 = (1.0 / (1.0 - m)).astype(L), L(1.0 - 0.115)
    w = 1 + xe ** nl
    Co = mass * np.where(Pc > 0, S1 * w ** (-ml) + L(0.115), 1)
    dCo = mass * np.where(Pc > 0, S1 * ml * nl * alpha.astype(L) * xe ** (nl - 1) * w ** (-ml - 1), 0)
    assert np.all(np.abs(C - Co) <= 16 * EPS * np.abs(Co))
    assert np.all(np.abs(dC - dCo) <= 64 * EPS * np.abs(dCo) + 1e-300)


@pytest.mark.parametrize("same_m", [True, False])
def test_residual_and_jacobian(same_m):
    r = np.random.default_rng(6)
    n = 512
    m, alpha = r.uniform(0.1, 0.9, n), 10.0 ** r.uniform(-5, -3, n)
    mm = m if same_m else r.uniform(0.1, 0.9, n)
    x = 10.0 ** r.uniform(-6, 0.5, n)  # both sides of the smoothing at Se = 0.99
    U = 101325.0 - x / alpha
    t = handle(m, alpha, mm)
    t.set_dtime(100.0)
    Uprev, Ut = U + r.normal(0, 10.0, n), r.normal(0, 5.0, n)
    t.presolve(Uprev)
    o = Oracle(t.setup_view())
    o.snes_presolve(Uprev, 100.0)
    for R, J, (Ro, Rm), (Jo, Jm) in (
            (*t.snes_function_jacobian(U), o.snes_function(U, with_mag=True), o.snes_jacobian(U, with_mag=True)),
            (*t.ifunction_ijacobian(0.0, U, Ut, 0.01), o.ts_ifunction(U, Ut, with_mag=True),
             o.ts_ijacobian(U, Ut, 0.01, with_mag=True))):
        assert np.all(np.abs(R - Ro) <= 1e-12 * Rm)
        assert np.all(np.abs(J - Jo) <= 1e-10 * Jm)


# wet to very dry: the plain formula of kr loses 7 digits at x = 100
@pytest.mark.parametrize("log_x", [(-1.5, 0), (0, 2), (2, 6)])
def test_relative_permeability(log_x):
    """kr of dry soil in extended precision, from the flux between two cells
    (accumulation suppressed by a huge time step).  Tolerance 1e-12: kr itself
    is within 1e-13 of 300-bit arithmetic, the flux adds a few roundings."""
    r = np.random.default_rng(9)
    n = 256
    T.options_clear()
    t = T.create_richards_mpfao()
    xy, quads = W.structured_surface(1, 1, 1.0, 1.0)
    blocks = []
    for b in range(n):
        s = xy.copy()
        s[:, 0] += 2.0 * b
        blocks.append((s, quads, W.layered_z(4, 2, 1.0)))
    t.set_extruded_meshes(blocks)
    t.set_from_options()
    m, alpha = np.repeat(r.uniform(0.2, 0.6, n), 2), np.repeat(10.0 ** r.uniform(-5, -3, n), 2)
    t.set_vangenuchten_values(m, alpha)
    t.set_mualem_values(m)
    t.set_constant_isotropic_permeability(1e-12)
    t.set_boundary_pressure_type_function(lambda x, y, z: np.full(np.shape(x), T.NEUMANN_BC))
    t.set_water_density_type(T.WATER_DENSITY_CONSTANT)
    t.setup()
    x = 10.0 ** r.uniform(*log_x, 2 * n)
    x[1::2] = 3.0 * x[::2]
    U = 101325.0 - x / alpha
    t.set_dtime(1e60)
    t.presolve(U)
    R = t.snes_function(U)[::2]
    v = t.setup_view()
    L = np.longdouble
    # every vertex of a block has one row, its face's up cell first: sum the four
    q = np.zeros(n, dtype=L)
    for k in range(v["nverts"]):
        r0, r1, c0 = v["v_row_off"][k], v["v_row_off"][k + 1], v["v_col_off"][k]
        if r1 > r0:
            Tr = v["trans"][v["v_trans_off"][k]:v["v_trans_off"][k] + 2].astype(L)
            cols = v["col_ext"][c0:c0 + 2]
            q[cols[0] // 2] += Tr @ U[cols].astype(L) + L(998.0) * L(v["gravdis"][v["row_face"][r0]])
    up = np.where(q < 0, np.arange(n) * 2, np.arange(n) * 2 + 1)
    ml = m[up].astype(L)
    w = 1 + ((101325.0 - U[up]) * alpha[up]).astype(L) ** (1.0 / (1.0 - m[up])).astype(L)
    kr = w ** (-ml / 2) * np.expm1(ml * np.log1p(-1 / w)) ** 2
    flux = -q * L(998.0) * kr / L(9.94e-4)
    dry = w ** (-ml) < 0.99
    assert dry.sum() > n // 2
    assert np.all(np.abs(R - flux)[dry] <= 1e-12 * np.abs(flux)[dry])
