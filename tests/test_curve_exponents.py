"""van Genuchten parameters m above 1, for which n = 1 / (1 - m) is negative:
outside the model's sense but accepted, so every call follows the formula.
Saturation and its derivative against extended precision, residual and
Jacobian (with the Mualem m of the saturation and another one) against the
oracle.

Tolerances: as in test_curve_powers.py (16 and 64 eps; a power's rounded base
contributes up to m = 4 roundings); the parity tests' bars, 1e-12 and 1e-10,
with x = alpha Pc >= 1, where kr does not cancel."""
import numpy as np
import pytest

import tdycore_gb300 as T
from tdycore_gb300 import workloads as W
from oracle import Oracle

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52
NC = 216


def handle(m, alpha, mm):
    T.options_clear()
    t = W.box_column(6, 6, 6, density=T.WATER_DENSITY_CONSTANT, bc_type=T.NEUMANN_BC)
    t.set_vangenuchten_values(m, alpha)
    t.set_mualem_values(mm)
    t.setup()
    return t


@pytest.mark.parametrize("m_range", [(1.05, 1.5), (1.5, 4.0)])
def test_saturation(m_range):
    r = np.random.default_rng(7)
    m, alpha = r.uniform(*m_range, NC), 10.0 ** r.uniform(-6, -3, NC)
    U = 101325.0 - 10.0 ** r.uniform(-3, 3, NC) / alpha
    C, dC = handle(m, alpha, m).transient_variable(U, with_derivative=True)
    L = np.longdouble
    ml, nl = m.astype(L), (1.0 / (1.0 - m)).astype(L)
    x = ((101325.0 - U) * alpha).astype(L)
    w, S1 = 1 + x ** nl, L(1.0 - 0.115)
    mass = L(998.0) * L(0.115) * handle(m, alpha, m).cell_volumes().astype(L)
    Co = mass * (S1 * w ** (-ml) + L(0.115))
    dCo = mass * S1 * ml * nl * alpha.astype(L) * x ** (nl - 1) * w ** (-ml - 1)
    assert np.all(np.abs(C - Co) <= 16 * EPS * np.abs(Co))
    assert np.all(np.abs(dC - dCo) <= 64 * EPS * np.abs(dCo) + 1e-300)


@pytest.mark.parametrize("same_m", [True, False])
def test_residual_and_jacobian(same_m):
    r = np.random.default_rng(8)
    m, alpha = r.uniform(1.5, 3.0, NC), 10.0 ** r.uniform(-5, -3, NC)
    mm = m if same_m else r.uniform(0.2, 0.8, NC)
    U = 101325.0 - 10.0 ** r.uniform(0, 1.5, NC) / alpha
    t = handle(m, alpha, mm)
    t.set_dtime(100.0)
    Uprev, Ut = U + r.normal(0, 10.0, NC), r.normal(0, 5.0, NC)
    t.presolve(Uprev)
    o = Oracle(t.setup_view())
    o.snes_presolve(Uprev, 100.0)
    for R, J, (Ro, Rm), (Jo, Jm) in (
            (*t.snes_function_jacobian(U), o.snes_function(U, with_mag=True), o.snes_jacobian(U, with_mag=True)),
            (*t.ifunction_ijacobian(0.0, U, Ut, 0.01), o.ts_ifunction(U, Ut, with_mag=True),
             o.ts_ijacobian(U, Ut, 0.01, with_mag=True))):
        assert np.all(np.abs(R - Ro) <= 1e-12 * Rm)
        assert np.all(np.abs(J - Jo) <= 1e-10 * Jm)
