"""Residual and Jacobian at the vertices and cells outside the regular
hexahedral interior, against the oracle at the parity tests' bars (1e-12 and
1e-10 of the terms' magnitudes): few and many of them (their kernels' launch
and lane choices differ), small and large vertices, one-cell-wide columns, and
columns of one to many layers, with both Jacobian arithmetics."""
import numpy as np
import pytest

import tdycore_gb300 as T
from tdycore_gb300 import workloads as W
from oracle import Oracle

pytestmark = pytest.mark.gpu


def prisms(npts, nlayers):
    t, U, _ = W.wedge_extruded(npts=npts, nlayers=nlayers, seed_offset=2)
    return t, U


def columns(ninst):
    t, U, _ = W.batched_columns(ninst, seed_offset=4)
    return t, U


def box(nx, ny, nz, bc):
    t = W.box_column(nx, ny, nz, density=T.WATER_DENSITY_CONSTANT, bc_type=bc, pfunc=lambda x, y, z: 100000.0)
    return t, 101000.0 + np.random.default_rng(1).normal(0, 4e3, nx * ny * nz)


CASES = {"prisms_few": lambda: prisms(12, 2), "prisms_many": lambda: prisms(1200, 20), "columns": lambda: columns(6),
         "line": lambda: box(1, 1, 9, T.DIRICHLET_BC), "sheet": lambda: box(33, 1, 3, T.SEEPAGE_BC),
         "slab": lambda: box(7, 9, 2, T.NEUMANN_BC), "row": lambda: box(130, 2, 1, T.DIRICHLET_BC)}


@pytest.mark.parametrize("arithmetic", ["DOUBLE_FLOAT", "FP64"])
@pytest.mark.parametrize("name", list(CASES))
def test_parity(name, arithmetic):
    T.options_clear()
    if arithmetic == "FP64":
        T.options_insert("-tdy_jacobian_arithmetic FP64")
    t, U = CASES[name]()
    T.options_clear()
    t.setup()
    t.set_dtime(600.0)
    U = U + np.random.default_rng(2).normal(0, 500.0, U.size)
    Uprev = U + np.random.default_rng(3).normal(0, 50.0, U.size)
    t.presolve(Uprev)
    R, J = t.snes_function_jacobian(U)
    o = Oracle(t.setup_view())
    o.snes_presolve(Uprev, 600.0)
    (Ro, Rm), (Jo, Jm) = o.snes_function(U, with_mag=True), o.snes_jacobian(U, with_mag=True)
    assert np.all(np.abs(R - Ro) <= 1e-12 * Rm)
    assert np.all(np.abs(J - Jo) <= 1e-10 * Jm)
    assert np.array_equal(t.snes_function(U), R) and np.array_equal(t.snes_jacobian(U), J)
