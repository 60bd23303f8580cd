"""Jacobian of interior hexahedral vertices in double-float against the same
with FP64 products (1e-10 of the oracle's magnitudes of the terms, the parity
tests' bar; the oracle's own kr loses its digits in the driest cells), and the
residual against the oracle, where the paths part:
saturated cells only (no upwind-derivative terms), mixed, cells so dry that
the products of a vertex do not fit one scale beside wet ones, dry cells only,
on jittered and orthogonal meshes (whose Trans has zeros and rounding noise),
with constant and pressure-dependent density."""
import numpy as np
import pytest

import tdycore_gb300 as T
from tdycore_gb300 import workloads as W
from oracle import Oracle

pytestmark = pytest.mark.gpu


def suction(kind, n, rng):
    if kind == "saturated":
        return -rng.uniform(1e3, 1e5, n)
    if kind == "mixed":
        return rng.normal(0.0, 2e4, n)
    if kind == "dry_beside_wet":  # kr down to 1e-60 beside 1
        return np.where(rng.random(n) < 0.5, 10.0 ** rng.uniform(5, 9, n), -1e4)
    return 10.0 ** rng.uniform(4, 6, n)


@pytest.mark.parametrize("density", [T.WATER_DENSITY_CONSTANT, T.WATER_DENSITY_EXPONENTIAL])
@pytest.mark.parametrize("jitter", [0.1, 0.0])
@pytest.mark.parametrize("kind", ["saturated", "mixed", "dry_beside_wet", "dry"])
def test_parity(kind, jitter, density):
    got = {}
    for arithmetic in ("FP64", "DOUBLE_FLOAT"):
        T.options_clear()
        T.options_insert("-tdy_jacobian_arithmetic " + arithmetic)
        t, U, _ = W.spe10_like(9, 7, 6, lx=54.0, ly=21.0, lz=3.6, jitter=jitter, seed_offset=3)
        T.options_clear()
        t.set_water_density_type(density)
        t.setup()
        U = 101325.0 - suction(kind, U.size, np.random.default_rng(8))
        t.set_dtime(900.0)
        t.presolve(U)
        got[arithmetic] = t.snes_function_jacobian(U)
    R, J = got["DOUBLE_FLOAT"]
    o = Oracle(t.setup_view())
    o.snes_presolve(U, 900.0)
    (Ro, Rm), (_, Jm) = o.snes_function(U, with_mag=True), o.snes_jacobian(U, with_mag=True)
    assert np.array_equal(R, got["FP64"][0])
    assert np.all(np.abs(R - Ro) <= 1e-12 * Rm)
    assert np.all(np.abs(J - got["FP64"][1]) <= 1e-10 * Jm)
