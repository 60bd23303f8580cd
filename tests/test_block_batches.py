"""Batches of uneven instances on the block schedule, whose launch classes
share one amount of shared memory: every batch size of a server's cohort has
to launch, and give the tile schedule's bits."""
import numpy as np
import pytest

import tdycore_gb300 as T
from tdycore_gb300.workloads import layered_z, structured_surface

pytestmark = pytest.mark.gpu

BATCHES = [
    [(2, 3, 81), (3, 4, 53), (1, 1, 94), (6, 5, 18)],
    [(2, 8, 15), (1, 7, 60), (5, 3, 77), (2, 8, 50), (8, 2, 27), (2, 4, 49), (1, 5, 36)],
    [(n, 1, 97) for n in range(1, 9)],
    [(n, n, 12) for n in range(1, 21)],
    [(40, 40, 4), (3, 3, 100), (1, 1, 100), (20, 20, 10), (30, 30, 3), (8, 8, 100)],
]


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("shapes", BATCHES, ids=range(len(BATCHES)))
def test_batches_launch(shapes, fp32):
    import torch

    T.options_clear()
    T.options_insert("-tdy_mpfao_setup_on_device")
    t = T.create_richards_mpfao()
    blocks, U, x0 = [], [], 0.0
    rng = np.random.default_rng(3)
    for nx, ny, nz in shapes:
        xy, quads = structured_surface(nx, ny, float(nx), float(ny))
        xy[:, 0] += x0
        x0 += nx + 1.0
        blocks.append((xy, quads, layered_z(xy.shape[0], nz, 0.3 * nz)))
        zc = np.repeat((np.arange(nz) + 0.5) * 0.3, nx * ny)
        U.append(101325.0 + 9787.0 * (0.2 * nz - zc) + rng.normal(0, 50.0, zc.size))
    t.set_extruded_meshes(blocks)
    t.set_from_options()
    T.options_clear()
    t.set_constant_isotropic_permeability(1e-12)
    t.set_boundary_pressure_type_function(lambda x, y, z: np.full(np.shape(x), T.NEUMANN_BC))
    t.setup()
    U = np.concatenate(U)
    got = {}
    for sched in ("tile", "block"):
        d = torch.tensor(U, dtype=torch.float64, device="cuda")
        _, its, _ = t.backward_euler_step_device(d, 3600.0, max_it=2, fp32=fp32, schedule=sched, linear_max_it=40)
        got[sched] = (d.cpu().numpy(), its)
    assert np.array_equal(got["block"][0], got["tile"][0])
    assert np.array_equal(got["block"][1], got["tile"][1])
