"""Block schedule of the inner solve against the tile schedule, at the sizes
where its splits change: cells below, at and above 256 (a CTA's threads) and
4096 (a reduction chunk), instances whose vectors, or whose z, no longer fit
shared memory, and the largest one of its 16-bit column indices (a larger
instance stays on the tile schedule); a single saturated cell without storage
has a singular system, which both give up at once.  The schedules perform the same
operations in the same order: the same bits are required."""
import numpy as np
import pytest

import tdycore_gb300 as T
from tdycore_gb300.workloads import layered_z, structured_surface

pytestmark = pytest.mark.gpu

SHAPES = [[(1, 1, 1)], [(1, 1, 7)], [(16, 16, 1)], [(257, 1, 1)], [(8, 8, 64)], [(17, 15, 17)], [(3, 3, 9), (8, 8, 100), (1, 2, 31)],
          [(40, 40, 10)], [(50, 50, 16)], [(64, 64, 16)], [(64, 64, 17), (5, 4, 3)]]


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("shapes", SHAPES, ids=lambda s: "+".join("x".join(map(str, t)) for t in s))
def test_block_equals_tile(shapes, fp32):
    import torch

    T.options_clear()
    T.options_insert("-tdy_mpfao_setup_on_device")
    t = T.create_richards_mpfao()
    blocks, U, x0 = [], [], 0.0
    rng = np.random.default_rng(11)
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
    src = np.zeros(U.size)
    src[::3] = 1e-5
    t.set_source_sink_values(src)
    got = {}
    for sched in ("tile", "block"):
        d = torch.tensor(U, dtype=torch.float64, device="cuda")
        st, its, _ = t.backward_euler_step_device(d, 3600.0, max_it=2, fp32=fp32, schedule=sched, linear_max_it=40)
        got[sched] = (d.cpu().numpy(), its, st)
    small = sum(nx * ny * nz <= 65536 for nx, ny, nz in shapes)
    assert got["block"][2]["block_instances"] == small and got["tile"][2]["block_instances"] == 0
    assert np.array_equal(got["block"][0], got["tile"][0])
    assert np.array_equal(got["block"][1], got["tile"][1])
    assert got["block"][2]["linear_iterations"] == got["tile"][2]["linear_iterations"]
