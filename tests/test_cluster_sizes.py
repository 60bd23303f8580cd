"""Clusters of the inner solve's preconditioner at the sizes where a warp's
split of the rows changes (a row per lane up to 32, two up to 64, the largest
cluster) beside cells on their diagonal: with every coupling strong a column
of up to 64 cells is one cluster, its factors are the whole Jacobian's and
BiCGStab ends after one iteration at every Newton iteration; the step equals
the line-preconditioned one (both are within the Newton tolerance of the
solution; 1e-9 as in the test of the 54-cell column)."""
import numpy as np
import pytest

import tdycore_gb300 as T
from tdycore_gb300.workloads import box_column

pytestmark = pytest.mark.gpu


def column(nz):
    T.options_clear()
    t = box_column(1, 1, nz, pfunc=lambda x, y, z: 99000.0)
    t.set_boundary_pressure_type_function(
        lambda x, y, z: np.where(np.asarray(z) > 1 - 1e-9, T.DIRICHLET_BC, T.NEUMANN_BC))
    t.setup()
    zc = t.cell_centroids()[:, 2]
    return t, 101325.0 + 998.0 * 9.8068 * (0.5 - zc) + np.random.default_rng(nz).normal(0, 300, nz)


@pytest.mark.parametrize("nz", [1, 2, 31, 32, 33, 63, 64, 65])
def test_column_is_one_cluster(nz):
    import torch

    U, st = {}, {}
    for precond in ("clusters", "lines"):
        t, Un = column(nz)
        d = torch.tensor(Un, dtype=torch.float64, device="cuda")
        st[precond], its, _ = t.backward_euler_step_device(d, 3600.0, rtol=1e-8, fp32=False, precond=precond,
                                                           cluster_threshold=1e-300)
        U[precond] = d.cpu().numpy()
        assert st[precond]["converged"] == 1, st
    c = st["clusters"]
    one = 2 <= nz <= 64
    assert c["precond_used"] == T.PRECOND_CLUSTERS and c["clusters"] == one, c
    assert c["cluster_cells"] == (nz if one else 0) and c["cluster_cells_diagonal"] == (nz if nz > 64 else 0), c
    if nz <= 64:
        assert c["linear_iterations"] == c["newton_iterations"] >= 1, c
    assert np.max(np.abs(U["clusters"] - U["lines"]) / np.abs(U["lines"])) < 1e-9


@pytest.mark.parametrize("triangles,layers", [(60, 3), (500, 9), (2000, 20)])
@pytest.mark.parametrize("tau", [0.02, 0.05, 0.3, 1e300])
def test_clusters_are_the_connected_components(triangles, layers, tau):
    """Number and cells of the clusters of the first inner solve against the
    connected components of the strong couplings of the Jacobian there."""
    import torch
    from scipy.sparse import coo_matrix
    from scipy.sparse.csgraph import connected_components

    from tdycore_gb300.workloads import infiltration_prisms

    T.options_clear()
    t, U, top, src, _ = infiltration_prisms(triangles, layers)
    t.setup()
    t.set_source_sink_values(src, cells=top)
    n = t.ncells
    d = torch.tensor(U, dtype=torch.float64, device="cuda")
    st, _, _ = t.backward_euler_step_device(d, 600.0, max_it=1, precond="clusters", cluster_threshold=tau)
    t.set_dtime(600.0)
    t.presolve(U)
    J = np.abs(t.snes_jacobian(U))
    row, col = np.repeat(np.arange(n), np.diff(t.rowptr)), t.colidx
    diag = np.zeros(n)
    diag[row[row == col]] = J[row == col]
    strong = (row != col) & (J > 0) & (J >= tau * np.sqrt(diag[row] * diag[col]))
    label = connected_components(coo_matrix((strong[strong], (row[strong], col[strong])), shape=(n, n)), directed=False)[1]
    size = np.bincount(label)
    used = (size >= 2) & (size <= 64)
    assert st["precond_used"] == T.PRECOND_CLUSTERS
    assert (st["clusters"], st["cluster_cells"], st["cluster_cells_diagonal"]) == (
        used.sum(), size[used].sum(), size[size > 64].sum())
