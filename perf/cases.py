"""The work users of this framework have it do, as timed cases.

A case names a mesh with its sizes, the call made on it and the options used
in earnest:

* mesh ``box``    -- the unit cube of the reference's regression problems;
  ``hex``    -- jittered hexahedra with a correlated random permeability, the
  SPE10 model-2 extents (any nx x ny x nz); ``prism`` -- extruded Delaunay
  triangles with full-tensor permeability, dry soil; ``batch`` -- independent
  hexahedral columns in one handle (what the batching server builds).
* call ``fj`` (SNES residual and Jacobian, device buffers), ``f`` (residual
  only: line-search trials), ``ij`` (TS residual and Jacobian, device
  buffers), ``host`` (residual and Jacobian into page-locked host buffers),
  ``host_split`` (residual, then Jacobian, pageable host arrays: PETSc's two
  callbacks), ``newton`` (one backward-Euler step of the device Newton).
* ``density`` constant or exponential; ``arithmetic`` of the Jacobian products
  double_float or fp64; for Newton ``fp32`` inner solves or not, and ``precond``.
"""
from __future__ import annotations

import math

import numpy as np
import torch

GRAVITY, PREF, RHO0, VISCOSITY = 9.8068, 101325.0, 998.0, 9.94e-4
LX, LY, LZ = 365.76, 670.56, 51.816  # extents of the 60 x 220 x 85 grid


def _case(name, mesh, call, **kw):
    c = {"name": name, "mesh": mesh, "call": call, "density": "constant", "arithmetic": "double_float", "nx": 0,
         "ny": 0, "nz": 0, "instances": 0, "triangles": 0, "layers": 0, "fp32": True, "precond": "lines"}
    c.update(kw)
    return c


def listed():
    return [
        # the regression problems: PETSc's two callbacks on host arrays, once per Newton iteration
        _case("regression_host_split", "box", "host_split", density="exponential", nx=5, ny=5, nz=5),
        # a small box in HBM: launches and latency
        _case("box_fj", "hex", "fj", nx=10, ny=10, nz=10),
        # the same box advanced one step by the device Newton in plain FP64
        _case("box_newton_fp64", "box", "newton", nx=10, ny=10, nz=10, fp32=False),
        # the headline grid: one Newton iteration's residual and Jacobian
        _case("grid_fj", "hex", "fj", nx=60, ny=220, nz=85),
        # line-search trials on a quarter of that grid
        _case("grid_f", "hex", "f", nx=60, ny=110, nz=40),
        # an application that keeps R and J in its own page-locked host memory
        _case("grid_host", "hex", "host", nx=60, ny=110, nz=40),
        # PETSc TS form, compressible water, strict FP64 Jacobian, odd sizes
        _case("grid_ij_fp64", "hex", "ij", nx=31, ny=57, nz=23, density="exponential", arithmetic="fp64"),
        # watershed prisms in dry soil (every cell unsaturated)
        _case("prism_fj", "prism", "fj", triangles=5000, layers=40),
        # the same kind of mesh advanced one step, mixed precision, cluster preconditioner
        _case("prism_newton", "prism", "newton", triangles=1000, layers=20, precond="clusters"),
        # a batch of columns: one Newton iteration's residual and Jacobian
        _case("batch_fj", "batch", "fj", instances=512),
        # a server's cohorts: one step of every request, mixed precision and FP64
        _case("batch_newton", "batch", "newton", instances=192),
        _case("batch_newton_fp64", "batch", "newton", instances=32, fp32=False),
    ]


def _drawn(mesh, call, **kw):
    c = _case("", mesh, call, **kw)
    del c["name"]
    return c


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ones' ranges, sizes spread over their logarithm."""
    kind = rng.choice(["hex", "hex", "prism", "batch", "batch_newton", "box", "prism_newton"])
    density = rng.choice(["constant", "constant", "exponential"])
    arithmetic = rng.choice(["double_float", "double_float", "fp64"])
    if kind == "hex":
        call = rng.choice(["fj", "fj", "f", "ij", "host", "host_split"])
        most = 60 * 220 * 85 if call in ("fj", "f", "ij") else 264_000
        cells = _log_uniform(rng, 200, most)
        nx = max(1, round((cells ** (1 / 3)) * rng.uniform(0.5, 1.2)))
        ny = max(1, round((cells / nx) ** 0.5 * rng.uniform(0.7, 1.6)))
        nz = max(1, cells // (nx * ny))
        return _drawn("hex", call, nx=nx, ny=ny, nz=nz, density=density, arithmetic=arithmetic)
    if kind == "box":
        call = rng.choice(["host_split", "newton"])
        n = [rng.randint(1, 11) for _ in range(2)] + [rng.randint(3, 15)]
        return _drawn("box", call, nx=n[0], ny=n[1], nz=n[2], fp32=rng.random() < 0.5,
                     density=density if call == "host_split" else "constant")
    if kind == "prism":
        layers = rng.randint(3, 40)
        return _drawn("prism", rng.choice(["fj", "f", "ij"]), layers=layers, density=density,
                     arithmetic=arithmetic, triangles=_log_uniform(rng, 40, 200_000 // layers))
    if kind == "prism_newton":
        layers = rng.randint(4, 20)
        return _drawn("prism", "newton", layers=layers, triangles=_log_uniform(rng, 60, 1000), precond="clusters",
                     fp32=rng.random() < 0.7)
    if kind == "batch":
        return _drawn("batch", "fj", instances=_log_uniform(rng, 2, 512), arithmetic=arithmetic)
    fp32 = rng.random() < 0.6
    return _drawn("batch", "newton", instances=_log_uniform(rng, 2, 192 if fp32 else 32), fp32=fp32)


# ---------------------------------------------------------------------------
# inputs


def _rng(seed, sub):
    return np.random.default_rng([int(seed), sub])


def _smooth(g, sigma=5.0):
    """Gaussian smoothing (periodic, by FFT), then zero mean and unit deviation."""
    f = np.fft.rfftn(g)
    for axis, n in enumerate(g.shape):
        k = np.fft.rfftfreq(n) if axis == g.ndim - 1 else np.fft.fftfreq(n)
        shape = [1] * g.ndim
        shape[axis] = -1
        f *= np.exp(-2.0 * (math.pi * sigma * k) ** 2).reshape(shape)
    g = np.fft.irfftn(f, g.shape, axes=tuple(range(g.ndim)))
    s = g.std()
    return (g - g.mean()) / s if s > 0 else g * 0.0


def _iso(k, kz=1.0):
    K = np.zeros((k.size, 9))
    K[:, 0] = K[:, 4] = k
    K[:, 8] = kz * k
    return K


def _column_shapes(ninst):
    """The batch's instance sizes (a property of the case, not of the seed)."""
    r = _rng(77, 1)
    return r.integers(1, 9, ninst), r.integers(1, 9, ninst), r.integers(10, 101, ninst), r.uniform(0.05, 0.5, ninst)


def _prism_surface(triangles):
    from tdycore_gb300.workloads import delaunay_surface

    return delaunay_surface(max(triangles // 2, 3), 1000.0, 1000.0, _rng(78, 2))


def _problem(case, seed):
    """Meshes, materials, boundary data and states as plain arrays."""
    from tdycore_gb300.workloads import layered_z, random_spd, structured_surface

    mesh, p = case["mesh"], {"source": None, "dt": 1800.0}
    r = _rng(seed, 0)
    if mesh == "batch":
        nx, ny, nz, dz = _column_shapes(case["instances"])
        ncell = (nx * ny * nz).astype(np.int64)
        blocks, x0, xs, U = [], 0.0, [], []
        for b in range(nx.size):
            xy, quads = structured_surface(int(nx[b]), int(ny[b]), float(nx[b]), float(ny[b]))
            xy[:, 0] += x0
            xs.append(x0)
            x0 += nx[b] + 1.0
            depth = dz[b] * nz[b]
            blocks.append((xy, quads, layered_z(xy.shape[0], int(nz[b]), depth)))
            zc = (np.arange(nz[b]) + 0.5) * dz[b]
            U.append(np.repeat(PREF + RHO0 * GRAVITY * (0.6 * depth - zc), nx[b] * ny[b]))
        one = lambda v: np.repeat(v, ncell)  # noqa: E731
        n = nx.size
        depth = dz * nz
        p.update(K=_iso(one(10.0 ** r.normal(-12.0, 1.0, n))), poro=one(r.uniform(0.05, 0.35, n)), sr=0.15,
                 m=one(r.uniform(0.2, 0.6, n)), alpha=one(10.0 ** r.uniform(-5.0, -3.0, n)), dt=3600.0,
                 top=PREF + RHO0 * GRAVITY * (0.6 * depth - depth) + 2000.0, blocks=blocks, xs=np.array(xs))
        p["U"] = np.concatenate(U) + r.normal(0.0, 10.0, int(ncell.sum()))
        p["Uprev"] = p["U"] + r.normal(0.0, 10.0, p["U"].size)
    elif mesh == "prism":
        xy, tris = _prism_surface(case["triangles"])
        nl, nt = case["layers"], tris.shape[0]
        levels = np.concatenate([[0.0], np.cumsum(r.uniform(0.1, 2.0, nl))])
        n = nl * nt
        K = random_spd(n, r, rotation="vertical").reshape(n, 9)
        a, b, c = xy[tris[:, 0]], xy[tris[:, 1]], xy[tris[:, 2]]
        area = 0.5 * np.abs((b[:, 0] - a[:, 0]) * (c[:, 1] - a[:, 1]) - (b[:, 1] - a[:, 1]) * (c[:, 0] - a[:, 0]))
        source = np.zeros(n)
        source[(nl - 1) * nt:] = RHO0 * 1e-7 * area
        p.update(blocks=[(xy, tris, np.repeat(levels[:, None], xy.shape[0], axis=1))], K=K, sr=0.15,
                 poro=r.uniform(0.05, 0.35, n), m=np.full(n, 0.5), alpha=np.full(n, 1e-4), source=source, top=None,
                 dt=20.0, U=np.full(n, PREF - 2e4))
        p["Uprev"] = p["U"]
        if case["call"] != "newton":  # a state inside a Newton iteration
            p["U"] = p["U"] + r.normal(0.0, 2e3, n)
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        n = nx * ny * nz
        if mesh == "box":
            xy, quads = structured_surface(nx, ny, 1.0, 1.0)
            blocks = [(xy, quads, layered_z(xy.shape[0], nz, 1.0))]
            zc = np.repeat((np.arange(nz) + 0.5) / nz, nx * ny)
            p.update(blocks=blocks, alpha=np.full(n, 1e-4), box=True)
            if case["call"] == "newton":  # infiltration: the start 60 kPa below hydrostatic
                p.update(K=_iso(np.full(n, 1e-11)), poro=np.full(n, 0.25), sr=0.15, m=np.full(n, 0.3), top=np.array([PREF]))
                p["U"] = PREF + RHO0 * GRAVITY * (1.0 - zc) - 6e4 + r.normal(0.0, 10.0, n)
            else:  # every boundary face at its cell's pressure
                p.update(K=_iso(np.full(n, 1e-10)), poro=np.full(n, 0.115), sr=0.115, m=np.full(n, 0.8), top="cell")
                p["U"] = PREF + RHO0 * GRAVITY * (0.5 - zc) + r.normal(0.0, 3e3, n)
        else:
            lx, ly, lz = LX * nx / 60, LY * ny / 220, LZ * nz / 85
            xy, quads = structured_surface(nx, ny, lx, ly, 0.10, r)
            z = layered_z(xy.shape[0], nz, lz, 0.10, r)
            k = 10.0 ** (-13.0 + 1.5 * _smooth(r.standard_normal((nz, ny, nx))).ravel())
            p.update(blocks=[(xy, quads, z)], K=_iso(k, 0.1), poro=r.uniform(0.05, 0.35, n), sr=0.15,
                     m=r.uniform(0.2, 0.6, n), alpha=10.0 ** r.uniform(-5.0, -3.0, n), top=np.array([PREF]))
            zl = z.reshape(nz + 1, ny + 1, nx + 1)
            zc = 0.25 * (zl[:, :-1, :-1] + zl[:, :-1, 1:] + zl[:, 1:, :-1] + zl[:, 1:, 1:])
            zc = (0.5 * (zc[:-1] + zc[1:])).ravel()
            p["U"] = PREF + RHO0 * GRAVITY * (lz - zc) + r.normal(0.0, 5e3, n)
        p["Uprev"] = p["U"] + r.normal(0.0, 500.0, n)
    p["Ut"] = r.normal(0.0, 5.0, p["U"].size)
    p["shift"] = 1.0 / p["dt"]
    return p


def _handle(case, p):
    """The framework's handle on that problem, set up."""
    import tdycore_gb300 as T

    T.options_clear()
    T.options_insert("-tdy_mpfao_setup_on_device")
    if case["arithmetic"] == "fp64":
        T.options_insert("-tdy_jacobian_arithmetic FP64")
    t = T.create_richards_mpfao()
    blocks = p["blocks"]
    if p.get("box"):
        t.set_box_mesh(case["nx"], case["ny"], case["nz"])
    elif len(blocks) == 1 and case["mesh"] != "batch":
        t.set_extruded_mesh(*blocks[0])
    else:
        t.set_extruded_meshes(blocks)
    t.set_from_options()
    T.options_clear()
    t.set_permeability_values(p["K"])
    t.set_porosity_values(p["poro"])
    t.set_vangenuchten_values(p["m"], p["alpha"])
    t.set_mualem_values(p["m"])
    t.set_constant_residual_saturation(p["sr"])
    t.set_water_density_type(T.WATER_DENSITY_EXPONENTIAL if case["density"] == "exponential" else T.WATER_DENSITY_CONSTANT)
    if p["source"] is not None:
        t.set_source_sink_values(p["source"])
    top = p["top"]
    if top is None:
        t.set_boundary_pressure_type_function(lambda x, y, z: np.full(np.shape(x), T.NEUMANN_BC))
    elif not isinstance(top, str):
        ztop = np.array([b[2].max() for b in blocks])
        xs = p.get("xs", np.zeros(1))

        def block_of(x):
            return np.clip(np.searchsorted(xs - 0.5, np.asarray(x), side="right") - 1, 0, xs.size - 1)

        t.set_boundary_pressure_type_function(
            lambda x, y, z: np.where(np.asarray(z) > ztop[block_of(x)] - 1e-7, T.DIRICHLET_BC, T.NEUMANN_BC))
        t.set_boundary_pressure_function(lambda x, y, z: top[block_of(x)])
    t.setup()
    return t


class _State:
    pass


_streams = []


def _stream():
    """The program's compute stream: every handle's work goes to it."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def prepare(case, seed):
    p = _problem(case, seed)
    s = _State()
    s.case, s.dt, s.shift = case, p["dt"], p["shift"]
    s.t = _handle(case, p)
    s.t.set_dtime(p["dt"])
    s.t.presolve(p["Uprev"])
    call = case["call"]
    if call in ("host", "host_split"):
        if call == "host":
            pinned = lambda n: torch.empty(n, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()  # noqa: E731
            s.U, s.R, s.J = pinned(s.t.ncells), pinned(s.t.ncells), pinned(s.t.nnz)
            s.U[:] = p["U"]
        else:
            s.U = np.ascontiguousarray(p["U"])
        return s
    dev = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    s.stream = _stream()
    s.U0 = dev(p["U"])
    s.U = torch.empty_like(s.U0)
    if call != "newton":
        s.R = torch.empty_like(s.U0)
        s.J = torch.empty(s.t.nnz, dtype=torch.float64, device="cuda") if call != "f" else None
        s.Ut = dev(p["Ut"]) if call == "ij" else None
    torch.cuda.synchronize()
    return s


def run(s):
    call, t = s.case["call"], s.t
    if call == "host_split":
        return {"R": t.snes_function(s.U), "J": t.snes_jacobian(s.U)}
    if call == "host":
        R, J = t.snes_function_jacobian(s.U, s.R, s.J)
        return {"R": R, "J": J}
    st = s.stream.cuda_stream
    if call == "newton":
        with torch.cuda.stream(s.stream):
            s.U.copy_(s.U0)
        _, its, _ = t.backward_euler_step_device(s.U, s.dt, fp32=s.case["fp32"], precond=s.case["precond"], stream=st)
        return {"U": s.U, "iterations": its, "status": t.instance_status()}
    if call == "ij":
        t.ifunction_ijacobian_device(0.0, s.U0, s.Ut, s.shift, s.R, s.J, stream=st)
        return {"R": s.R, "J": s.J}
    t.snes_function_jacobian_device(s.U0, s.R, s.J, stream=st)
    return {"R": s.R} if s.J is None else {"R": s.R, "J": s.J}


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _counts(nint2, nedge2, npoly2, nl, top):
    """(sum of rows x columns, of rows, of rows x internal columns, of squared
    cells) over a block's vertices: per surface vertex nint2 polygons and
    nedge2 inner edges; a Dirichlet top adds a row and a column per top face."""
    s, e = nint2.astype(np.float64), nedge2.astype(np.float64)
    mid, rows_mid = 2 * s, 2 * e + s
    end = s + e * 0
    d = s if top else 0 * s
    rc = (nl - 1) * (rows_mid * mid).sum() + (e * end).sum() + ((e + d) * (end + d)).sum()
    r = (nl - 1) * rows_mid.sum() + e.sum() + (e + d).sum()
    rn = (nl - 1) * (rows_mid * mid).sum() + (e * end).sum() + ((e + d) * end).sum()
    return rc, r, rn


def _surface_counts(nv2, cells):
    """Polygons and inner edges at each surface vertex; pairs of polygons sharing a vertex."""
    n = cells.shape[1]
    nint = np.bincount(cells.ravel(), minlength=nv2)
    a, b = cells.ravel(), np.roll(cells, -1, axis=1).ravel()
    key, cnt = np.unique(np.minimum(a, b).astype(np.int64) * nv2 + np.maximum(a, b), return_counts=True)
    key = key[cnt == 2]
    nedge = np.bincount(np.concatenate([key // nv2, key % nv2]), minlength=nv2)
    # polygons around a polygon (itself included) by inclusion-exclusion over shared vertices and edges
    pairs = (nint.astype(np.int64) ** 2).sum() - 2 * key.size - (n - 1) * cells.shape[0]
    return nint, nedge, pairs


def _work_block(nv2, cells, nl, top):
    nint, nedge, pairs = _surface_counts(nv2, cells)
    rc, r, rn = _counts(nint, nedge, cells.shape[0], nl, top)
    nnz = pairs * (3 * nl - 2)
    return np.array([nl * cells.shape[0], rc, r, rn, nnz], dtype=np.float64)


def work(case):
    """Each input read once, each output written once (the transmissibility
    rows, a gravity term per row, seven fields and the pressure per cell, R and
    J), and the arithmetic of the rows and of the Jacobian products.  A Newton
    step: three iterations' residuals and Jacobians, and four Krylov iterations
    (two products with the matrix in the inner precision) in each."""
    from tdycore_gb300.workloads import structured_surface

    mesh = case["mesh"]
    top = mesh != "prism"
    if mesh == "prism":
        xy, tris = _prism_surface(case["triangles"])
        tot = _work_block(xy.shape[0], tris, case["layers"], top)
    elif mesh == "batch":
        nx, ny, nz, _ = _column_shapes(case["instances"])
        tot = 0
        for b in range(nx.size):
            xy, quads = structured_surface(int(nx[b]), int(ny[b]), 1.0, 1.0)
            tot = tot + _work_block(xy.shape[0], quads, int(nz[b]), top)
    else:
        xy, quads = structured_surface(case["nx"], case["ny"], 1.0, 1.0)
        tot = _work_block(xy.shape[0], quads, case["nz"], top)
    nc, rc, r, rn, nnz = (float(v) for v in tot)
    if case["call"] == "f":
        return {"bytes": 8 * (rc + r + 9 * nc), "flops": 2 * rc + 8 * r + 100 * nc}
    nbytes, flops = 8 * (rc + r + 9 * nc + nnz), 2 * rc + 8 * r + 100 * nc + 4 * rn
    if case["call"] == "newton":
        size = 4 if case["fp32"] else 8
        nbytes = 3 * nbytes + 3 * 4 * 2 * (size + 4) * nnz
        flops = 3 * flops + 3 * 4 * 2 * 2 * nnz
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same outputs in plain torch, 64 bits


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    return a / torch.sqrt(_dot(a, a)).unsqueeze(-1)


def _topology(blocks, dev):
    """Vertices, cells and faces of the extruded blocks: horizontal faces of
    every block first, then vertical ones."""
    n = blocks[0][1].shape[1]
    vx, cverts, cfaces, hverts, vverts, hcells, vcells, htop = [], [], [], [], [], [], [], []
    v0 = c0 = h0 = e0 = 0
    for b, (xy, cells, z) in enumerate(blocks):
        nv2, nc2, nl = xy.shape[0], cells.shape[0], z.shape[0] - 1
        cells = cells.astype(np.int64)
        vx.append(np.concatenate([np.tile(xy, (nl + 1, 1)), z.reshape(-1, 1)], axis=1))
        lay = np.arange(nl)[:, None, None]
        cverts.append((v0 + np.concatenate([cells[None] + lay * nv2, cells[None] + (lay + 1) * nv2], axis=2)).reshape(-1, 2 * n))
        a, bb = cells, np.roll(cells, -1, axis=1)
        key, first, inv = np.unique((np.minimum(a, bb) * nv2 + np.maximum(a, bb)).ravel(), return_index=True, return_inverse=True)
        inv = inv.reshape(nc2, n)
        ea, eb = a.ravel()[first], bb.ravel()[first]
        ne = key.size
        ec = np.full((ne, 2), -1, dtype=np.int64)
        order = np.argsort(inv.ravel(), kind="stable")
        poly = np.repeat(np.arange(nc2), n)[order]
        start = np.searchsorted(inv.ravel()[order], np.arange(ne))
        cnt = np.bincount(inv.ravel(), minlength=ne)
        ec[:, 1] = poly[start]
        two = cnt == 2
        ec[two, 0], ec[two, 1] = poly[start[two]], poly[start[two] + 1]
        hverts.append((v0 + cells[None] + np.arange(nl + 1)[:, None, None] * nv2).reshape(-1, n))
        hc = np.full((nl + 1, nc2, 2), -1, dtype=np.int64)
        ids = c0 + np.arange(nl)[:, None] * nc2 + np.arange(nc2)[None]
        hc[1:, :, 0], hc[:-1, :, 1] = ids, ids
        hc[-1, :, 1], hc[-1, :, 0] = ids[-1], -1  # a boundary face: its cell second
        hcells.append(hc.reshape(-1, 2))
        t = np.full((nl + 1, nc2), -1, dtype=np.int64)
        t[-1] = b
        htop.append(t.ravel())
        lay = np.arange(nl)[:, None]
        vverts.append((v0 + np.stack([ea + lay * nv2, eb + lay * nv2, eb + (lay + 1) * nv2, ea + (lay + 1) * nv2], axis=2)).reshape(-1, 4))
        vcells.append(np.where(ec[None] >= 0, c0 + ec[None] + np.arange(nl)[:, None, None] * nc2, -1).reshape(-1, 2))
        lay = np.arange(nl)[:, None, None]
        c = np.arange(nc2)[None, :, None]
        cfaces.append(np.concatenate([h0 + lay * nc2 + c, h0 + (lay + 1) * nc2 + c, -1 - (e0 + lay * ne + inv[None])], axis=2).reshape(-1, 2 + n))
        v0, c0, h0, e0 = v0 + (nl + 1) * nv2, c0 + nl * nc2, h0 + (nl + 1) * nc2, e0 + nl * ne
    cf = np.concatenate(cfaces)
    cf = np.where(cf < 0, h0 - 1 - cf, cf)
    to = lambda v: torch.as_tensor(np.concatenate(v), device=dev)  # noqa: E731
    return {"n": n, "nh": h0, "vx": to(vx), "cverts": to(cverts), "cfaces": torch.as_tensor(cf, device=dev), "hverts": to(hverts),
            "vverts": to(vverts), "fcells": to(hcells + vcells), "htop": torch.cat([to(htop), torch.full((e0,), -1, device=dev)])}


def _geometry(m):
    """Areas, centroids, normals (first to second cell, inward on the
    boundary), subface areas; cell volumes and centroids."""
    vx, n, nh = m["vx"], m["n"], m["nh"]
    area, cen, nrm, fan = [], [], [], []
    for verts in (m["hverts"], m["vverts"]):
        P = vx[verts]
        c0 = P.mean(1, keepdim=True)
        a, b = P - c0, P.roll(-1, 1) - c0
        w = _cross(a, b)
        t = 0.5 * torch.sqrt(_dot(w, w))
        area.append(t.sum(1))
        cen.append((t.unsqueeze(-1) * (c0 + P + P.roll(-1, 1)) / 3.0).sum(1) / area[-1].unsqueeze(-1))
        nrm.append(_unit(_cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])) if verts.shape[1] == 3 else _unit(w).sum(1) / 4.0)
        fan.append((P, c0))
    m["area"], m["fcen"], nrm = torch.cat(area), torch.cat(cen), torch.cat(nrm)
    sub = torch.cat([torch.full_like(area[0], n), torch.full_like(area[1], 4)])
    m["subarea"] = m["area"] / sub
    apex = vx[m["cverts"]].mean(1)
    vol, mom = 0.0, 0.0
    for k in range(2 + n):
        P, c0 = fan[0 if k < 2 else 1]
        f = m["cfaces"][:, k] - (0 if k < 2 else nh)
        a, b, c = P[f], P[f].roll(-1, 1), c0[f]
        ax = apex.unsqueeze(1)
        v = _dot(_cross(a - ax, b - ax), c - ax).abs() / 6.0
        vol = vol + v.sum(1)
        mom = mom + (v.unsqueeze(-1) * (ax + c + a + b) / 4.0).sum(1)
    m["vol"], m["ccen"] = vol, mom / vol.unsqueeze(-1)
    c0, c1 = m["fcells"][:, 0], m["fcells"][:, 1]
    d = m["ccen"][c1] - torch.where((c0 >= 0).unsqueeze(-1), m["ccen"][c0.clamp(min=0)], m["fcen"])
    m["nrm"] = torch.where((_dot(nrm, d) < 0).unsqueeze(-1), -nrm, nrm)


def _gravity_term(m, K):
    """Per face: subface area (n . K_f u) (g . u), u between the centroids, K_f
    the distance-weighted harmonic mean with its negative and negligible
    entries dropped."""
    c0, c1 = m["fcells"][:, 0], m["fcells"][:, 1]
    inner = (c0 >= 0).unsqueeze(-1)
    xu = torch.where(inner, m["ccen"][c0.clamp(min=0)], m["fcen"])
    u = _unit(m["ccen"][c1] - xu)
    dup = torch.sqrt(_dot(xu - m["fcen"], xu - m["fcen"]))
    ddn = torch.sqrt(_dot(m["ccen"][c1] - m["fcen"], m["ccen"][c1] - m["fcen"]))
    w = (dup / (dup + ddn)).reshape(-1, 1, 1)
    Ki = torch.linalg.inv(K)
    Kf = torch.linalg.inv(w * Ki[torch.where(c0 >= 0, c0, c1)] + (1.0 - w) * Ki[c1])
    Kf = torch.where((Kf < 0) | (Kf.abs() < 2.220446049250313e-16), torch.zeros_like(Kf), Kf)
    return m["subarea"] * _dot(m["nrm"], (Kf @ u.unsqueeze(-1)).squeeze(-1)) * GRAVITY * u[:, 2]


def _interaction_regions(m, K, dirichlet, neumann):
    """Groups of vertices of one shape: transmissibility rows T (rows x
    columns), row faces, the local index of each row's first and second cell
    (-1: the boundary), column cells and column boundary faces."""
    dev, n, nf = m["vx"].device, m["n"], m["area"].numel()
    cf, nc = m["cfaces"], m["cfaces"].shape[0]
    faces = []
    for end in (0, 1):
        for j in range(n):
            faces.append(torch.stack([cf[:, end], cf[:, 2 + j], cf[:, 2 + (j - 1) % n]], 1))
    face = torch.stack(faces, 1).reshape(-1, 3)
    vert = m["cverts"].reshape(-1)
    cell = torch.arange(nc, device=dev).repeat_interleave(2 * n)
    order = torch.argsort(vert, stable=True)
    face, vert, cell = face[order], vert[order], cell[order]
    fc, xc = m["fcen"][face], m["ccen"][cell]
    swap = _dot(_cross(fc[:, 1] - fc[:, 0], fc[:, 2] - fc[:, 0]), xc - m["vx"][vert]) < 0
    face = torch.where(swap.unsqueeze(-1), face[:, [0, 2, 1]], face)
    fc = m["fcen"][face] - xc.unsqueeze(1)
    vol6 = _dot(_cross(fc[:, 0], fc[:, 1]), fc[:, 2]).abs()
    nu = torch.stack([_cross(fc[:, 1], fc[:, 2]), _cross(fc[:, 2], fc[:, 0]), _cross(fc[:, 0], fc[:, 1])], 1)
    G = m["nrm"][face] @ (nu @ K[cell].transpose(1, 2)).transpose(1, 2)
    G = G * (m["subarea"][face] / vol6.unsqueeze(-1)).unsqueeze(-1)
    # subfaces: (vertex, face) pairs in order, and each one's rank among its vertex's unknowns, knowns, rows
    key, sf = torch.unique(vert.unsqueeze(-1) * nf + face, return_inverse=True)
    kv, kf = key // nf, key % nf
    nv = m["vx"].shape[0]

    def rank(flag):
        c = torch.cumsum(flag.long(), 0)
        per = torch.zeros(nv, dtype=torch.long, device=dev).index_add_(0, kv, flag.long())
        return c - 1 - (torch.cumsum(per, 0) - per)[kv], per

    unk, nunk = rank(~dirichlet[kf])
    knw, nknw = rank(dirichlet[kf])
    row, nrow = rank(~neumann[kf])
    nint = torch.bincount(vert, minlength=nv)
    local = torch.arange(vert.numel(), device=dev) - (torch.cumsum(nint, 0) - nint)[vert]
    shape = ((nunk * 256 + nknw) * 256 + nint) * 256 + nrow
    groups = []
    for g in torch.unique(shape[nint > 0]).tolist():
        members = torch.nonzero((shape == g) & (nint > 0)).reshape(-1)
        step = 100_000
        for o in range(0, members.numel(), step):
            mem = members[o:o + step]
            groups.append(_region_group(m, mem, nv, vert, cell, face, local, sf, kv, kf, unk, knw, row, G, dirichlet, neumann,
                                        (int(nunk[mem[0]]), int(nknw[mem[0]]), int(nint[mem[0]]), int(nrow[mem[0]]))))
    return groups


def _region_group(m, mem, nv, vert, cell, face, local, sf, kv, kf, unk, knw, row, G, dirichlet, neumann, sizes):
    U, Kn, N, Rw = sizes
    dev, f64 = G.device, G.dtype
    pos = torch.full((nv,), -1, dtype=torch.long, device=dev)
    pos[mem] = torch.arange(mem.numel(), device=dev)
    s = torch.nonzero(pos[vert] >= 0).reshape(-1)
    v, c, a = pos[vert[s]], cell[s], local[s]
    A = torch.zeros(mem.numel(), U, U, dtype=f64, device=dev)
    B = torch.zeros(mem.numel(), U, N + Kn, dtype=f64, device=dev)
    C = torch.zeros(mem.numel(), Rw, U, dtype=f64, device=dev)
    T = torch.zeros(mem.numel(), Rw, N + Kn, dtype=f64, device=dev)
    rface = torch.zeros(mem.numel(), Rw, dtype=torch.long, device=dev)
    lup = torch.full((mem.numel(), Rw), -1, dtype=torch.long, device=dev)
    ldn = torch.full((mem.numel(), Rw), -1, dtype=torch.long, device=dev)
    ccell = torch.zeros(mem.numel(), N, dtype=torch.long, device=dev)
    cbnd = torch.zeros(mem.numel(), Kn, dtype=torch.long, device=dev)
    ccell[v, a] = c
    for i in range(3):
        fi, si = face[s, i], sf[s, i]
        first = (m["fcells"][fi, 0] == c) | (m["fcells"][fi, 0] < 0)
        sign = torch.where(first, 1.0, -1.0).to(f64)
        eq = ~dirichlet[fi]
        out = first & ~neumann[fi]
        gi = G[s, i]
        tot = gi.sum(1)
        B.index_put_((v[eq], unk[si][eq], a[eq]), (sign * tot)[eq], accumulate=True)
        T.index_put_((v[out], row[si][out], a[out]), tot[out], accumulate=True)
        rface[v[out], row[si][out]] = fi[out]
        inner = m["fcells"][fi, 0] >= 0
        up, dn = inner & first, ~neumann[fi] & ~(inner & first)
        lup[v[up], row[si][up]] = a[up]
        ldn[v[dn], row[si][dn]] = a[dn]
        for j in range(3):
            sj = sf[s, j]
            kj = dirichlet[face[s, j]]
            q = eq & ~kj
            A.index_put_((v[q], unk[si][q], unk[sj][q]), (sign * gi[:, j])[q], accumulate=True)
            q = eq & kj
            B.index_put_((v[q], unk[si][q], N + knw[sj][q]), -(sign * gi[:, j])[q], accumulate=True)
            q = out & ~kj
            C.index_put_((v[q], row[si][q], unk[sj][q]), -gi[q, j], accumulate=True)
            q = out & kj
            T.index_put_((v[q], row[si][q], N + knw[sj][q]), -gi[q, j], accumulate=True)
        k = dirichlet[fi]
        cbnd[v[k], knw[si][k]] = fi[k]
    if U:
        T = T + C @ torch.linalg.solve(A, B)
    return {"T": T, "face": rface, "lup": lup, "ldn": ldn, "cell": ccell, "bnd": cbnd}


def _density(kind, p):
    if kind == "constant":
        return torch.full_like(p, RHO0), torch.zeros_like(p), torch.zeros_like(p)
    r = 997.16 * torch.exp(1e-8 * (p - PREF))
    low = p < PREF
    z = torch.zeros_like(p)
    return torch.where(low, z + 997.16, r), torch.where(low, z, 1e-8 * r), torch.where(low, z, 1e-16 * r)


def _smoothing(mm, device):
    """The cubic that takes kr from its value and slope at Se = 0.99 to 1, flat, at Se = 1."""
    x0, x1, x2, dx = 0.995, 0.99, 1.0, 0.005
    so = x1 ** (1.0 / mm)
    t = 1.0 - (1.0 - so) ** mm
    kr = math.sqrt(x1) * t * t
    slope = 0.5 * kr / x1 + 2.0 * x1 ** (1.0 / mm - 0.5) * (1.0 - so) ** (mm - 1.0) * t
    a, b = (x1 - x0) / dx, (x2 - x0) / dx
    M = np.array([[1, b, b * b, b ** 3], [1, a, a * a, a ** 3], [0, 1 / dx, 2 * b / dx, 3 * b * b / dx],
                  [0, 1 / dx, 2 * a / dx, 3 * a * a / dx]])
    return M, kr, slope


def _curves(p, m, alpha, sr):
    """S, dS/dP, d2S/dP2, kr, dkr/dP of van Genuchten and smoothed Mualem."""
    pc = PREF - p
    wet = pc <= 0
    x = torch.where(wet, torch.ones_like(pc), pc) * alpha
    n = 1.0 / (1.0 - m)
    xn = x ** n
    one = 1.0 + xn
    se = one ** (-m)
    pcs = torch.where(wet, torch.ones_like(pc), pc)
    dse = -m * n * alpha * xn * se / (x * one)
    d2se = m * n * xn * (se / (one * one)) * ((m * n + 1.0) * xn - n + 1.0) / (pcs * pcs)
    so = 1.0 / one  # Se^(1/m)
    tmp = (xn / one) ** m  # (1 - so)^m
    f = -torch.expm1(m * torch.log1p(-so))
    kr = torch.sqrt(se) * f * f
    dkr = 0.5 * kr / se + 2.0 * (so / torch.sqrt(se)) * (tmp / (xn / one)) * f
    x0, x1, dx = 0.995, 0.99, 0.005
    M, _, _ = _smoothing(0.5, p.device)
    so1 = x1 ** (1.0 / m)
    t1 = 1.0 - (1.0 - so1) ** m
    kr1 = math.sqrt(x1) * t1 * t1
    sl1 = 0.5 * kr1 / x1 + 2.0 * x1 ** (1.0 / m - 0.5) * (1.0 - so1) ** (m - 1.0) * t1
    Mi = torch.as_tensor(np.linalg.inv(M), device=p.device)
    co = torch.stack([torch.ones_like(m), kr1, torch.zeros_like(m), sl1], -1) @ Mi.T
    xt = (torch.where(wet, torch.ones_like(se), se) - x0) / dx
    krs = co[:, 0] + xt * (co[:, 1] + xt * (co[:, 2] + xt * co[:, 3]))
    dkrs = (co[:, 1] + xt * (2.0 * co[:, 2] + xt * 3.0 * co[:, 3])) / dx
    high = wet | (se > x1)
    kr, dkr = torch.where(high, krs, kr), torch.where(high, dkrs, dkr)
    zero = torch.zeros_like(p)
    dS = torch.where(wet, zero, -dse * (1.0 - sr))
    return (torch.where(wet, zero + 1.0, (1.0 - sr) * se + sr), dS, torch.where(wet, zero, (1.0 - sr) * d2se), kr,
            torch.where(wet, zero, dkr * dS / (1.0 - sr)))


class _Exact:
    """Residual and Jacobian of a problem in plain torch, 64 bits."""

    def __init__(self, case, p):
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        to = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.case, self.p, self.dev = case, p, dev
        m = self.m = _topology(p["blocks"], dev)
        _geometry(m)
        K = to(p["K"]).reshape(-1, 3, 3)
        outer = m["fcells"][:, 0] < 0
        top = p["top"]
        self.bval = None
        if top is None:
            dirichlet = torch.zeros_like(outer)
        elif isinstance(top, str):
            dirichlet = outer
        else:
            dirichlet = m["htop"] >= 0
            self.bval = to(top)[m["htop"].clamp(min=0)]
        self.G = _gravity_term(m, K)
        self.groups = _interaction_regions(m, K, dirichlet, outer & ~dirichlet)
        self.dirichlet = dirichlet
        self.poro, self.mm, self.alpha = to(p["poro"]), to(p["m"]), to(p["alpha"])
        self.source = to(p["source"]) if p["source"] is not None else torch.zeros_like(self.poro)
        self.nc = self.poro.numel()
        keys = [torch.unique((g["cell"].unsqueeze(2) * self.nc + g["cell"].unsqueeze(1)).reshape(-1)) for g in self.groups]
        self.keys = torch.unique(torch.cat(keys))
        self.diag = torch.searchsorted(self.keys, torch.arange(self.nc, device=dev) * (self.nc + 1))
        self.Uprev, self.Ut = to(p["Uprev"]), to(p["Ut"])

    def _mass(self, U):
        rho, drho, d2rho = _density(self.case["density"], U)
        S, dS, d2S, kr, dkr = _curves(U, self.mm, self.alpha, self.p["sr"])
        return rho, drho, d2rho, S, dS, d2S, kr, dkr

    def __call__(self, U, jac=True, prev=None):
        p, m, nc, dev = self.p, self.m, self.nc, self.dev
        rho, drho, d2rho, S, dS, d2S, kr, dkr = self._mass(U)
        poro, vol = self.poro, m["vol"]
        # extended state: cells, then faces (the Dirichlet ones are used)
        c1 = m["fcells"][:, 1]
        bp = U[c1] if self.bval is None else self.bval
        bkr = _curves(bp, self.mm[c1], self.alpha[c1], p["sr"])[3]
        brho = _density(self.case["density"], torch.full_like(bp, PREF))[0]
        P, lam = torch.cat([U, bp]), torch.cat([kr, bkr]) / VISCOSITY
        half, dhalf = 0.5 * torch.cat([rho, brho]), 0.5 * torch.cat([drho, torch.zeros_like(bp)])
        dlam = torch.cat([dkr, torch.zeros_like(bp)]) / VISCOSITY
        R = torch.zeros(nc, dtype=torch.float64, device=dev)
        J = torch.zeros(self.keys.numel(), dtype=torch.float64, device=dev) if jac else None
        for g in self.groups:
            N, T = g["cell"].shape[1], g["T"]
            if T.shape[1] == 0:
                continue
            cols = torch.cat([g["cell"], nc + g["bnd"]], 1)
            TP = (T @ P[cols].unsqueeze(-1)).squeeze(-1)
            f = g["face"]
            c0 = m["fcells"][f, 0]
            eu, ed = torch.where(c0 >= 0, c0, nc + f), m["fcells"][f, 1]
            den = half[eu] + half[ed]
            q = TP + den * self.G[f]
            down = q < 0
            lm = torch.where(down, lam[eu], lam[ed])
            w = den * lm
            flux = -w * q
            inner = (c0 >= 0).reshape(-1)
            R.index_add_(0, c0.reshape(-1)[inner], flux.reshape(-1)[inner])
            R.index_add_(0, ed.reshape(-1), -flux.reshape(-1))
            if not jac:
                continue
            g2 = q + den * self.G[f]
            Eu = dhalf[eu] * lm * g2 + den * torch.where(down, dlam[eu], torch.zeros_like(q)) * q
            Ed = dhalf[ed] * lm * g2 + den * torch.where(down, torch.zeros_like(q), dlam[ed]) * q
            V = -w.unsqueeze(-1) * T[:, :, :N]
            vi = torch.arange(V.shape[0], device=dev).unsqueeze(1).expand_as(f)
            ri = torch.arange(V.shape[1], device=dev).unsqueeze(0).expand_as(f)
            for loc, E in ((g["lup"], Eu), (g["ldn"], Ed)):
                k = loc >= 0
                V.index_put_((vi[k], ri[k], loc[k]), -E[k], accumulate=True)
            colc = g["cell"].unsqueeze(1).expand_as(V)
            for rows, sgn in ((eu, 1.0), (ed, -1.0)):
                k = (rows < nc).unsqueeze(-1).expand_as(V)
                key = (rows.unsqueeze(-1) * nc + colc)[k]
                J.index_add_(0, torch.searchsorted(self.keys, key), sgn * V[k])
        dmass = poro * (drho * S + rho * dS)
        if self.case["call"] == "ij":
            d2mass = poro * (2.0 * drho * dS + S * d2rho + rho * d2S)
            R += dmass * self.Ut * vol - self.source * vol
            diag = (p["shift"] * dmass + d2mass * self.Ut) * vol
        else:
            if prev is None:
                prev = self.Uprev
            pr, _, _, pS = self._mass(prev)[:4]
            R += (rho * S - pr * pS) * poro * vol / p["dt"] - self.source
            diag = dmass * vol / p["dt"]
        if jac:
            J.index_add_(0, self.diag, diag)
        return R, J

    def step(self):
        """The solution of one backward-Euler step from U by damped Newton with dense solves."""
        U0 = torch.as_tensor(self.p["U"], dtype=torch.float64, device=self.dev)
        U, best = U0.clone(), math.inf
        rows, cols = self.keys // self.nc, self.keys % self.nc
        for _ in range(60):
            R, J = self(U, prev=U0)
            norm = float(R.norm())
            D = torch.zeros(self.nc, self.nc, dtype=torch.float64, device=self.dev)
            D[rows, cols] = J
            d = torch.linalg.solve(D, R)
            lam = 1.0
            while lam > 1e-4 and float(self(U - lam * d, jac=False, prev=U0)[0].norm()) > (1 - 1e-4 * lam) * norm:
                lam *= 0.5
            if lam <= 1e-4:  # at the rounding floor
                break
            U = U - lam * d
        return U


def exact(case, seed):
    call = case["call"]
    if call == "newton":
        if case["mesh"] != "box":
            return None  # no direct solve of these in the time
        return {"U": _Exact(case, _problem(case, seed)).step(), "iterations": None, "status": None}
    p = _problem(case, seed)
    R, J = _Exact(case, p)(torch.as_tensor(p["U"], dtype=torch.float64, device="cuda" if torch.cuda.is_available() else "cpu"),
                           jac=call != "f")
    return {"R": R} if J is None else {"R": R, "J": J}
