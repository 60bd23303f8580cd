"""The library linked against fake_cudart.cpp (argument 1), in a process of its
own: what its device Newton does when a runtime call is refused."""
import ctypes
import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parents[2]))
_cdll = ctypes.CDLL
ctypes.CDLL = lambda name, *a, **k: _cdll(sys.argv[1] if "libtdycore" in str(name) else name, *a, **k)
import tdycore_gb300 as T  # noqa: E402
from tdycore_gb300.workloads import layered_z, structured_surface  # noqa: E402

fake = _cdll(sys.argv[1])
for name in ("fake_calls", "fake_launches", "fake_violations", "fake_in_flight", "fake_null_stream"):
    getattr(fake, name).restype = ctypes.c_longlong
fake.fake_arm.argtypes = [ctypes.c_longlong]


def handle():
    """Instances of three launch classes of the block schedule."""
    t = T.create_richards_mpfao()
    blocks, x0 = [], 0.0
    for n, nz in ((1, 4), (4, 20), (8, 8)):
        xy, quads = structured_surface(n, n, float(n), float(n))
        xy[:, 0] += x0
        x0 += n + 1.0
        blocks.append((xy, quads, layered_z(xy.shape[0], nz, 0.3 * nz)))
    t.set_extruded_meshes(blocks)
    t.set_from_options()
    t.set_constant_isotropic_permeability(1e-12)
    t.set_boundary_pressure_type_function(lambda x, y, z: np.full(np.shape(x), T.NEUMANN_BC))
    t.setup()
    return t


def new_stream():
    st = ctypes.c_void_p()
    assert fake.cudaStreamCreateWithFlags(ctypes.byref(st), 1) == 0
    return st.value


def step(t, U, k=0, **kw):
    """One step whose k-th call is refused (0: none); whether it succeeded."""
    fake.fake_arm(k)
    try:
        t.backward_euler_step_device(U.ctypes.data, 10.0, max_it=1, **kw)
        ok = True
    except T.TDyError:
        ok = False
    return ok


def refusals(stream):
    """Every call of a step refused in turn: the step fails, leaves nothing in
    flight, and the handle's memory is freed after its last use."""
    st = new_stream() if stream == "caller" else None
    for k in range(1, 10000):
        t = handle()
        U = np.full(t.ncells, 1e5)
        ok = step(t, U, k, schedule="block", stream=st)
        calls, flying = fake.fake_calls(), fake.fake_in_flight()
        fake.fake_arm(0)
        t.destroy()
        assert flying == 0 and fake.fake_violations() == 0 and fake.fake_in_flight() == 0, k
        if calls < k:
            assert ok and k > 100, k
            return
    raise AssertionError("the step never ended")


def again():
    """A refused step, then the same step on the same handle: it succeeds, makes
    the copy or launch that was refused, and nothing goes to the null stream.  (The handles live to the end, so that
    each takes new streams and events.)"""
    handles = []
    for k in range(1, 10000):
        t = handle()
        handles.append(t)
        U = np.full(t.ncells, 1e5)
        step(t, U, k, schedule="block")
        calls = fake.fake_calls()
        assert step(t, U, schedule="block") and fake.fake_null_stream() == 0 and not fake.fake_missed(), k
        if calls < k:
            assert k > 100, k
            return
    raise AssertionError("the step never ended")


def tuning(first):
    """The schedule is timed once for each precision of a size class, whichever
    comes first.  (The timed solves take 16 launches more than a step's own.)"""
    def extra(t, fp32):
        n = []
        for _ in range(2):
            assert step(t, U, fp32=fp32, spmv_threads=4)
            n.append(fake.fake_launches())
        return n[0] - n[1]

    t, order = handle(), (first == "fp32", first != "fp32")
    U = np.full(t.ncells, 1e5)
    assert [extra(t, fp32) > 8 for fp32 in order] == [True, True]
    t = handle()  # another of the class
    assert [extra(t, fp32) > 8 for fp32 in order] == [False, False]


if __name__ == "__main__":
    globals()[sys.argv[2]](*sys.argv[3:])
