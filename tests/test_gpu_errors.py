"""A kernel whose bounded wait for its own copies gave up leaves a flag, and
no call hands out results from then on.  The flag is set from the host here:
no kernel can be made to lose a copy."""

import ctypes as C

import numpy as np
import pytest

import gfb
from gfb import mesh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prob():
    spec = mesh.MeshSpec(nx=5, ny=4, nz=4, dx=500.0, dy=500.0, dz=500.0, order=4, jitter=0.05, seed=3,
                         pml={f: 1 for f in ("xmin", "xmax", "ymin", "ymax", "zmax")})
    mat = mesh.seeded_layers(3, 4 * 500.0)
    return mesh.build_problem(spec, mat, np.asarray([1400.0, 1100.0, 800.0]), nsteps=80, snapshot_stride=4,
                              record_depth_max_m=500.0)


def inject(s):
    fn = s.lib.gfb_inject_kernel_error
    fn.restype, fn.argtypes = C.c_int, [C.c_void_p]
    assert fn(s.h) == 0


@pytest.mark.parametrize("prec", [gfb.FP64, gfb.FP32])
@pytest.mark.parametrize("slots", [1, 4])  # one slot: the snapshots read are spilled ones
def test_no_result_leaves_a_solver_with_an_abandoned_launch(prob, prec, slots):
    s = gfb.Solver(prob, dirs=[0, 2], precision=prec, record_slots=slots)
    s.advance(9)
    s.synchronize()
    s.state(0)
    s.read_record(0)
    inject(s)
    calls = {
        "synchronize": s.synchronize,
        "state": lambda: s.state(1),
        "checkpoint": s.checkpoint,
        "read_record": lambda: s.read_record(1),
        "read_record_f32": lambda: s.read_record(1, dtype=np.float32),
        "read_green": s.read_green,
        "drain": s.drain,
        "advance_timed": lambda: s.advance_timed(1),
        "advance_profiled": lambda: s.advance_profiled(1),
        "run": lambda: s.run(4),
    }
    for name, call in calls.items():
        with pytest.raises(gfb.GfbError, match="the state is invalid"):
            call()
            pytest.fail(f"{name} returned a result")
    s.close()
    s = gfb.Solver(prob, dirs=[0, 2], precision=prec, record_slots=slots)  # other solvers are not concerned
    s.run(9)
    s.state(0)
    s.close()
