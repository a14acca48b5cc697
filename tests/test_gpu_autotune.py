"""GFB_FLAG_AUTOTUNE compares what a step takes with each kernel.  The default's
assembly is part of its node pass; timed as a pass of its own it lost against
kernels that make the step a quarter longer (501 against 399 us on 40 x 40 x 20
cells).  Tuning leaves no trace in the state."""

import numpy as np
import pytest

import gfb
from gfb import mesh

pytestmark = pytest.mark.gpu


def test_autotuner_keeps_the_faster_step():
    spec = mesh.MeshSpec(nx=40, ny=40, nz=20, dx=500.0, dy=500.0, dz=500.0, order=4, seed=2,
                         pml={f: 4 for f in ("xmin", "xmax", "ymin", "ymax", "zmax")})
    prob = mesh.build_problem(spec, mesh.seeded_layers(2, 10000.0), np.asarray([9100.0, 9200.0, 2800.0]), nsteps=40,
                              record_depth_max_m=500.0)
    a = gfb.Solver(prob, dirs=[0, 1, 2], precision=gfb.FP32, record=False)
    b = gfb.Solver(prob, dirs=[0, 1, 2], precision=gfb.FP32, record=False, flags=gfb.FLAG_AUTOTUNE)
    assert not b.by_colour and b.info()["elem_variant"] == 0
    assert a.checkpoint()[200:] == b.checkpoint()[200:]  # past the header, which holds the flags
    for s in (a, b):
        s.advance(12)
    for f in range(3):
        for x, y in zip(a.state(f), b.state(f)):
            np.testing.assert_array_equal(x, y)
    a.close()
    b.close()
