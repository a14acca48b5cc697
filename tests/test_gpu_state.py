"""gfb_get_state reads the state in ranges of nodes: through the contribution
buffer (one FP32 wavefield's is smaller than the state, so two ranges), or
through page-locked memory in a solver without that buffer, with no device
memory of its own (a full device is where such a solver comes from).

What comes back is what was set: u and a exactly as stored (a in the precision's
type); v exactly in FP64, in FP32 from the half-step velocity w = v + dt/2 a, kept
in float, with one rounding of w: at most 2^-24 of the largest |w|."""

import numpy as np
import pytest

import gfb
from gfb import mesh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def prob():
    # 73 x 73 x 69 nodes: more than one range of 8 MiB
    spec = mesh.MeshSpec(nx=18, ny=18, nz=17, dx=500.0, dy=500.0, dz=500.0, order=4, seed=2)
    p = mesh.build_problem(spec, mesh.seeded_layers(2, 17 * 500.0), np.asarray([4100.0, 4200.0, 800.0]), nsteps=10,
                           record_depth_max_m=500.0, with_cpml=False)
    p.pop("damping", None)
    assert p["n_node"] * 24 > 8 << 20
    return p


@pytest.mark.parametrize("prec", [gfb.FP64, gfb.FP32])
@pytest.mark.parametrize("dirs", [[2], [0, 1]])
@pytest.mark.parametrize("flags", [0, gfb.FLAG_COLOUR])
def test_state_round_trip(prob, dirs, prec, flags):
    rng = np.random.default_rng(8)
    s = gfb.Solver(prob, dirs=dirs, precision=prec, record=False, flags=flags)
    want = [[rng.standard_normal((prob["n_node"], 3)) * k for k in (1.0, 3.0, 50.0)] for _ in dirs]
    for f, x in enumerate(want):
        s.set_state(f, 0, *x)
    mem = s.info()["device_bytes"]
    for f, (u, v, a) in enumerate(want):
        gu, gv, ga = s.state(f)
        np.testing.assert_array_equal(gu, u)
        if prec == gfb.FP64:
            np.testing.assert_array_equal(gv, v)
            np.testing.assert_array_equal(ga, a)
        else:
            np.testing.assert_array_equal(ga, a.astype(np.float32))
            w = np.abs(v).max() + 0.5 * prob["dt"] * np.abs(a).max()
            assert np.abs(gv - v).max() <= 2.0**-24 * w * 1.01
    if flags & gfb.FLAG_COLOUR:
        assert s.info()["device_bytes"] == mem
    s.close()


def test_states_read_twice_and_between_steps(prob):
    """The buffer that the state goes through belongs to the steps: they are the
    same with and without a read-out between them, by both ways out."""
    out = []
    for flags, read in ((0, False), (0, True), (gfb.FLAG_COLOUR, False), (gfb.FLAG_COLOUR, True)):
        s = gfb.Solver(prob, dirs=[0], precision=gfb.FP32, record=False, flags=flags)
        s.set_state(0, 0, np.random.default_rng(1).standard_normal((prob["n_node"], 3)))
        for _ in range(3):
            s.advance(4)
            if read:
                s.state(0)
        out.append(s.state(0))
        for x, y in zip(out[-1], s.state(0)):
            np.testing.assert_array_equal(x, y)
        s.close()
    for i in (0, 2):
        for x, y in zip(out[i], out[i + 1]):
            np.testing.assert_array_equal(x, y)
