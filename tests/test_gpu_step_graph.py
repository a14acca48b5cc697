"""A step's kernels overlap when a graph replays them (each waits for what it
reads, gfb::pdl_wait) and follow one another when launched one by one: the same
values bit for bit, over the shapes whose chains differ -- the plane kernel, the
line kernel that the node passes wait out, ngll 3, per-cell C-PML, no C-PML, only
C-PML cells, several models of which one finishes."""

import numpy as np
import pytest

import gfb
from gfb import mesh

pytestmark = pytest.mark.gpu


def problem(order=4, pml=1, cpml=True, n=(7, 6, 5), seed=4):
    spec = mesh.MeshSpec(nx=n[0], ny=n[1], nz=n[2], dx=500.0, dy=500.0, dz=500.0, order=order, jitter=0.05, seed=seed,
                         pml={f: pml for f in ("xmin", "xmax", "ymin", "ymax", "zmax")})
    return mesh.build_problem(spec, mesh.seeded_layers(seed, n[2] * 500.0), np.asarray([1700.0, 1300.0, 700.0]),
                              nsteps=60, snapshot_stride=7, record_depth_max_m=500.0, with_cpml=cpml)


def outputs(make, flags):
    s = make(flags)
    s.advance(3)
    out = s.run(41)
    st = [s.state(f) for f in range(s.n_field)]
    s.close()
    return out, st


@pytest.mark.parametrize("order,dirs,prec,more", [
    (4, [0, 1, 2], gfb.FP32, {}), (4, [1], gfb.FP32, {}), (2, [2, 0], gfb.FP32, {}), (3, [0, 1, 2], gfb.FP32, {}),
    (4, [0, 1, 2], gfb.FP32, {"cpml": False}), (4, [2], gfb.FP64, {}), (4, [0, 1], gfb.FP32, {"flags": gfb.FLAG_CELL_PML}),
    (4, [0, 1, 2], gfb.FP32, {"all_pml": True}),
])
def test_replayed_steps_equal_steps_launched_one_by_one(order, dirs, prec, more):
    prob = problem(order, cpml=more.get("cpml", True))
    if more.get("all_pml"):  # no plain node is left: the C-PML pass alone
        on = np.asarray(prob["pml_region"]) != 0
        nn = (order + 1) ** 3
        al, ab = (np.array(prob[k], dtype=np.float64).reshape(len(on), nn, -1) for k in ("pml_coef_alpha", "pml_coef_abar"))
        al[:] = al[on][0, 0]
        ab[..., 0] += 1e-3 * (ab == 0.0).all(-1)
        prob.update(pml_region=np.ones_like(prob["pml_region"]), pml_coef_alpha=al, pml_coef_abar=ab)

    def make(flags):
        s = gfb.Solver(prob, dirs=dirs, precision=prec, flags=flags | more.get("flags", 0))
        if more.get("all_pml"):
            assert s.info()["n_pml_node"] == prob["n_node"]
        return s

    compare(outputs(make, 0), outputs(make, gfb.FLAG_NO_GRAPH))


@pytest.mark.parametrize("prec", [gfb.FP32, gfb.FP64])
def test_replayed_batch_equals_one_launched_one_by_one(prec):
    probs = [problem(n=(5 + k, 5, 4), seed=6 + k) for k in range(3)]

    def make(flags):
        return gfb.BatchSolver(probs, dirs=[0, 1, 2], precision=prec, flags=flags, n_steps=[60, 23, 44])

    compare(outputs(make, 0), outputs(make, gfb.FLAG_NO_GRAPH))


def compare(a, b):
    for f in a[0]:
        for k in a[0][f]:
            np.testing.assert_array_equal(a[0][f][k], b[0][f][k], err_msg=f"field {f} {k}")
    for x, y in zip(a[1], b[1]):
        assert np.isfinite(x[0]).all() and np.abs(x[0]).max() > 0
        for p, q in zip(x, y):
            np.testing.assert_array_equal(p, q)


def test_runs_of_every_length():
    """Graphs of one to five steps, in any order, with and without snapshots."""
    prob = problem()
    for stride in (0, 4, 7):
        prob["snapshot_stride"] = stride
        out = []
        for flags in (0, gfb.FLAG_NO_GRAPH):
            s = gfb.Solver(prob, dirs=[0, 1, 2], precision=gfb.FP32, flags=flags)
            for n in (4, 1, 9, 3, 2, 5, 11, 0, 8):
                s.advance(n)
            assert s.step == 43
            s.synchronize()
            n_launch = s.info()["kernel_launches"]
            out.append((s.drain(), [s.state(f) for f in range(3)], n_launch))
            s.close()
        assert out[0][2] == out[1][2]
        compare(out[0], out[1])
