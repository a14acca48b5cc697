"""Assembly by colour, what a solver falls back to where the contribution
buffer does not fit on the device, taken with GFB_FLAG_COLOUR: every call against
the default assembly on the same mesh.

Tolerance: the two sum the same products in another order.  A value of a step's
force is a sum of at most ~4 ngll^2 + 8 such terms, so 40 steps from the same state
differ by at most ~40 * 150 eps relative to the largest value: 7e-13 (FP64), 3.6e-4
(FP32)."""

import numpy as np
import pytest

import gfb
from gfb import mesh

pytestmark = pytest.mark.gpu
TOL = {gfb.FP64: 7e-13, gfb.FP32: 3.6e-4}


def problem(order=4, n=(6, 5, 4), seed=4, cpml=True, stride=10):
    spec = mesh.MeshSpec(nx=n[0], ny=n[1], nz=n[2], dx=500.0, dy=500.0, dz=500.0, order=order, jitter=0.05, seed=seed,
                         pml={f: 1 for f in ("xmin", "xmax", "ymin", "ymax", "zmax")})
    return mesh.build_problem(spec, mesh.seeded_layers(seed, n[2] * 500.0), np.asarray([1700.0, 1300.0, 700.0]),
                              nsteps=60, snapshot_stride=stride, record_depth_max_m=500.0, with_cpml=cpml)


def kick(s, n_node, steps=40):
    rng = np.random.default_rng(2)
    for f in range(s.n_field):
        s.set_state(f, 0, *(rng.standard_normal((n_node, 3)) * k for k in (1e-3, 1e-1, 1.0)))
    out = s.run(steps)
    return out, [s.state(f) for f in range(s.n_field)]


def close(a, b, tol):
    for f in a[0]:
        np.testing.assert_array_equal(a[0][f]["steps"], b[0][f]["steps"])
        for k in ("strain", "u", "v", "a"):
            x, y = a[0][f][k], b[0][f][k]
            assert np.isfinite(y).all() and np.abs(y).max() > 0
            assert np.abs(x - y).max() <= tol * np.abs(y).max(), (f, k)
    for x, y in zip(a[1], b[1]):
        for p, q in zip(x, y):
            assert np.abs(p - q).max() <= tol * np.abs(q).max()


@pytest.mark.parametrize("prec", [gfb.FP64, gfb.FP32])
@pytest.mark.parametrize("order,dirs,cpml", [(2, [0, 1, 2], True), (3, [2], True), (4, [0, 1, 2], True), (4, [1, 0], False),
                                             (5, [0, 1, 2], True), (5, [1], False)])
def test_by_colour_equals_the_default(order, dirs, cpml, prec):
    prob = problem(order, cpml=cpml)
    a = gfb.Solver(prob, dirs=dirs, precision=prec)
    b = gfb.Solver(prob, dirs=dirs, precision=prec, flags=gfb.FLAG_COLOUR)
    assert not a.by_colour and b.by_colour
    contributions = prob["n_cell"] * (order + 1) ** 3 * len(dirs) * 3 * (8 if prec == gfb.FP64 else 4)
    assert a.info()["device_bytes"] - b.info()["device_bytes"] >= contributions
    close(kick(b, prob["n_node"]), kick(a, prob["n_node"]), TOL[prec])
    # a checkpoint of the one is refused by the other (the flags differ), and
    # continues bit for bit in a solver built alike
    with pytest.raises(gfb.GfbError, match="built like this one"):
        b.restore(a.checkpoint())
    c = gfb.Solver(prob, dirs=dirs, precision=prec, flags=gfb.FLAG_COLOUR)
    c.restore(b.checkpoint())
    for s in (b, c):
        s.advance(7)
    for f in range(len(dirs)):
        for p, q in zip(b.state(f), c.state(f)):
            np.testing.assert_array_equal(p, q)
    for s in (a, b, c):
        s.close()


def test_sources_by_colour():
    prob = problem()
    ids, w = np.asarray(prob["src_cell_ids"]), np.asarray(prob["src_weights"])
    sets = [{"src_cell_ids": ids, "src_weights": w, "stf": prob["stf"]},
            {"src_cell_ids": ids + 1, "src_weights": w, "stf": 0.5 * np.asarray(prob["stf"])}]

    def make(flags):
        return gfb.Solver(prob, dirs=[0, 1, 2] * 2, precision=gfb.FP32, sources=sets, field_source=[0] * 3 + [1] * 3, flags=flags)

    a, b = make(0), make(gfb.FLAG_COLOUR)
    assert b.by_colour
    close(kick(b, prob["n_node"]), kick(a, prob["n_node"]), TOL[gfb.FP32])
    a.close()
    b.close()


@pytest.mark.parametrize("prec", [gfb.FP64, gfb.FP32])
def test_batch_by_colour(prec):
    probs = [problem(n=(5 + k, 5, 4), seed=6 + k) for k in range(3)]
    n_node = sum(p["n_node"] for p in probs)

    def make(flags):
        return gfb.BatchSolver(probs, dirs=[0, 2], precision=prec, flags=flags, n_steps=[60, 17, 29])

    a, b = make(0), make(gfb.FLAG_COLOUR)
    assert b.by_colour
    close(kick(b, n_node), kick(a, n_node), TOL[prec])
    a.close()
    b.close()


def test_selected_kernels_report_their_assembly():
    prob = problem()
    s = gfb.Solver(prob, dirs=[0], precision=gfb.FP32)
    for variant, colour in ((0, False), (1, True), (-1, True), (0, False)):
        s.select_element_kernel(variant)
        assert s.by_colour == colour
    s.close()
    for flags in (gfb.FLAG_POINT_KERNEL, gfb.FLAG_FUSED_NODE):
        s = gfb.Solver(prob, dirs=[0], precision=gfb.FP64, flags=flags)
        assert s.by_colour
        s.close()


@pytest.mark.parametrize("order,fields", [(2, 1), (2, 3), (3, 2), (4, 3), (4, 6), (4, 9), (4, 12), (5, 3)])
def test_by_colour_runs_the_line_kernel(order, fields):
    """Every FP32 shape has it; the point kernel takes up to twice the time."""
    prob = problem(order)
    ids, w = np.asarray(prob["src_cell_ids"]), np.asarray(prob["src_weights"])
    src = {"src_cell_ids": ids, "src_weights": w, "stf": prob["stf"]}
    more = dict(sources=[src], field_source=[0] * fields) if fields > 3 else {}

    def make(flags):
        return gfb.Solver(prob, dirs=[f % 3 for f in range(fields)], precision=gfb.FP32, flags=flags, **more)

    a, b = make(0), make(gfb.FLAG_COLOUR)
    assert b.by_colour and b.info()["elem_kernel"] == 1 and b.info()["cells_per_group"] >= 1
    close(kick(b, prob["n_node"]), kick(a, prob["n_node"]), TOL[gfb.FP32])
    a.close()
    b.close()


@pytest.mark.parametrize("prec", [gfb.FP64, gfb.FP32])
@pytest.mark.parametrize("ngll,n", [(3, 18518), (3, 18519), (4, 2), (5, 3999), (5, 4000), (6, 2315)])
def test_element_residual_by_either_assembly(ngll, n, prec):
    """On both sides of the size where the call changes its assembly: the same
    cells one by one (K_e is linear, so the sums differ by rounding alone)."""
    rng = np.random.default_rng(ngll)
    P = n * ngll**3
    dxi = rng.uniform(-0.3, 0.3, (P, 9))
    dxi[:, [0, 4, 8]] += 1.0
    a = [rng.uniform(0.5, 1.5, P) for _ in range(3)]
    u = rng.standard_normal((P, 3))
    r = gfb.element_residual(dxi, *a, u, ngll, prec).reshape(n, -1)
    k = np.r_[0, n // 2, n - 1]
    q = (k[:, None] * ngll**3 + np.arange(ngll**3)).ravel()
    one = gfb.element_residual(dxi[q], *(x[q] for x in a), u[q], ngll, prec).reshape(len(k), -1)
    assert np.isfinite(r).all()
    assert np.abs(r[k] - one).max() <= TOL[prec] * np.abs(one).max()
