"""The gather element kernel and the assembling node passes against assembly
by colour (GFB_FLAG_POINT_KERNEL): the same steps on meshes whose cells are
not a multiple of a warp's, with the node shared by many cells that needs the
long touch list, in every kernel shape.

Tolerance: the two sum the same products in another order.  A contraction and
an assembly add at most ~100 terms per value, so a step's force differs by at
most ~100 eps of the largest term, and six steps from the same state add six
such errors to the velocity: 1e-12 (FP64, eps 1.1e-16) and 4e-5 (FP32, eps 6e-8)
relative to the largest value leave room for the growth of the terms."""

import numpy as np
import pytest

import gfb

pytestmark = pytest.mark.gpu


def fan(ngll, n_cell, shared, seed, cpml=False):
    """Random cells in a chain: each shares its last xi face with the next
    one's first, and point ``shared`` of every cell is one node."""
    rng = np.random.default_rng(seed)
    nn, n2 = ngll**3, ngll**2
    ib = np.empty((n_cell, nn), dtype=np.int64)
    n_node = 0
    for e in range(n_cell):
        ib[e] = n_node + np.arange(nn)
        n_node += nn
        if e:
            ib[e, :n2] = ib[e - 1, nn - n2:]
        if e:
            ib[e, shared] = ib[0, shared]
    ids, ib = np.unique(ib, return_inverse=True)
    ib = ib.reshape(n_cell, nn)
    P = n_cell * nn
    dxi = rng.uniform(-0.3, 0.3, (P, 9))
    dxi[:, [0, 4, 8]] += 1.0
    mu = rng.uniform(0.5, 1.5, P)
    mu[rng.random(P) < 0.02] = 0.0  # points that add nothing
    prob = {"ngll": ngll, "n_cell": n_cell, "n_node": len(ids), "ibool": ib, "dxi_dx": dxi,
            "jacobian": rng.uniform(0.5, 1.5, P), "lambda": rng.uniform(0.5, 1.5, P), "mu": mu,
            "density": np.ones(P), "mass": rng.uniform(0.5, 1.5, P), "dt": 0.02, "snapshot_stride": 0,
            "src_cell_ids": np.array([n_cell - 1]), "src_weights": rng.uniform(0, 1, (1, nn)),
            "stf": np.ones(20)}
    if cpml:
        prob["pml_region"] = (np.arange(n_cell) % 2).astype(np.int32)
        prob["pml_coef_alpha"] = rng.uniform(0.1, 0.4, (P, 9))
        prob["pml_coef_abar"] = rng.uniform(-0.2, 0.2, (P, 5))
    return prob


def states(prob, dirs, prec, flags):
    s = gfb.Solver(prob, dirs=dirs, precision=prec, flags=flags, record=False)
    rng = np.random.default_rng(9)
    for f in range(len(dirs)):
        s.set_state(f, 0, *(rng.standard_normal((prob["n_node"], 3)) for _ in range(3)))
    s.advance(6)
    out = [s.state(f) for f in range(len(dirs))]
    s.close()
    return out


@pytest.mark.parametrize("prec,tol", [(gfb.FP64, 1e-12), (gfb.FP32, 4e-5)])
@pytest.mark.parametrize("ngll,n_cell,dirs", [(3, 1, [0]), (3, 7, [0, 1, 2]), (4, 5, [2, 0]), (5, 1, [1]),
                                              (5, 1, [2, 1, 0]),
                                              (5, 13, [0, 1, 2]), (5, 37, [2]), (6, 2, [0]), (6, 7, [1, 2, 0])])
def test_gather_assembly_equals_assembly_by_colour(ngll, n_cell, dirs, prec, tol):
    for cpml in (False, True):
        prob = fan(ngll, n_cell, (ngll**3) // 2, 100 * ngll + n_cell, cpml)
        flags = gfb.FLAG_CELL_PML if cpml else 0
        a = states(prob, dirs, prec, flags)
        b = states(prob, dirs, prec, flags | gfb.FLAG_POINT_KERNEL)
        for x, y in zip(a, b):
            for p, q in zip(x, y):
                assert np.isfinite(q).all() and np.abs(q).max() > 0
                assert np.abs(p - q).max() <= tol * np.abs(q).max()
