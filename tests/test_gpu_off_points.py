"""A point with mu <= 0 adds nothing, whatever else is stored at it
(element_cpu.cpp:42-43): collapsed and void cells leave infinities and NaN in
dxi_dx, lambda and the Jacobian there, and a void cell's own field may hold
anything.  Every element kernel against the same mesh with harmless values at
those points, bit for bit, and K_e u against the oracle.

Tolerance against the oracle: a value is a sum of at most ~4,000 products
(3 directions of a contraction of contractions, ngll^2 terms each), so the
relative rounding is below 4000 eps / 2: 5e-13 (FP64), 2.4e-4 (FP32) of the
largest value."""

import numpy as np
import pytest

import gfb
import oracle

pytestmark = pytest.mark.gpu

BAD = (np.inf, -np.inf, np.nan, 1e300)


def mesh_with_off_points(ngll, n_cell, seed, bad):
    """A chain of cells; a tenth of their points off, the last cell wholly."""
    rng = np.random.default_rng(seed)
    nn, n2 = ngll**3, ngll**2
    ib = np.arange(n_cell * nn).reshape(n_cell, nn)
    for e in range(1, n_cell):
        ib[e, :n2] = ib[e - 1, nn - n2:]
    ids, ib = np.unique(ib, return_inverse=True)
    ib = ib.reshape(n_cell, nn)
    P = n_cell * nn
    dxi = rng.uniform(-0.3, 0.3, (P, 9))
    dxi[:, [0, 4, 8]] += 1.0
    jac, lam, mu = (rng.uniform(0.5, 1.5, P) for _ in range(3))
    off = rng.random(P) < 0.1
    off[-nn:] = True
    mu[off] = -rng.integers(0, 2, off.sum()).astype(float)  # 0 and -1
    weights = rng.uniform(0, 1, (1, nn))
    if bad:
        k = rng.integers(0, len(BAD), (off.sum(), 11))
        v = np.array(BAD)[k]
        dxi[off], jac[off], lam[off] = v[:, :9], v[:, 9], v[:, 10]
    return {"ngll": ngll, "n_cell": n_cell, "n_node": len(ids), "ibool": ib, "dxi_dx": dxi, "jacobian": jac,
            "lambda": lam, "mu": mu, "density": np.ones(P), "mass": np.full(P, 1.0), "dt": 0.02,
            "snapshot_stride": 0, "src_cell_ids": np.array([0]), "src_weights": weights,
            "stf": np.ones(20)}


def final(prob, dirs, prec, flags=0, variant=None):
    s = gfb.Solver(prob, dirs=dirs, precision=prec, flags=flags, record=False)
    if variant is not None:
        s.select_element_kernel(variant)
    rng = np.random.default_rng(9)
    for f in range(len(dirs)):
        s.set_state(f, 0, *(rng.standard_normal((prob["n_node"], 3)) for _ in range(3)))
    s.advance(5)
    out = [x for f in range(len(dirs)) for x in s.state(f)]
    s.close()
    return out


@pytest.mark.parametrize("prec", [gfb.FP64, gfb.FP32])
@pytest.mark.parametrize("ngll,n_cell,dirs", [(3, 7, [0, 1, 2]), (4, 5, [1]), (5, 9, [0, 1, 2]), (5, 6, [2]), (6, 3, [0, 2])])
def test_points_that_add_nothing_add_nothing(ngll, n_cell, dirs, prec):
    good, bad = (mesh_with_off_points(ngll, n_cell, 5, b) for b in (False, True))
    kernels = [{}, {"flags": gfb.FLAG_POINT_KERNEL}, {"flags": gfb.FLAG_FUSED_NODE}]
    if prec == gfb.FP32 and ngll == 5:
        kernels += [{"variant": v} for v in (1, 2, 3)]
    for k in kernels:
        a, b = final(good, dirs, prec, **k), final(bad, dirs, prec, **k)
        for x, y in zip(a, b):
            assert np.isfinite(x).all() and np.abs(x).max() > 0
            np.testing.assert_array_equal(x, y, err_msg=str(k))


@pytest.mark.parametrize("prec,tol", [(gfb.FP64, 5e-13), (gfb.FP32, 2.4e-4)])
@pytest.mark.parametrize("ngll", [3, 4, 5, 6])
def test_residual_of_cells_with_void_points(ngll, prec, tol):
    n, nn = 6, ngll**3
    p = mesh_with_off_points(ngll, n, 8, True)
    u = np.random.default_rng(3).standard_normal((n * nn, 3))
    u[-nn:] = np.nan  # the void cell's own field
    r = gfb.element_residual(p["dxi_dx"], p["jacobian"], p["lambda"], p["mu"], u, ngll, prec).reshape(-1, 3)
    ref = oracle.element_residual(p["dxi_dx"], p["jacobian"], p["lambda"], p["mu"], u, ngll).reshape(-1, 3)
    assert np.isfinite(ref).all() and (ref[-nn:] == 0.0).all()
    assert np.isfinite(r).all() and (r[-nn:] == 0.0).all()
    assert np.abs(r - ref).max() <= tol * np.abs(ref).max()
