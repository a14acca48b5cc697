"""The default element kernels on meshes large enough that an item of work is a
cell group with all its wavefields and every warp takes at least two items, with a
remainder (below that they split an item by wavefield): the loop over the
wavefields on one copy of the geometry, the bulk stores of whole chunks, the second
fill of every stage.  Against assembly by colour, whose kernels share none of it.

Tolerance: the two sum the same products in another order.  A contraction and an
assembly add at most ~150 terms per value, so a step's force differs by at most ~150
eps of the largest term, and six steps from the same state add six such errors to
the velocity: 1e-12 (FP64, eps 1.1e-16) and 5.4e-5 (FP32, eps 6e-8) of the largest
value."""

import numpy as np
import pytest

import gfb

pytestmark = pytest.mark.gpu
TOL = {gfb.FP64: 1e-12, gfb.FP32: 5.4e-5}
SHARE = 20  # cells that share one more node: the long lists of touches


def chain(ngll, n_cell, seed):
    """Random cells in a chain, each sharing its last xi face with the next one's
    first; the middle point of every SHARE cells is one node."""
    rng = np.random.default_rng(seed)
    nn, n2 = ngll**3, ngll**2
    ib = np.arange(n_cell * nn).reshape(n_cell, nn)
    ib[1:, :n2] = ib[:-1, nn - n2:]
    ib[:, nn // 2] = ib[np.arange(n_cell) // SHARE * SHARE, nn // 2]
    ids, ib = np.unique(ib, return_inverse=True)
    P = n_cell * nn
    dxi = rng.uniform(-0.3, 0.3, (P, 9))
    dxi[:, [0, 4, 8]] += 1.0
    return {"ngll": ngll, "n_cell": n_cell, "n_node": len(ids), "ibool": ib.reshape(n_cell, nn), "dxi_dx": dxi,
            "jacobian": rng.uniform(0.5, 1.5, P), "lambda": rng.uniform(0.5, 1.5, P), "mu": rng.uniform(0.5, 1.5, P),
            "density": np.ones(P), "mass": rng.uniform(0.5, 1.5, P), "dt": 0.02, "snapshot_stride": 0,
            "src_cell_ids": np.array([n_cell - 1]), "src_weights": rng.uniform(0, 1, (1, nn)), "stf": np.ones(20),
            "nsteps": 20}


def cells_for_two_items(ngll, dirs, prec, **more):
    """A cell count that gives every group of threads two whole items and some a
    third, ending in an incomplete group."""
    s = gfb.Solver(chain(ngll, 2, 0), dirs=dirs, precision=prec, record=False, **more)
    i = s.info()
    s.close()
    groups = i["elem_blocks"] * (1 if ngll == 6 else 4)
    n = int(2.3 * groups * i["cells_per_group"])
    return n + 1 if i["cells_per_group"] == 1 or n % i["cells_per_group"] == 0 else n


def states(make, n_node, flags):
    s = make(flags)
    assert s.by_colour == (flags != 0)
    rng = np.random.default_rng(9)
    for f in range(s.n_field):
        s.set_state(f, 0, *(rng.standard_normal((n_node, 3)) for _ in range(3)))
    s.advance(6)
    out = [x for f in range(s.n_field) for x in s.state(f)]
    s.close()
    return out


def compare(make, n_node, prec):
    for p, q in zip(states(make, n_node, 0), states(make, n_node, gfb.FLAG_COLOUR)):
        assert np.isfinite(q).all() and np.abs(q).max() > 0
        assert np.abs(p - q).max() <= TOL[prec] * np.abs(q).max()


@pytest.mark.parametrize("prec", [gfb.FP64, gfb.FP32])
@pytest.mark.parametrize("ngll,fields", [(3, 2), (3, 3), (4, 2), (4, 3), (5, 1), (5, 2), (5, 3), (5, 6), (6, 2), (6, 3)])
def test_whole_items(ngll, fields, prec):
    dirs = [(f + 1) % 3 for f in range(fields)]

    def more(prob):
        if fields <= 3:
            return {}
        src = {k: prob[k] for k in ("src_cell_ids", "src_weights", "stf")}
        other = dict(src, src_cell_ids=np.array([prob["n_cell"] // 2]))
        return {"sources": [src, other], "field_source": [f // 3 for f in range(fields)]}

    n = cells_for_two_items(ngll, dirs, prec, **more(chain(ngll, 2, 0)))
    prob = chain(ngll, n, 7)
    compare(lambda flags: gfb.Solver(prob, dirs=dirs, precision=prec, record=False, flags=flags, **more(prob)),
            prob["n_node"], prec)


def test_twelve_wavefields():
    dirs = [0, 1, 2] * 4
    src = {"src_cell_ids": np.array([1]), "src_weights": np.ones((1, 125)), "stf": np.ones(20)}
    more = {"sources": [src], "field_source": [0] * 12}
    prob = chain(5, cells_for_two_items(5, dirs, gfb.FP32, **more), 3)
    compare(lambda flags: gfb.Solver(prob, dirs=dirs, precision=gfb.FP32, record=False, flags=flags, **more),
            prob["n_node"], gfb.FP32)


@pytest.mark.parametrize("ngll,dirs,prec", [(5, [0, 1, 2], gfb.FP32), (4, [0, 2], gfb.FP32), (5, [1, 2], gfb.FP64)])
def test_whole_items_of_a_batch(ngll, dirs, prec):
    """Three uneven models, of which one has taken its steps after two, another
    after four."""
    n = cells_for_two_items(ngll, dirs, prec)
    probs = [chain(ngll, m, 20 + m % 7) for m in (n // 2 + 3, n // 3, n // 4 + 1)]
    n_node = sum(p["n_node"] for p in probs)
    compare(lambda flags: gfb.BatchSolver(probs, dirs=dirs, precision=prec, flags=flags, n_steps=[20, 2, 4]), n_node, prec)
