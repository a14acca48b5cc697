"""gfb_get_info describes the element kernel that runs."""

import numpy as np
import pytest

import gfb

pytestmark = pytest.mark.gpu


def chain(ngll, n_cell):
    nn = ngll**3
    P = n_cell * nn
    return {"ngll": ngll, "n_cell": n_cell, "n_node": P, "ibool": np.arange(P),
            "dxi_dx": np.tile(np.eye(3).ravel(), P), "jacobian": np.ones(P), "lambda": np.ones(P), "mu": np.ones(P),
            "density": np.ones(P), "mass": np.ones(P), "dt": 0.01}


@pytest.mark.parametrize("ngll,dirs,prec,kernel,cells,per_sm", [
    (5, [0, 1, 2], gfb.FP32, 1, 2, 2),     # a warp of the plane kernel: two cells
    (5, [0], gfb.FP32, 1, 1, None), (5, [0, 1, 2], gfb.FP64, 1, 1, None),
    (3, [0, 1, 2], gfb.FP32, 1, 3, None), (4, [0, 1, 2], gfb.FP64, 1, 2, None), (6, [1], gfb.FP32, 1, 3, None),
])
def test_info_of_the_default_kernel(ngll, dirs, prec, kernel, cells, per_sm):
    import torch

    n_sm = torch.cuda.get_device_properties(0).multi_processor_count
    s = gfb.Solver(chain(ngll, 3), dirs=dirs, precision=prec, record=False)
    i = s.info()
    assert (i["elem_kernel"], i["cells_per_group"]) == (kernel, cells)
    assert i["elem_blocks"] % n_sm == 0 and i["elem_blocks"] > 0
    if per_sm:
        assert i["elem_blocks"] == per_sm * n_sm
    s.close()
    p = gfb.Solver(chain(ngll, 3), dirs=dirs, precision=prec, record=False, flags=gfb.FLAG_POINT_KERNEL)
    assert (p.info()["elem_kernel"], p.info()["cells_per_group"]) == (0, 0)
    p.close()
