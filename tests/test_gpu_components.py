"""Strong components of the pressure multigrid (runs along k, then hooks between runs) against
scipy's labelling of the same links.

The level-1 owner of each 2x2x2 block is the component with most members in it (ties: the smallest
id), ids being the smallest voxel index of a component, so the labels are checked through
ls_pressure_mg_level. All Pore voxels carry the same permeability here, so every link between two
of them is strong. Row lengths around the warp's 32 cells, runs that cross warps and rows, thin
grids.
"""
import numpy as np
import pytest

from helpers import params
from leachingsim_gb300.runtime import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 8, 31), (9, 10, 32), (8, 9, 33), (12, 6, 70), (4, 40, 5), (20, 16, 64)])
@pytest.mark.parametrize("porosity", [0.3, 0.6])
def test_level_one_owners_match_scipy(shape, porosity):
    import torch
    from scipy import ndimage
    rng = np.random.default_rng(shape[2])
    lab = np.where(rng.random(shape) < porosity, 2, 3).astype(np.uint8)
    lab[0] = 1
    g = Context(shape, params=params(press_rtol=1e-6))
    g.upload("label", lab)
    g.init_all()
    g.pressure_setup(3600.0)
    g.pressure_solve_start(torch.zeros(shape, device="cuda"), 0.0)
    got = g.mg_level(1)["comp"]
    g.close()
    # every Pore voxel is an unknown: one with a Pore or Air neighbour has a link above the floor,
    # an isolated one (links of ~1e-22 to Rock) has a floored diagonal and is none
    pore = lab == 2
    fluid = np.pad(lab <= 2, 1)
    near = sum(np.roll(fluid, d, ax) for ax in range(3) for d in (1, -1))[1:-1, 1:-1, 1:-1] > 0
    unknown = pore & near
    idx = np.arange(lab.size).reshape(shape)
    comp, n = ndimage.label(unknown)
    root = ndimage.minimum(idx, comp, np.arange(1, n + 1)).astype(np.int64)
    ids = np.where(unknown, np.concatenate([[-1], root])[comp], -1)
    want = np.full(tuple((s + 1) // 2 for s in shape), -1)
    for c in np.ndindex(want.shape):
        v = ids[tuple(slice(2 * q, 2 * q + 2) for q in c)].ravel()
        v = v[v >= 0]
        if v.size:
            u, m = np.unique(v, return_counts=True)
            want[c] = u[m == m.max()].min()
    np.testing.assert_array_equal(got, want)
