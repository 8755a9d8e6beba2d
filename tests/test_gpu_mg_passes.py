"""The finest-level passes on pairs of cells (FP32, even extent along k): the same pressure as the
FP64 inner solver, whose passes take single cells, and the same iterations as the FP32 passes on
single cells take on the box with one more solid plane at the end of k (odd extent).

Tolerances: both pressures have a residual below 1e-12 of the right-hand side and the condition of
these operators is below 1e5 (1e2 voxels across, squared, times the spread of the links), so they
agree to 1e-7 of the largest. The boxes end in two solid planes, so a third one changes the system
only behind them and each inner solve may end one iteration earlier or later.

Shapes: one coarse level; odd extents over i and j, so that the last blocks hold one plane or row;
a flat box; rows longer than a block of threads; several level kernels above the fused ones.
"""
import numpy as np
import pytest

from leachingsim_gb300 import _abi
from leachingsim_gb300.geometry import grf_geometry

pytestmark = pytest.mark.gpu


def _solve(lab, solver):
    import torch
    from leachingsim_gb300.runtime import Context
    ctx = Context(lab.shape, params=_abi.default_params(press_rtol=1e-12, press_solver=solver))
    ctx.upload("label", lab)
    ctx.init_all()
    ctx.pressure_setup(3600.0)
    ok, info = ctx.pressure_solve_start(torch.zeros(lab.shape, device="cuda"), 0.0)
    p = ctx.download("pressure").copy()
    ctx.close()
    assert ok
    return info["iterations"], info["outer_iterations"], p


@pytest.mark.parametrize("cells", [None, "0"])
@pytest.mark.parametrize("shape", [(6, 8, 8), (25, 31, 34), (4, 300, 42), (40, 9, 600), (90, 71, 64)])
def test_pairs_match_single_cells(monkeypatch, shape, cells):
    if cells is not None:
        monkeypatch.setenv("LS_MG_TAIL_CELLS", cells)
    lab, _ = grf_geometry(shape, porosity=0.4, corr_len=2.0, mineral_fraction=0.1, seed=7, air_inlet=True)
    lab[2:, :, -2:] = _abi.ROCK
    its, outer, p = _solve(lab, _abi.PRESS_MIXED)
    _, _, p64 = _solve(lab, _abi.PRESS_FP64)
    assert np.abs(p - p64).max() <= 1e-7 * np.abs(p64).max()
    odd = np.ascontiguousarray(np.concatenate([lab, lab[:, :, -1:]], axis=2))
    its_odd, outer_odd, _ = _solve(odd, _abi.PRESS_MIXED)
    assert abs(its - its_odd) <= max(outer, outer_odd)
