"""The coarse multigrid levels run as one launch (k_mg_fused) against the same cycle as one
kernel per step (LS_MG_TAIL_CELLS=0): the same operations in the same order and the same
reduction trees, so the same iterations and the same pressure bit for bit.

Shapes: a hierarchy of one coarse level; one that fits one block; a cluster with a K-cycle level of
8,736 cells (just below the bound, odd extents) and the small levels in its first block; a level
of 3,876 cells below two that keep their kernels; a flat box whose slabs would be thinner than a
plane (its first levels keep their kernels). Both inner precisions, graphs on and off.
"""
import numpy as np
import pytest

from leachingsim_gb300 import _abi
from leachingsim_gb300.geometry import grf_geometry

pytestmark = pytest.mark.gpu


def _solve(monkeypatch, lab, cells, graphs, solver):
    import torch
    from leachingsim_gb300.runtime import Context
    monkeypatch.setenv("LS_MG_GRAPHS", graphs)
    if cells is None:
        monkeypatch.delenv("LS_MG_TAIL_CELLS", raising=False)
    else:
        monkeypatch.setenv("LS_MG_TAIL_CELLS", str(cells))
    ctx = Context(lab.shape, params=_abi.default_params(press_rtol=1e-10, press_solver=solver))
    ctx.upload("label", lab)
    ctx.init_all()
    ctx.pressure_setup(3600.0)
    ok, info = ctx.pressure_solve_start(torch.zeros(lab.shape, device="cuda"), 0.0)
    p = ctx.download("pressure", padded=True).copy()
    ctx.close()
    return ok, info["iterations"], info["outer_iterations"], p


@pytest.mark.parametrize("shape", [(6, 8, 8), (24, 20, 22), (61, 83, 101), (150, 96, 130), (4, 300, 41)])
@pytest.mark.parametrize("solver", [_abi.PRESS_MIXED, _abi.PRESS_FP64])
def test_fused_levels_match_level_kernels(monkeypatch, shape, solver):
    lab, _ = grf_geometry(shape, porosity=0.4, corr_len=2.0, mineral_fraction=0.1, seed=5, air_inlet=True)
    ref = _solve(monkeypatch, lab, 0, "0", solver)
    for graphs in ("0", "1"):
        got = _solve(monkeypatch, lab, None, graphs, solver)
        assert got[:3] == ref[:3]
        assert np.array_equal(got[3], ref[3])
