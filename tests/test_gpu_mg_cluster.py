"""The fused coarse multigrid levels (k_mg_fused) on a cluster of 8 blocks, the form for devices
that cannot hold 16, and without a cluster (LS_MG_CLUSTER): other slab sizes, other levels refused
for thin slabs or shared memory, other shares of the FP64 coarsest level, the same operations in the same
order. Iterations and pressure must be those of the level kernels bit for bit.

Shapes as in test_gpu_mg_fused.py (one coarse level; one block; a K-cycle level of 8,736 cells; a level
of 3,876 cells; a flat box with thin slabs) and 26x60x42: its level of 8,190 cells has planes of 630,
which a slab of 1,024 (8 blocks) holds and one of 512 (16) does not.
"""
import numpy as np
import pytest

from leachingsim_gb300 import _abi
from leachingsim_gb300.geometry import grf_geometry
from test_gpu_mg_fused import _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(6, 8, 8), (24, 20, 22), (61, 83, 101), (150, 96, 130), (4, 300, 41), (26, 60, 42)])
@pytest.mark.parametrize("solver", [_abi.PRESS_MIXED, _abi.PRESS_FP64])
def test_clusters_match_level_kernels(monkeypatch, shape, solver):
    lab, _ = grf_geometry(shape, porosity=0.4, corr_len=2.0, mineral_fraction=0.1, seed=5, air_inlet=True)
    ref = _solve(monkeypatch, lab, 0, "0", solver)
    for blocks, graphs in ((16, "1"), (8, "0"), (8, "1"), (0, "1")):
        monkeypatch.setenv("LS_MG_CLUSTER", str(blocks))
        got = _solve(monkeypatch, lab, 9000, graphs, solver)  # the cluster's levels in FP32 too
        assert got[:3] == ref[:3], blocks
        assert np.array_equal(got[3], ref[3]), blocks


@pytest.mark.parametrize("shape,solver,fused", [((40, 40, 40), _abi.PRESS_FP64, False),   # 125 cells
                                                ((48, 48, 48), _abi.PRESS_FP64, False),   # 216
                                                ((48, 52, 48), _abi.PRESS_FP64, True),    # 252
                                                ((64, 64, 64), _abi.PRESS_FP64, True),    # 512
                                                ((40, 40, 40), _abi.PRESS_MIXED, True)])
def test_default_rule(monkeypatch, shape, solver, fused):
    """Which levels run fused by default (FP64: by the size of the coarsest level), by the launches of a
    solve; the results are those of the level kernels."""
    lab, _ = grf_geometry(shape, porosity=0.4, corr_len=2.0, mineral_fraction=0.1, seed=5, air_inlet=True)
    count = []
    for cells in (None, 0):
        r, n = _counted(monkeypatch, lab, cells, solver)
        count.append(n)
        if cells is None:
            got = r
    assert got[:3] == r[:3] and np.array_equal(got[3], r[3])
    assert (count[0] < count[1]) == fused and (fused or count[0] == count[1])


def _counted(monkeypatch, lab, cells, solver):
    from leachingsim_gb300 import runtime as rt
    launches, close = [], rt.Context.close
    monkeypatch.setattr(rt.Context, "close", lambda self: (launches.append(self.launches()), close(self))[1])
    r = _solve(monkeypatch, lab, cells, "0", solver)
    monkeypatch.setattr(rt.Context, "close", close)
    return r, launches[0]
