"""Work lists of the change-tracked kernels where their bit words meet the ends of rows, planes and
the box, with one and with several words per warp: after changes of single voxels (the corners, the
ends of rows and planes, random others) the kept and re-evaluated values must be bitwise those of a
fresh context with the same state.

Shapes: rows shorter than a word (several ends per word), of two voxels (the fewest), of exactly one and of one
more than one word; a box smaller than a word; boxes of 2 and of 16 words per warp.
"""
import numpy as np
import pytest

from helpers import params, small_grf

pytestmark = pytest.mark.gpu

STATE = ["label", "frac", "precipitate", "saturation", "pressure", "conc", "acid", "flux_x", "flux_y", "flux_z"]
PROPS = ["permeability", "viscosity", "rel_perm", "cap_pressure"]


def _evaluate(g):
    g.props()
    g.pressure_setup(5.0)
    g.flux()


@pytest.mark.parametrize("shape", [(5, 7, 3), (6, 40, 2), (3, 3, 3), (9, 6, 32), (7, 5, 33), (12, 11, 70),
                                   (64, 100, 101), (170, 160, 190)])
def test_changed_voxels_match_fresh_evaluation(shape):
    from leachingsim_gb300.runtime import Context
    rng = np.random.default_rng(sum(shape))
    lab = small_grf(shape, seed=3) if min(shape) > 8 else rng.choice(
        np.array([1, 2, 3, 4], np.uint8), size=shape, p=[0.1, 0.6, 0.2, 0.1])
    p = params()
    g = Context(shape, params=p)
    g.upload("label", lab)
    g.init_all()
    g.upload("acid", rng.uniform(0.0, 1.0, shape))
    _evaluate(g)
    okg = g.transport(1.0, 3)[0]
    assert okg
    I, J, K = shape
    ends = [(i, j, k) for i in (0, I // 2, I - 1) for j in (0, J // 2, J - 1) for k in (0, K // 2, K - 1)]
    some = [tuple(int(rng.integers(0, n)) for n in shape) for _ in range(12)]
    for group in (ends[::2], ends[1::2], some):
        idx = tuple(np.array(group).T)
        sat, label = g.download("saturation"), g.download("label")
        sat[idx] = sat[idx] * 0.75 + 0.05
        label[idx] = np.where(label[idx] == 2, 3, 2)
        g.upload("saturation", sat)
        g.upload("label", label)
        h = Context(shape, params=p)
        for f in STATE:
            h.upload(f, g.download(f, padded=True), padded=True)
        _evaluate(g)
        _evaluate(h)
        x = rng.normal(size=lab.size)
        np.testing.assert_array_equal(g.pressure_apply(x), h.pressure_apply(x))
        np.testing.assert_array_equal(g.pressure_rhs(), h.pressure_rhs())
        for f in PROPS + ["flux_x", "flux_y", "flux_z"]:
            np.testing.assert_array_equal(g.download(f, padded=True), h.download(f, padded=True), err_msg=f)
        assert g.transport(1.0, 3)[0] == h.transport(1.0, 3)[0]
        for f in ("conc", "acid", "flux_x", "flux_y", "flux_z"):
            np.testing.assert_array_equal(g.download(f, padded=True), h.download(f, padded=True), err_msg=f)
        h.close()
    g.close()
