"""Work lists of the change-tracked kernels with 32 words per warp, which grids above 9.96 million
voxels take: every lane owns a word, so the shuffles have no idle lanes. As
test_gpu_scan_words.py: after changes of single voxels the kept and re-evaluated values must be
bitwise those of a fresh context with the same state. 201 x 225 x 227 voxels: rows that are no multiple of
32, a last warp of 15 words and a last word of 27 bits."""
import numpy as np
import pytest

from helpers import params
from test_gpu_scan_words import PROPS, STATE, _evaluate

pytestmark = pytest.mark.gpu


def test_changed_voxels_match_fresh_evaluation():
    from leachingsim_gb300.runtime import Context
    shape = (201, 225, 227)
    rng = np.random.default_rng(9)
    lab = rng.choice(np.array([1, 2, 3, 4], np.uint8), size=shape, p=[0.1, 0.6, 0.2, 0.1])
    p = params()
    g = Context(shape, params=p)
    g.upload("label", lab)
    g.init_all()
    g.upload("acid", rng.random(shape))
    _evaluate(g)
    assert g.transport(1.0, 3)[0]
    I, J, K = shape
    where = [(i, j, k) for i in (0, I // 2, I - 1) for j in (0, J // 2, J - 1) for k in (0, K // 2, K - 1)]
    where += [tuple(int(rng.integers(0, n)) for n in shape) for _ in range(300)]
    idx = tuple(np.array(where).T)
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
    assert g.transport(1.0, 3)[0] and h.transport(1.0, 3)[0]
    for f in ("conc", "acid", "flux_x", "flux_y", "flux_z"):
        np.testing.assert_array_equal(g.download(f, padded=True), h.download(f, padded=True), err_msg=f)
    h.close()
    g.close()
