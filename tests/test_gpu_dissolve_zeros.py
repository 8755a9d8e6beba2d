"""Signs of zeros in the dissolution update: a face with acid -0.0 has the flux -0.0, and its share
of the loss, (-0.0) / flux_sum, is -0.0, so the face's acid becomes -0.0 - loss * (-0.0) = +0.0.
Compared as bits with the oracle's sequential sweep (an equality of values takes -0.0 for 0.0)."""
import numpy as np
import pytest

from helpers import params
from leachingsim_gb300.runtime import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("label_bytes", [1, 2])
@pytest.mark.parametrize("share", [0.05, 0.4, 1.0])  # of the voxels with acid -0.0
def test_zero_signs_match_oracle(oracle_mod, label_bytes, share):
    shape = (13, 9, 22)
    rng = np.random.default_rng(3)
    dtype = np.uint8 if label_bytes == 1 else np.uint16
    lab = rng.choice([1, 2, 3, 4, 5], size=shape, p=[0.05, 0.35, 0.25, 0.3, 0.05]).astype(dtype)
    acid = np.where(rng.random(shape) < share, -0.0, rng.random(shape))
    frac = np.where(lab >= 4, rng.uniform(0.05, 1.0, shape), 0.0).astype(np.float32)
    p = params(kreac=0.7, D=1.3, dx=0.9, time_scalar=3.0)
    o = oracle_mod.Oracle(shape, label_bytes=label_bytes, params=p, mode=oracle_mod.SOLVE_TIGHT)
    o.load_labels(lab)
    o.init_all()
    g = Context(shape, label_bytes=label_bytes, params=p)
    g.upload("label", lab)
    g.init_all()
    for f, v in (("frac", frac), ("acid", acid)):
        o.set(f, v)
        g.upload(f, v)
    for _ in range(2):
        assert o.dissolve(1.0)[0] == g.dissolve(1.0)[0]
        for f in ("acid", "conc", "precipitate"):
            np.testing.assert_array_equal(g.download(f).view(np.int64),
                                          np.ascontiguousarray(o.get(f), dtype=np.float64).view(np.int64), err_msg=f)
        np.testing.assert_array_equal(g.download("frac").view(np.int32),
                                      np.ascontiguousarray(o.get("frac"), dtype=np.float32).view(np.int32))
    g.close()
