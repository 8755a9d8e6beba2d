"""Transport solves to a tolerance near the unit roundoff: the rounding of the residual pass must
not keep its norm above what FP64 reaches (the order of its terms decides the size of the partial
sums, most at long time steps, where 1/dt is a small part of the diagonal)."""
import numpy as np
import pytest

from helpers import params
from leachingsim_gb300.runtime import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(32, 40, 40), (21, 30, 33)])  # even and odd rows
@pytest.mark.parametrize("dt", [1.0, 30.0, 1e3, 1e6])
def test_converges_near_unit_roundoff(shape, dt):
    rng = np.random.default_rng(5)
    n, jk = int(np.prod(shape)), shape[1] * shape[2]
    lab = np.random.default_rng(4).choice(np.array([1, 2, 3, 4, 5], np.uint8), size=shape, p=[0.05, 0.5, 0.3, 0.1, 0.05])
    g = Context(shape, params=params(conc_rtol=1.5e-16, alpha_transfer=0.05, Dpore_fac=0.8))
    g.upload("label", lab)
    for f in ("flux_x", "flux_y", "flux_z"):
        g.upload(f, 0.1 * rng.standard_normal(n))
    for f in ("conc", "acid"):
        g.upload(f, 0.5 + 0.1 * np.sin(np.arange(n + jk) * 1e-3), padded=True)
    ok, ci, ai = g.transport(dt, 3)
    assert ok, (ci, ai)
    g.close()
