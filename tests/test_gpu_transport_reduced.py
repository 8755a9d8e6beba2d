"""The red-black reduced inner solve of the transport systems against a dense solve.

Row lengths around the layout's edges (a row of one colour holds ceil(K / 2) elements rounded up
to 4): single and odd elements, exactly one chunk, one element past it, several chunks. The
matrix comes column by column from ls_transport_apply (bit-exact with the oracle's assembled
operator, test_gpu_parity.py), the right-hand side is the implicit step's: the old value over
dt, or the old value on Precipitate rows. The solve stops at a Jacobi-scaled residual of 1e-13;
the scaled matrices are diagonally dominant with a condition number below 30 here (excess
1/dt = 1 of a diagonal of at most about 7 + |q|), so 1e-11 bounds the relative error.
"""
import numpy as np
import pytest

from helpers import params, rel_l2
from leachingsim_gb300.runtime import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 2, 3), (4, 3, 7), (3, 5, 8), (5, 4, 9), (2, 9, 16), (7, 3, 17),
                                   (4, 6, 33)])
@pytest.mark.parametrize("which,label_bytes", [(1, 1), (2, 2), (3, 1)])
def test_transport_matches_dense_solve(shape, which, label_bytes):
    rng = np.random.default_rng(shape[2] * 10 + which)
    n, jk = int(np.prod(shape)), shape[1] * shape[2]
    lab = rng.choice([1, 2, 3, 4, 5, 7], size=shape, p=[0.1, 0.4, 0.25, 0.1, 0.1, 0.05])
    g = Context(shape, label_bytes=label_bytes, params=params(conc_rtol=1e-13, alpha_transfer=0.1, Dpore_fac=0.7))
    g.upload("label", lab.astype(np.uint8 if label_bytes == 1 else np.uint16))
    for f in ("flux_x", "flux_y", "flux_z"):
        g.upload(f, 0.3 * rng.standard_normal(n))
    old = {f: rng.random(n + jk) for f in ("conc", "acid")}
    for f in old:
        g.upload(f, old[f], padded=True)
    A = np.stack([g.transport_apply(1.0, e) for e in np.eye(n)], axis=1)
    ok, ci, ai = g.transport(1.0, which)
    assert ok, (ci, ai)
    for bit, f in ((1, "conc"), (2, "acid")):
        got = g.download(f, padded=True).ravel()
        if not which & bit:
            np.testing.assert_array_equal(got, old[f])
            continue
        x = np.linalg.solve(A, old[f][:n])  # dt = 1
        assert rel_l2(got[jk:], x) < 1e-11, (f, rel_l2(got[jk:], x))
        np.testing.assert_array_equal(got[:jk], old[f][:jk])  # the plane below the solution keeps its values
    g.close()
