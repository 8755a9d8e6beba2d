"""Transport systems with a few extreme rows: faces with fluxes of 1e6 among ordinary ones, so that some
rows take in far more than they give off and their links outweigh their diagonal 1e5 times. The
solve on the reduced system fails on most of these (FP32's rounding times the links of both halves); started
again on the whole system it converges. All layouts of the red-black halves (rows along k, j and
i; odd and even), both label widths, one and two species, theta 1 and 0.5.

The result is checked by its residual in FP64: A comes column by column from ls_transport_apply. With
rows of 1e6 and values near 1 the check's own rounding is below 1e-8 of the scaled right-hand side.
"""
import numpy as np
import pytest

from helpers import params
from leachingsim_gb300.runtime import Context

pytestmark = pytest.mark.gpu

CASES = [(shape, seed, which, lb, theta)
         for shape, seed in (((7, 4, 3), 0), ((2, 9, 5), 7), ((5, 6, 8), 4), ((5, 6, 8), 6))
         for which, lb, theta in ((3, 1, 1.0), (1, 2, 1.0), (2, 1, 1.0), (3, 2, 0.5))]
CASES += [((2, 9, 5), 0, 3, 2, 0.5), ((6, 12, 2), 12, 3, 1, 1.0), ((5, 9, 3), 11, 3, 1, 1.0), ((3, 30, 2), 0, 3, 1, 1.0),
          ((8, 5, 2), 1, 3, 1, 1.0), ((4, 6, 12), 2, 3, 2, 0.5)]


def scaled_residual(A, b, x):
    d = np.diag(A)
    return np.linalg.norm((A @ x - b) / d) / np.linalg.norm(b / d)


@pytest.mark.parametrize("shape,seed,which,label_bytes,theta", CASES)
def test_extreme_rows_converge(shape, seed, which, label_bytes, theta):
    rng = np.random.default_rng(seed)
    n, jk = int(np.prod(shape)), shape[1] * shape[2]
    lab = np.random.default_rng(seed).choice(np.array([1, 2, 3, 4, 5], np.uint8 if label_bytes == 1 else np.uint16),
                                             size=shape, p=[0.05, 0.6, 0.2, 0.1, 0.05])
    flux = [0.3 * rng.standard_normal(n) for _ in range(3)]
    for _ in range(10):
        flux[rng.integers(3)][rng.integers(n)] = 1e6 * rng.choice([-1, 1])
    old = {f: rng.random(n + jk) for f in ("conc", "acid")}

    def context(th):
        g = Context(shape, label_bytes=label_bytes, params=params(conc_rtol=1e-6, theta=th, alpha_transfer=0.05, Dpore_fac=0.8))
        g.upload("label", lab)
        for f, v in zip(("flux_x", "flux_y", "flux_z"), flux):
            g.upload(f, v)
        for f in old:
            g.upload(f, old[f], padded=True)
        return g

    g = context(theta)
    A = np.stack([g.transport_apply(1.0, e) for e in np.eye(n)], axis=1)
    half = np.zeros_like(A)  # the explicit half of the flow links
    if theta != 1.0:
        h = context(1.0)
        half = np.stack([h.transport_apply(1.0, e) for e in np.eye(n)], axis=1) - A
        h.close()
    for again in range(2):  # the second time with everything allocated
        for f in old:
            g.upload(f, old[f], padded=True)
        ok, ci, ai = g.transport(1.0, which)
        assert ok, (ci, ai)
        for bit, f in ((1, "conc"), (2, "acid")):
            got = g.download(f, padded=True).ravel()
            if not which & bit:
                np.testing.assert_array_equal(got, old[f])
                continue
            assert scaled_residual(A, old[f][:n] - half @ old[f][:n], got[jk:]) < 1e-6 + 1e-8
            np.testing.assert_array_equal(got[:jk], old[f][:jk])
    g.close()
