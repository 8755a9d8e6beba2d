"""Transport on grids with short rows along k, where the red-black layout runs its rows along j or i:
the solve against a dense one, the implicit saturation against the oracle, and the bytes that the
solve's arrays take.

Row lengths where the virtual elements of a row along k outweigh 3/8 of the real ones (2-5, 9-11, 17) with the
long extent along j (axis 1) or along i (axis 0), even and odd, and the lengths next to them (6, 8,
12), which keep their rows along k. The dense system and its tolerance are those of
test_gpu_transport_reduced.py; with theta = 0.5 the right-hand side has the explicit half, old - A_ex old,
and A = 1/dt + theta F + R (F: the flow links' part, R: the exchange's), so that
A(theta = 0.5) and A(theta = 1) give F / 2 as their difference.
"""
import numpy as np
import pytest

from helpers import params, rel_l2
from leachingsim_gb300.runtime import Context

pytestmark = pytest.mark.gpu

SHAPES = [(3, 33, 2), (2, 40, 3), (5, 18, 4), (4, 16, 5), (2, 34, 9), (33, 2, 2), (40, 3, 3), (19, 4, 5), (26, 2, 4),
          (3, 24, 6), (3, 17, 8), (2, 16, 12)]


def _context(shape, label_bytes, seed, **kw):
    rng = np.random.default_rng(seed)
    n = int(np.prod(shape))
    lab = rng.choice([1, 2, 3, 4, 5, 7], size=shape, p=[0.1, 0.4, 0.25, 0.1, 0.1, 0.05])
    g = Context(shape, label_bytes=label_bytes, params=params(conc_rtol=1e-13, alpha_transfer=0.1, Dpore_fac=0.7, **kw))
    g.upload("label", lab.astype(np.uint8 if label_bytes == 1 else np.uint16))
    for f in ("flux_x", "flux_y", "flux_z"):
        g.upload(f, 0.3 * rng.standard_normal(n))
    old = {f: rng.random(n + shape[1] * shape[2]) for f in ("conc", "acid")}
    for f in old:
        g.upload(f, old[f], padded=True)
    return g, lab.ravel(), old


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("which,label_bytes,theta", [(1, 1, 1.0), (2, 2, 1.0), (3, 1, 1.0), (3, 2, 0.5)])
def test_matches_dense_solve(shape, which, label_bytes, theta):
    n, jk = int(np.prod(shape)), shape[1] * shape[2]
    g, lab, old = _context(shape, label_bytes, shape[2] * 10 + which, theta=theta)
    A = np.stack([g.transport_apply(1.0, e) for e in np.eye(n)], axis=1)
    half = np.zeros_like(A)  # the explicit half of the flow links
    if theta != 1.0:
        h, _, _ = _context(shape, label_bytes, shape[2] * 10 + which, theta=1.0)
        half = np.stack([h.transport_apply(1.0, e) for e in np.eye(n)], axis=1) - A
        h.close()
    ok, ci, ai = g.transport(1.0, which)
    assert ok, (ci, ai)
    for bit, f in ((1, "conc"), (2, "acid")):
        got = g.download(f, padded=True).ravel()
        if not which & bit:
            np.testing.assert_array_equal(got, old[f])
            continue
        x = np.linalg.solve(A, old[f][:n] - half @ old[f][:n])  # dt = 1
        assert rel_l2(got[jk:], x) < 1e-11, (f, rel_l2(got[jk:], x))
        np.testing.assert_array_equal(got[:jk], old[f][:jk])
    g.close()


@pytest.mark.parametrize("shape", [(6, 33, 2), (40, 3, 3), (5, 20, 9), (4, 24, 6)])
def test_implicit_saturation_matches_oracle(oracle_mod, shape):
    rng = np.random.default_rng(8)
    lab = rng.choice(np.array([1, 2, 3, 4], np.uint8), size=shape, p=[0.1, 0.6, 0.2, 0.1])
    p = params(use_implicit_saturation=1, sat_rtol=1e-13)
    o = oracle_mod.Oracle(shape, params=p, mode=oracle_mod.SOLVE_TIGHT, rtol=1e-14)
    o.load_labels(lab)
    o.init_all()
    g = Context(shape, params=p)
    g.upload("label", lab)
    g.init_all()
    for f in ("flux_x", "flux_y", "flux_z"):
        v = rng.normal(0, 1e-3, (shape[0] + 1,) + shape[1:])
        o.set(f, v, padded=True)
        g.upload(f, v, padded=True)
    okg, validg, _ = g.saturation_implicit(1.0)
    oko, valido, _ = o.saturation_implicit(1.0)
    assert bool(okg) == bool(oko) and bool(validg) == bool(valido)
    # flux terms of 1e-3 beside porosity / dt: a condition near 1
    assert rel_l2(g.download("saturation", padded=True), o.get("saturation", padded=True)) < 1e-11
    o.close()
    g.close()


@pytest.mark.parametrize("shape", [(300, 300, k) for k in (2, 3, 4, 5, 9, 10, 11, 17)] + [(300, 3, 301), (301, 302, 24)])
def test_bytes_of_the_solve(shape):
    """Rows of FP64 coefficients, two right-hand sides, a reciprocal, a kind (81 bytes a voxel), the
    change-tracking copies (label, three fluxes: 25), work list and bits (4.6), and links, residuals
    and vectors: 88 as whole rows, 64 and the planes at the ends of the 16 + 4 arrays (of 4-byte elements) as
    red-black halves."""
    n = int(np.prod(shape))
    g = Context(shape, params=params())
    before = g.device_bytes()
    rng = np.random.default_rng(1)
    g.upload("label", rng.choice(np.array([2, 3], np.uint8), size=shape))
    g.upload("conc", rng.random(shape))
    assert g.transport(1.0, 3)[0]
    plane = max(shape[1] * shape[2], shape[0] * shape[2]) + 64
    assert g.device_bytes() - before <= (81 + 25 + 4.7 + 88) * n + 20 * 4 * plane + 65536
    g.close()
