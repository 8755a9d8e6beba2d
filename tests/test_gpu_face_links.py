"""Face links of the pressure operator, bit for bit against the same formula in NumPy: floored
permeabilities, their harmonic mean, divided by the Pore end's viscosity (kept reciprocal, or a
plain division where the operands leave its range).

One product per colour of (i + 2j + 3k) mod 7 with the colour's indicator: a row's seven points
have seven colours, so the product's value is one coefficient, exactly.

Permeabilities from 1e-300 to 1e3 with zeros and values at and around the floor; viscosities of two
values, of every voxel its own, and below and above the range of the reciprocal; uint8 and uint16.
"""
import numpy as np
import pytest

from helpers import params

pytestmark = pytest.mark.gpu

AIR, PORE = 1, 2


def _links(lab, perm, visc, axis):
    """|link| from each voxel to the next along the axis"""
    lo = tuple(slice(None, -1) if a == axis else slice(None) for a in range(3))
    hi = tuple(slice(1, None) if a == axis else slice(None) for a in range(3))

    def link(s, n):
        ks = np.where(perm[s] < 1e-25, 1e-25, perm[s])
        kn = np.where(lab[n] == AIR, 1e-9, perm[n])
        kn = np.where(kn < 1e-25, 1e-25, kn)
        return ((2.0 * ks * kn) / (ks + kn)) / visc[s]

    with np.errstate(all="ignore"):
        return np.where(lab[lo] == PORE, link(lo, hi), np.where(lab[hi] == PORE, link(hi, lo), 0.0)), lo, hi


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("visc_kind", ["two", "own", "tiny", "huge"])
def test_links_match_formula(visc_kind, dtype):
    from leachingsim_gb300.runtime import Context
    shape = (9, 11, 35)
    rng = np.random.default_rng(17)
    lab = rng.choice(np.array([1, 2, 3, 4, 5], dtype), size=shape, p=[0.15, 0.5, 0.15, 0.1, 0.1])
    perm = 10.0 ** rng.uniform(-18, 3, shape)
    odd = rng.random(shape)
    perm[odd < 0.05] = 0.0
    perm[(odd >= 0.05) & (odd < 0.1)] = 1e-300
    perm[(odd >= 0.1) & (odd < 0.15)] = 1e-25
    perm[(odd >= 0.15) & (odd < 0.2)] = np.nextafter(1e-25, 0.0)
    visc = {"two": np.where(lab == AIR, 1.8e-5, 1e-3), "own": 10.0 ** rng.uniform(-6, 2, shape),
            "tiny": np.full(shape, 1e-95), "huge": np.full(shape, 1e95)}[visc_kind]
    g = Context(shape, label_bytes=np.dtype(dtype).itemsize, params=params())
    g.upload("label", lab)
    g.init_all()
    g.upload("permeability", perm)
    g.upload("viscosity", visc)
    g.pressure_setup(0.0)
    i, j, k = np.indices(shape)
    colour = (i + 2 * j + 3 * k) % 7
    col = np.empty((7,) + shape)
    for c in range(7):
        col[c] = g.pressure_apply((colour == c).astype(np.float64)).reshape(shape)
    g.close()
    for axis in range(3):
        ref, lo, hi = _links(lab, perm, visc, axis)
        for s, n in ((lo, hi), (hi, lo)):  # the row of either end, where it is a Pore row
            got = np.abs(np.take_along_axis(col[(slice(None),) + s], colour[n][None], 0)[0])
            rows = lab[s] == PORE
            np.testing.assert_array_equal(got[rows], ref[rows])
