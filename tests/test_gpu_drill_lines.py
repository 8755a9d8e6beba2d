"""Drilled centre lines with points exactly between two voxels, where the integer steps hand the
point to its floating-point form: whole result equal to the oracle's numpy.linspace and round.

A line of n steps over offsets with an odd multiple of n/2 meets such points (offset 1 of 2 steps, 3
of 6, 5 of 10, 20 of 40); squares and non-squares for the number of steps, both directions, and a
line longer than 4,096 voxels, whose length is a double square root.
"""
import numpy as np
import pytest

from oracle import geometry_oracle as go

pytestmark = pytest.mark.gpu

OFFSETS = [(2, 1, 0), (0, 1, 2), (4, 2, 1), (6, 3, 3), (10, 5, 1), (-6, 3, -2), (-2, -1, 2), (8, -4, 19), (20, 19, -20),
           (-20, 10, 5), (3, 4, 0), (-12, 0, 5), (1, 1, 1), (7, -7, 7), (0, -20, 10), (15, -20, 0)]


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("q", range(len(OFFSETS)))
def test_lines_match_oracle(q, dtype):
    from leachingsim_gb300.runtime import geom_fracture
    lab = np.full((42, 43, 41), 3, dtype)
    lab[20, 21, 20] = 2
    o = OFFSETS[q]
    lab[20 + o[0], 21 + o[1], 20 + o[2]] = 4
    ref, nref, eref = go.fracture(lab)
    out, n, enc = geom_fracture(lab)
    np.testing.assert_array_equal(out, ref)
    assert (n, enc) == (nref, eref)


@pytest.mark.parametrize("shape,pore,sulphide", [((1, 3, 4200), (0, 0, 2), (0, 1, 4190)),
                                                 ((2, 4200, 3), (1, 4197, 2), (0, 5, 0)),
                                                 ((4100, 2, 2), (4098, 1, 0), (2, 0, 1))])
def test_long_lines_match_oracle(shape, pore, sulphide):
    from leachingsim_gb300.runtime import geom_fracture
    lab = np.full(shape, 3, np.uint8)
    lab[pore], lab[sulphide] = 2, 4
    ref, nref, eref = go.fracture(lab)
    out, n, enc = geom_fracture(lab)
    np.testing.assert_array_equal(out, ref)
    assert (n, enc) == (nref, eref)
