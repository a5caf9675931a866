"""GPU tests of the quadrature kernel at the edges of its passes over a quartet's points.

A CTA of W warps makes the points of W chunks at a time, a chunk holding 32 // n primitive quartets
of n = L/2 + 1 points (32 // 2n for erfc, which takes 2n points each), and cuts the tables in chunks,
in one buffer or two.  The primitive counts below are, for a pass of p primitive quartets: just below
p, p, just above p, and two passes with a remainder, for kernels of 1, 2, 4 and 8 warps with one buffer
and of 4 and 8 warps with two.  The first and third shell have the larger exponents, so that the class
run is the class named.

Tolerance: 1e-12 absolute, the bar of the FP64 form, on values of order 1 and below (contraction
coefficients sum to 1); the oracle is within 2e-15 of McMurchie-Davidson values there.
"""
import numpy as np
import pytest

from gbasis_b200 import _engine
from gbasis_b200.contractions import GeneralizedContractionShell
from oracle import eri_oracle as orc

pytestmark = pytest.mark.gpu

# class: primitives of the first and third shell, for 1/r and erf (p), for erfc (p / 2)
CASES = {
    (1, 2, 2, 0): ([(3, 3), (5, 2), (11, 1), (8, 3)], [(4, 1), (5, 1), (3, 2), (11, 1)]),
    (2, 1, 1, 1): ([(6, 3), (5, 4), (7, 3), (8, 5), (7, 6)], [(3, 3), (5, 2), (11, 1), (7, 3)]),
    (2, 2, 2, 2): ([(11, 2), (6, 4), (5, 5), (8, 6), (7, 7)], [(11, 1), (4, 3), (7, 2), (5, 5)]),
    (2, 3, 1, 1): ([(6, 5), (8, 4), (11, 3), (9, 7), (11, 6)], [(5, 3), (4, 4), (6, 3), (11, 3)]),
    (3, 2, 1, 1): ([(6, 5), (8, 4), (11, 3), (10, 7)], [(5, 3), (4, 4), (11, 3)]),
    (3, 2, 2, 3): ([(6, 6), (8, 5), (7, 6), (9, 9)], [(5, 3), (4, 4), (6, 3), (11, 3)]),
    (3, 3, 3, 3): ([(6, 5), (8, 4), (11, 3), (9, 7), (11, 6)], [(5, 3), (4, 4), (6, 3), (11, 3)]),
}
CENTERS = [(0.0, 0.1, 0.0), (0.4, -0.3, 0.5), (0.9, 0.2, -0.1), (0.3, 0.0, 0.6)]


def quartet(cls, counts, coord):
    rng = np.random.default_rng([int("1%d%d%d%d" % cls), *counts])
    shells = []
    for l, k, f, c in zip(cls, (counts[0], 1, counts[1], 1), (1.5, 0.6, 1.5, 0.6), CENTERS):
        w = rng.uniform(0.2, 1.0, k)
        shells.append(GeneralizedContractionShell(l, np.array(c), w / w.sum(),
                                                  f * 1.06 ** np.arange(k), coord))
    return shells


def block(shells, raw, potential):
    """The (AB|CD) block of the four shells' tensor."""
    db = _engine.DeviceBasis(shells, raw=raw)
    if potential[0]:
        db.set_potential(*potential)
    full = db.full_host("chemist")
    db.close()
    n = [s.num_cart if raw else s.num_sph for s in shells]
    o = np.cumsum([0] + n)
    return full[o[0]:o[1], o[1]:o[2], o[2]:o[3], o[3]:o[4]]


@pytest.mark.parametrize("potential", [(0, 0.0), (1, 0.7), (2, 0.7)])
@pytest.mark.parametrize("cls", CASES)
def test_pass_edges_against_oracle(cls, potential):
    for counts in CASES[cls][potential[0] == 2]:
        check(cls, counts, potential)


def check(cls, counts, potential):
    shells = quartet(cls, counts, "spherical")
    raw = orc.construct_array_contraction(*shells, reorder="exponent", potential=potential)
    raw = raw[0, :, 0, :, 0, :, 0, :]
    got = block(shells, True, potential)
    assert got.shape == raw.shape
    np.testing.assert_allclose(got, raw, rtol=0, atol=1e-12)
    W = [orc._shell_matrix(s, "spherical") for s in shells]
    ref = np.einsum("pa,qb,rc,sd,abcd->pqrs", *W, raw, optimize=True)
    got = block(shells, False, potential)
    assert got.shape == ref.shape
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-12)
