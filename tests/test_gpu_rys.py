"""GPU tests of the quadrature kernel at the edges of its point chunks and of its tables.

A chunk holds 32 // n primitive quartets of n = L/2 + 1 points, so the primitive counts below are
one quartet, a full chunk, a full chunk and one, and several chunks; the separations put T of the
primitive quartets in the tables, across the switch to the Hermite limit, and beyond it.
Tolerance: 1e-12 absolute, the bar of the FP64 form, on values of order 1 and below.
"""
import numpy as np
import pytest

from gbasis_b200 import electron_repulsion as er
from gbasis_b200.contractions import GeneralizedContractionShell
from oracle import eri_oracle as orc

pytestmark = pytest.mark.gpu


def _shell(rng, l, k, center):
    # a narrow exponent range: the contracted recursions of the oracle keep their digits
    exps = 0.6 * 1.15 ** np.arange(k, dtype=float) * rng.uniform(0.9, 1.1)
    return GeneralizedContractionShell(l, np.asarray(center, dtype=float), rng.uniform(0.2, 1.0, k),
                                       exps, "cartesian")


@pytest.mark.parametrize("distance", [0.7, 9.0, 30.0])
@pytest.mark.parametrize("cls,prims", [
    ((2, 1, 1, 1), (1, 1, 1, 1)), ((2, 1, 1, 1), (5, 1, 2, 1)), ((2, 1, 1, 1), (11, 1, 1, 1)),
    ((1, 2, 2, 0), (3, 1, 7, 1)), ((2, 2, 1, 1), (4, 1, 2, 1)), ((2, 2, 1, 1), (3, 1, 3, 1)),
    ((2, 2, 2, 2), (1, 1, 1, 1)), ((2, 2, 2, 2), (3, 1, 2, 1)), ((2, 2, 2, 2), (2, 2, 2, 1)),
    ((3, 0, 3, 0), (7, 1, 1, 1)), ((3, 2, 3, 2), (1, 1, 5, 1)), ((3, 2, 3, 2), (2, 1, 3, 1)),
    ((3, 3, 3, 3), (1, 1, 1, 1)), ((3, 3, 3, 3), (2, 1, 2, 1)), ((3, 3, 3, 3), (5, 1, 1, 1)),
])
def test_chunk_edges_against_oracle(cls, prims, distance):
    rng = np.random.default_rng([int("%d%d%d%d" % cls), *prims])
    centers = [(0.0, 0.1, 0.0), (0.4, -0.3, 0.5), (distance, 0.2, -0.1), (distance - 0.5, 0.0, 0.6)]
    shells = [_shell(rng, l, k, c) for l, k, c in zip(cls, prims, centers)]
    got = er.ElectronRepulsionIntegral.construct_array_contraction(*shells)
    ref = orc.construct_array_contraction(*shells, reorder="exponent")
    assert got.shape == ref.shape
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-12)
