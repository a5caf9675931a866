"""GPU tests of the recursion centre of pairs with an s shell (register and quadrature kernels).

A pair of a tight s shell and a diffuse shell far from it runs with the diffuse shell as the
centre, far from the pair's own centre; one primitive quartet and several.  Tolerance: 1e-12
absolute, the bar of the FP64 form, on values of order 1 and below.  The whole tensors are compared
with the McMurchie-Davidson values of the performance cases: on (ff|ff) of these shells the oracle's
own recursions are 1.4e-12 off them.
"""
import importlib.util
import os

import numpy as np
import pytest

from gbasis_b200 import electron_repulsion as er
from gbasis_b200.contractions import GeneralizedContractionShell
from oracle import eri_oracle as orc

pytestmark = pytest.mark.gpu

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_spec = importlib.util.spec_from_file_location("perf_cases", os.path.join(_ROOT, "perf", "cases.py"))
perf_cases = importlib.util.module_from_spec(_spec)
_spec.loader.exec_module(perf_cases)

CLASSES = [(0, 1, 0, 0), (0, 1, 0, 1), (1, 0, 0, 1), (0, 2, 0, 1), (0, 2, 1, 0), (0, 2, 0, 2),
           (2, 0, 0, 2), (0, 2, 1, 1), (1, 1, 0, 1), (1, 2, 0, 1), (2, 1, 0, 1), (0, 3, 0, 0),
           (0, 3, 0, 1), (0, 3, 0, 2), (0, 3, 0, 3), (0, 3, 1, 2), (1, 2, 0, 2), (2, 2, 0, 2),
           (3, 1, 0, 1), (3, 3, 0, 3)]


@pytest.mark.parametrize("coord", ["cartesian", "spherical"])
@pytest.mark.parametrize("prims", [1, 3])
@pytest.mark.parametrize("cls", CLASSES)
def test_flipped_pairs_against_oracle(cls, prims, coord):
    rng = np.random.default_rng([int("1%d%d%d%d" % cls), prims])
    centers = [(0.0, 0.1, 0.0), (1.4, -0.9, 1.1), (0.3, 0.2, -0.8), (-1.0, 1.2, 0.5)]
    shells = [GeneralizedContractionShell(
        l, np.array(c), rng.uniform(0.2, 1.0, prims),
        (60.0 if l == 0 else 0.5) * 1.3 ** np.arange(prims), coord) for l, c in zip(cls, centers)]
    if coord == "spherical":
        # whole tensor of the four shells: every orientation of every pair
        got = er.electron_repulsion_integral(shells, notation="chemist")
        ref = perf_cases._tensor([(s.angmom, s.coord, s.exps, np.asarray(s.coeffs).ravel())
                                  for s in shells], coord).cpu().numpy()
    else:
        got = er.ElectronRepulsionIntegral.construct_array_contraction(*shells)
        ref = orc.construct_array_contraction(*shells, reorder="exponent")
    assert got.shape == ref.shape
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-12)
