"""GPU tests of the ordered work lists of a batch: every quartet of a list runs exactly once.

Lists of 1 quartet, of less than, exactly and just over a warp's 32, of several warps' pieces with a
ragged end, and of one and many buckets of primitive counts; each molecule's tensor against its own
single-basis call.  Tolerance: 1e-13 of the largest element, the bar of the batch form.
"""
import numpy as np
import pytest

from gbasis_b200 import electron_repulsion as er
from gbasis_b200.batch import electron_repulsion_integral_batch
from gbasis_b200.contractions import GeneralizedContractionShell

pytestmark = pytest.mark.gpu


def _molecule(rng, n, prims):
    return [GeneralizedContractionShell(0, rng.uniform(-2, 2, 3), rng.uniform(0.2, 1.0, k),
                                        0.3 * 2.0 ** np.arange(k, dtype=float), "cartesian")
            for k in (prims[i % len(prims)] for i in range(n))]


# s shells per molecule: n shells give n (n + 1) / 2 pairs and the quartets of a triangle of those
@pytest.mark.parametrize("sizes", [(1,), (2,), (1,) * 32, (1,) * 33, (3, 1), (4, 3), (5, 6, 7), (13, 2, 9)])
@pytest.mark.parametrize("prims", [(2,), (1, 3, 6)])
def test_every_quartet_once(sizes, prims):
    rng = np.random.default_rng([len(sizes), sum(sizes), len(prims)])
    mols = [_molecule(rng, n, prims) for n in sizes]
    got = electron_repulsion_integral_batch(mols, notation="chemist")
    for m, t in zip(mols, got):
        ref = er.electron_repulsion_integral(m, notation="chemist")
        t = np.asarray(t.cpu()) if hasattr(t, "cpu") else np.asarray(t)
        assert t.shape == ref.shape
        np.testing.assert_allclose(t, ref, rtol=0, atol=1e-13 * abs(ref).max())
