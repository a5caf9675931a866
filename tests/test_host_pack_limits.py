"""CPU test: norms that the general packing accepts or refuses are the ones the fast packing does."""
import numpy as np
import pytest

from gbasis_b200 import _engine
from gbasis_b200.contractions import (GeneralizedContractionShell, default_cart_components,
                                      default_sph_components)


class _General(GeneralizedContractionShell):
    """Overrides the orders with the same values: takes the general path."""

    @property
    def angmom_components_cart(self):
        return default_cart_components(self.angmom)

    @property
    def angmom_components_sph(self):
        return default_sph_components(self.angmom)


INF = np.inf
NORMS = [[[INF] * 6, [2.0] * 6], [[2.0] * 6, [INF] * 6], [[INF] * 6, [2.0 * (1 + 1e-15)] + [2.0] * 5],
         [[-INF] * 6, [0.0] * 6], [[INF] * 5 + [1.0], [2.0] * 6], [[INF] * 5 + [-INF], [2.0] * 6],
         [[np.nan] * 6, [2.0] * 6], [[2.0 * (1 + 1e-13)] + [2.0] * 5, [2.0] * 6]]


@pytest.mark.filterwarnings("ignore::RuntimeWarning")
@pytest.mark.parametrize("norms", NORMS, ids=range(len(NORMS)))
def test_spherical_norms(norms):
    packed = []
    for cls in (_General, GeneralizedContractionShell):
        sh = cls(2, np.zeros(3), np.array([[0.5, 0.2], [0.4, 0.3]]), np.array([1.0, 2.0]), "spherical")
        sh.norm_cont = np.array(norms)
        try:
            packed.append(_engine.pack_basis([sh]))
        except NotImplementedError as e:
            packed.append(str(e))
    general, fast = packed
    assert type(general) is type(fast)
    if isinstance(general, str):
        assert general == fast
    else:
        for k in general:
            np.testing.assert_array_equal(general[k], fast[k])
