"""Packing of shells with the package's own component orders against the general path.

A subclass that overrides the order properties with the same values takes the general path, which
searches every component; both must pack the same arrays, bit for bit.
"""
import numpy as np
import pytest

from gbasis_b200 import _engine
from gbasis_b200.contractions import (GeneralizedContractionShell, default_cart_components,
                                      default_sph_components)


class _General(GeneralizedContractionShell):
    @property
    def angmom_components_cart(self):
        return default_cart_components(self.angmom)

    @property
    def angmom_components_sph(self):
        return default_sph_components(self.angmom)


def _shells(cls, coord):
    rng = np.random.default_rng(4)
    out = []
    for l in range(4):
        for m in (1, 2, 3):
            k = 1 + (l + m) % 4
            coeffs = rng.uniform(0.1, 1.0, size=(k, m))
            out.append(cls(l, rng.normal(size=3), coeffs[:, 0] if m == 1 else coeffs,
                           rng.uniform(0.2, 3.0, size=k), coord))
    return out


@pytest.mark.parametrize("coord", ["cartesian", "spherical"])
@pytest.mark.parametrize("override", [None, "cartesian", "spherical", "raw"])
def test_default_orders_pack_as_the_general_path(coord, override):
    types = None if override in (None, "raw") else [override] * 12
    raw = override == "raw"
    fast = _engine.pack_basis(_shells(GeneralizedContractionShell, coord), types, raw)
    slow = _engine.pack_basis(_shells(_General, coord), types, raw)
    assert not any(_engine._default_orders(s) for s in _shells(_General, coord))
    assert set(fast) == set(slow)
    for k in fast:
        assert fast[k].dtype == slow[k].dtype
        np.testing.assert_array_equal(fast[k], slow[k])


@pytest.mark.parametrize("cls", [GeneralizedContractionShell, _General])
def test_component_dependent_norm_is_refused_for_spherical(cls):
    sh = _shells(cls, "spherical")[6]
    sh.norm_cont = np.asarray(sh.norm_cont) * np.linspace(1.0, 2.0, sh.num_cart)
    with pytest.raises(NotImplementedError):
        _engine.pack_basis([sh])
    _engine.pack_basis([sh], ["cartesian"])
