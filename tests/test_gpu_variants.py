"""GPU tests of the heavy classes' selectable kernels (``gbx_set_block_config`` variants 1 and 2: line
kernel, split kernel or group form) over every heavy class, in the store, attenuated and Coulomb modes,
in a batch, and in the bounds-checking build where it is built.

Checker: the default kernels, which other tests hold against the oracle.  Tolerance: 1e-12 absolute on
tensors of values of order 1 and below (narrow exponent ranges: the older kernels' recursions keep their
digits); J and erfc sum as many such values as they have terms, 1e-12 of the largest element.
"""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from gbasis_b200 import _engine
from gbasis_b200.batch import EriBatch
from gbasis_b200.contractions import GeneralizedContractionShell

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "gbasis_b200", "csrc"))

import gen_eri  # noqa: E402

DEBUG_LIB = os.path.join(ROOT, "gbasis_b200", "_lib", "libgbx_eri_debug.so")


def _shells(coord, seed=11):
    """Three shells of each l with tight and diffuse ones: every ordered pair class."""
    rng = np.random.default_rng(seed)
    out = []
    for scale in (0.5, 0.8, 1.3):
        for l in range(4):
            w = rng.uniform(0.3, 1.0, 2)
            out.append(GeneralizedContractionShell(l, rng.uniform(-1.5, 1.5, 3), w / w.sum(),
                                                   scale * np.array([1.0, 1.4]) * rng.uniform(0.9, 1.1),
                                                   coord))
    return out


# the classes that have variants: beyond one thread's registers in their own order
HEAVY = {tuple(c) for c in gen_eri.canonical_classes(3) if not gen_eri.is_light(c)}


def _heavy(blocks):
    return [k for k, b in enumerate(blocks) if b[0] in HEAVY]


@pytest.mark.parametrize("coord", ["cartesian", "spherical"])
@pytest.mark.parametrize("variant", [1, 2])
def test_variants_equal_the_default_kernels(variant, coord):
    import torch
    db = _engine.DeviceBasis(_shells(coord), tuned=False)
    heavy = _heavy(db.blocks())
    assert {db.blocks()[k][0] for k in heavy} == HEAVY
    n = db.nbf
    rng = np.random.default_rng(3)
    D = rng.uniform(-0.5, 0.5, (n, n))
    D = torch.from_numpy(D + D.T).cuda()

    def values():
        out = []
        for potential in ((0, 0.0), (1, 0.6), (2, 0.6)):
            db.set_potential(*potential)
            out.append(torch.empty(n ** 4, dtype=torch.float64, device="cuda"))
            db.full_device(out[-1].data_ptr())
        db.set_potential(0, 0.0)
        J = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        _engine.check(_engine.lib().gbx_eri_coulomb_j(db.handle, ctypes.c_void_p(D.data_ptr()), 0.0,
                                                      ctypes.c_void_p(J.data_ptr()), None))
        torch.cuda.synchronize()
        return out + [J]
    ref = values()
    for k in heavy:
        db.set_block_config(k, variant)
    got = values()
    db.close()
    for r, g in zip(ref, got):
        assert float((g - r).abs().max()) <= 1e-12 * max(1.0, float(r.abs().max()))


@pytest.mark.parametrize("variant", [1, 2])
def test_variants_in_a_batch(variant):
    import torch
    mols = [_shells("spherical", s)[:4 + 4 * (s % 3)] for s in range(3)]
    b = EriBatch(mols)
    outs = [[torch.empty((n,) * 4, dtype=torch.float64, device="cuda") for n in b.nbf] for _ in range(2)]
    b.run(outs[0])
    for k in _heavy(b.types()):
        b.set_type_config(k, variant)
    b.run(outs[1])
    torch.cuda.synchronize()
    b.close()
    for r, g in zip(*outs):
        assert float((g - r).abs().max()) <= 1e-12


@pytest.mark.skipif(os.environ.get("GBX_DEBUG_BOUNDS") == "1", reason="runs in the child")
def test_variants_in_the_bounds_checking_build():
    if not os.path.exists(DEBUG_LIB):
        pytest.skip("libgbx_eri_debug.so is not built (python -m gbasis_b200.build --debug-bounds)")
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-m", "gpu", os.path.abspath(__file__)],
                       env=dict(os.environ, GBX_DEBUG_BOUNDS="1"), cwd=ROOT, capture_output=True,
                       text=True, timeout=1200)
    assert r.returncode == 0, (r.stdout[-3000:], r.stderr[-3000:])
    assert "6 passed, 1 skipped" in r.stdout
