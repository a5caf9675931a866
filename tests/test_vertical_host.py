"""CPU tests of the register kernels' generated recursion (vertical recursion on both sides) and of the
rule that swaps an s shell's pair, against the oracle."""
import os
import re
import sys

import numpy as np
import pytest

from gbasis_b200.autotune import light_class
from gbasis_b200.contractions import GeneralizedContractionShell
from oracle import eri_oracle as orc

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gbasis_b200", "csrc")
sys.path.insert(0, CSRC)

import gen_eri  # noqa: E402

EVERY = gen_eri.canonical_classes(3)
REGISTER = [c for c in EVERY if gen_eri.is_register(c)]


def _run(emit, env):
    lines = []
    emit(lines)
    exec("\n".join(re.sub(r"^(const )?(R|double) ", "", ln.strip().rstrip(";")) for ln in lines), env)


def test_kernel_classes():
    """Every class has a kernel class of the same total momentum and values; no pair of it starts
    with an s shell and ends with another; no class needs more registers than its own form did."""
    for c in EVERY:
        k, flip = gen_eri.kernel_class(c)
        assert (flip & 1, flip >> 1) == (int(c[0] == 0 < c[1]), int(c[2] == 0 < c[3]))
        assert sorted(k[:2]) == sorted(c[:2]) and sorted(k[2:]) == sorted(c[2:])
        assert not (k[0] == 0 < k[1]) and not (k[2] == 0 < k[3])
        assert gen_eri.kernel_class(k) == (k, 0)
        if gen_eri.is_light(c):
            assert gen_eri.is_light(k) and gen_eri.is_register(c)
        assert gen_eri.is_register(c) == gen_eri.is_register(k) == light_class(c)
        assert not gen_eri.is_register(c) or sum(k) <= gen_eri.MAX_EMIT_L


@pytest.mark.parametrize("tight", [False, True])
@pytest.mark.parametrize("cls", REGISTER)
def test_vertical_recursion_matches_oracle(cls, tight):
    """`tight`: s shells of exponent 40 far from their partners, so that a flipped pair's centre is
    far from P.  Values of order 1 at most; 1e-12 absolute as for the engine."""
    rng = np.random.default_rng([int("1%d%d%d%d" % cls), tight])
    shells = [GeneralizedContractionShell(
        l, rng.uniform(-1, 1, 3), np.array([1.0]),
        np.array([40.0 if tight and l == 0 else rng.uniform(0.3, 1.5)]), "cartesian") for l in cls]
    ref = orc.construct_array_contraction(*shells, reorder="exponent")[0, :, 0, :, 0, :, 0, :]
    k, flip = gen_eri.kernel_class(cls)
    run = list(shells)
    if flip & 1:
        run[:2] = run[1::-1]
    if flip & 2:
        run[2:] = run[:1:-1]
    (a, A), (b, B), (c, C), (d, D) = [(float(s.exps[0]), s.coord) for s in run]
    z, e = a + b, c + d
    P, Q = (a * A + b * B) / z, (c * C + d * D) / e
    PQ, rho = P - Q, z * e / (z + e)
    norm = np.prod([(2 * s.exps[0] / np.pi) ** 0.75 * (4 * s.exps[0]) ** (s.angmom / 2) for s in run])
    pref = 2 * np.pi ** 2.5 / (z * e * np.sqrt(z + e)) * norm \
        * np.exp(-a * b / z * (A - B) @ (A - B) - c * d / e * (C - D) @ (C - D))
    g, h = gen_eri.best_vertical(*k), gen_eri.HrrGen(*k)
    nc = [gen_eri.ncart(l) for l in k]
    env = dict(fma=lambda x, y, w: x * y + w, R=float, o2z=0.5 / z, rz=rho / z, o2e=0.5 / e, re=rho / e,
               o2s=0.5 / (z + e), F=[pref * float(orc.boys(m, rho * PQ @ PQ)) for m in range(sum(k) + 1)],
               acc=[0.0] * (len(g.E) * len(g.F)), out=[0.0] * int(np.prod(nc)))
    for i, x in enumerate("xyz"):
        env.update({"PA" + x: (P - A)[i], "WP" + x: -rho / z * PQ[i], "QC" + x: (Q - C)[i],
                    "WQ" + x: rho / e * PQ[i], "AB" + x: (A - B)[i], "CD" + x: (C - D)[i]})
    _run(g.emit, env)
    _run(h.emit, env)
    cn = [1 / np.sqrt(np.prod(orc.factorial2(2 * orc.cart_components(l) - 1), axis=1)) for l in k]
    got = np.einsum("abcd,a,b,c,d->abcd", np.array(env["out"]).reshape(nc), *cn)
    if flip & 1:
        got = got.transpose(1, 0, 2, 3)
    if flip & 2:
        got = got.transpose(0, 1, 3, 2)
    assert got.shape == ref.shape
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-12)
