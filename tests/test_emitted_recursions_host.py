"""CPU tests of recursions that the device compiles and no other CPU test runs.

The (ab|ss) structs of the point-charge kernel, s shells first included, executed with that kernel's
own arguments (rho / zeta = 1, the ket's all zero) against the point-charge oracle, and the unflipped
two-electron form of the same structs against the quartet oracle.  Values of order 1 and below; 1e-12
absolute as for the engine.
"""
import os
import re
import sys

import numpy as np
import pytest

from gbasis_b200.contractions import GeneralizedContractionShell
from oracle import eri_oracle as orc
from oracle import point_charge_oracle as pco

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gbasis_b200", "csrc")
sys.path.insert(0, CSRC)

import gen_eri  # noqa: E402

PAIRS = [(la, lb) for la in range(4) for lb in range(4)]


def _run(emit, env):
    lines = []
    emit(lines)
    exec("\n".join(re.sub(r"^(const )?(R|double) ", "", ln.strip().rstrip(";")) for ln in lines), env)


def _values(la, lb, A, B, F, **args):
    """Component-normalised (ab|00) of the emitted code, on scalars F and the recursion's arguments."""
    g, h = gen_eri.best_vertical(la, lb, 0, 0), gen_eri.HrrGen(la, lb, 0, 0)
    shape = gen_eri.ncart(la), gen_eri.ncart(lb)
    env = dict(fma=lambda x, y, w: x * y + w, R=float, F=F, acc=[0.0] * (len(g.E) * len(g.F)),
               out=[0.0] * (shape[0] * shape[1]))
    for k, v in args.items():
        if np.ndim(v):
            env.update({k + x: float(v[i]) for i, x in enumerate("xyz")})
        else:
            env[k] = float(v)
    for i, x in enumerate("xyz"):
        env.update({"AB" + x: (A - B)[i], "CD" + x: 0.0})
    _run(g.emit, env)
    _run(h.emit, env)
    cn = [1 / np.sqrt(np.prod(orc.factorial2(2 * orc.cart_components(l) - 1), axis=1)) for l in (la, lb)]
    return np.array(env["out"]).reshape(shape) * cn[0][:, None] * cn[1][None, :]


def _pair(la, lb, seed):
    rng = np.random.default_rng([la, lb, seed])
    sa, sb = (GeneralizedContractionShell(l, rng.uniform(-1, 1, 3), np.array([1.0]),
                                          np.array([rng.uniform(0.4, 2.0)]), "cartesian")
              for l in (la, lb))
    (a, A), (b, B) = [(float(s.exps[0]), s.coord) for s in (sa, sb)]
    z = a + b
    norm = np.prod([(2 * s.exps[0] / np.pi) ** 0.75 * (4 * s.exps[0]) ** (s.angmom / 2) for s in (sa, sb)])
    return rng, sa, sb, A, B, z, (a * A + b * B) / z, norm * np.exp(-a * b / z * (A - B) @ (A - B))


@pytest.mark.parametrize("la,lb", PAIRS)
def test_the_emitted_structs_are_the_ones_tested(la, lb):
    body = []
    gen_eri.best_vertical(la, lb, 0, 0).emit(body)
    text = "".join(body)
    assert text in re.sub(r"\n *", "", gen_eri.emit_all(3, [(la, lb, 0, 0)]))


@pytest.mark.parametrize("la,lb", PAIRS)
def test_point_charge_arguments(la, lb):
    rng, sa, sb, A, B, z, P, k = _pair(la, lb, 1)
    C, q = rng.uniform(-1, 1, 3), rng.uniform(0.5, 3.0)
    ref = pco.pair_contraction(sa, sb, C[None], np.array([q]))[0, :, 0, :, 0]
    PC = P - C
    F = [k * 2 * np.pi / z * float(orc.boys(m, z * PC @ PC)) for m in range(la + lb + 1)]
    zero = np.zeros(3)
    got = -q * _values(la, lb, A, B, F, PA=P - A, WP=-PC, o2z=0.5 / z, rz=1.0, QC=zero, WQ=zero, o2e=0.0,
                       re=0.0, o2s=0.0)
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-12)


@pytest.mark.parametrize("la,lb", PAIRS)
def test_unflipped_two_electron_arguments(la, lb):
    rng, sa, sb, A, B, z, P, k = _pair(la, lb, 2)
    _, sc, sd, C, D, e, Q, kk = _pair(0, 0, 3 + la + 4 * lb)
    ref = orc.quartet_cartesian(sa, sb, sc, sd)[:, :, 0, 0, 0, 0, 0, 0]
    PQ, rho = P - Q, z * e / (z + e)
    pref = 2 * np.pi ** 2.5 / (z * e * np.sqrt(z + e)) * k * kk
    F = [pref * float(orc.boys(m, rho * PQ @ PQ)) for m in range(la + lb + 1)]
    got = _values(la, lb, A, B, F, PA=P - A, WP=-rho / z * PQ, o2z=0.5 / z, rz=rho / z, QC=Q - C,
                  WQ=rho / e * PQ, o2e=0.5 / e, re=rho / e, o2s=0.5 / (z + e))
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-12)
