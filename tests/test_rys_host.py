"""CPU tests of the quadrature kernel's tables and plans (``csrc/gen_rys.py``).

The tables are evaluated as the device evaluates them (double precision Horner) and the generated
matrix products of every heavy class are executed from the emitted code and its table words, with
the device's table layout, against the direct recursion (``gen_lines.emulate``).
"""
import math
import os
import random
import re
import sys

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gbasis_b200", "csrc")
sys.path.insert(0, CSRC)

import gen_eri  # noqa: E402
import gen_lines  # noqa: E402
import gen_rys  # noqa: E402

HEAVY = [c for c in gen_eri.canonical_classes(3) if not gen_eri.is_light(c)]


def _boys(m, T):
    """F_m(T) by the ascending series (positive terms)."""
    term = total = 1.0 / (2 * m + 1)
    k = 0
    while term > total * 1e-18:
        k += 1
        term *= 2.0 * T / (2 * m + 2 * k + 1)
        total += term
    return math.exp(-T) * total


def _points(n, T, tab):
    """(x, w) of the n points as ``rys_point`` evaluates them."""
    if T < gen_rys.TMAX[n]:
        i = int(T)
        u = 2.0 * (T - i) - 1.0
        c = tab[i * (gen_rys.DEG + 1) * n * 2:(i + 1) * (gen_rys.DEG + 1) * n * 2]
        c = c.reshape(-1, n, 2, 2).transpose(0, 2, 1, 3).reshape(gen_rys.DEG + 1, n, 2)
        v = c[-1].copy()
        for d in range(gen_rys.DEG - 1, -1, -1):
            v = v * u + c[d]
        return v[:, 0], v[:, 1]
    h = tab[-4 * n:].reshape(n, 4)
    return h[:, 0] / T, h[:, 1] / math.sqrt(T)


@pytest.mark.parametrize("n", sorted(gen_rys.TMAX))
def test_points_reproduce_boys_values(n):
    """An n-point rule gives F_0 .. F_{2n-1}: interval edges and interiors, both sides of the switch
    to the Hermite limit.  Tolerance: each power multiplies the points' few-eps errors."""
    tab = np.array(gen_rys.root_table(n))
    top = gen_rys.TMAX[n]
    for T in [0.0, 1e-9, 0.3, 0.5, 0.999999, 1.0, 3.25, 7.75, 12.0, 20.5, 31.0, 44.4, top - 1e-9,
              float(top), top + 0.5, 150.0, 600.0]:
        x, w = _points(n, T, tab)
        for m in range(2 * n):
            ref = _boys(m, T) if T < 300 else 0.5 * math.gamma(m + 0.5) / T ** (m + 0.5)
            assert abs(float(np.sum(w * x ** m)) / ref - 1.0) < 2e-14 * (m + 1), (n, T, m)


def _reference(S, z, e, PA, QC, PQ):
    """[e0|f0] of one primitive quartet by the direct recursion in 40 digits (the transfer recursion
    loses digits in double precision when zeta / eta is large)."""
    from mpmath import gammainc, mp, mpf
    with mp.workdps(40):
        z, e = mpf(z), mpf(e)
        PQ, PA, QC = ([mpf(v) for v in w] for w in (PQ, PA, QC))
        rz = e / (z + e)
        T = z * rz * sum(v * v for v in PQ)
        F = [gammainc(m + mpf(1) / 2, 0, T) / (2 * T ** (m + mpf(1) / 2)) for m in range(S.L + 1)]
        ref = [mpf(0)] * (S.NE * S.NF)
        gen_lines.emulate(S, F, PA, [-rz * v for v in PQ], 1 / (2 * z), rz,
                          [z / e * a + c for a, c in zip(PA, QC)], z / e, 1 / (2 * e), ref)
        return np.array([float(v) for v in ref])


def _tables(p, x, w, PA, QC, PQ, z, e):
    """The 1-D tables of one primitive quartet in the device's layout, padding points included."""
    n, rf = len(x), p.rf
    ts = p.nE * rf * gen_rys.KS
    inv = 1.0 / (z + e)
    rz, re_, o2z, o2e = e * inv, z * inv, 0.5 / z, 0.5 / e
    tab = np.full(3 * ts, np.nan)
    for r in range((n + 3) & ~3):
        on = r < n
        xr = x[r] if on else 0.0
        B00, B10, B01 = (0.5 * xr * inv, o2z - xr * rz * o2z, o2e - xr * re_ * o2e) if on else (0, 0, 0)
        for ax in range(3):
            C = PA[ax] - xr * rz * PQ[ax] if on else 0.0
            D = QC[ax] + xr * re_ * PQ[ax] if on else 0.0
            t = np.zeros((p.nE, p.nF))
            t[0, 0] = (w[r] if on else 0.0) if ax == 2 else 1.0
            for a in range(1, p.nE):
                t[a, 0] = C * t[a - 1, 0] + ((a - 1) * B10 * t[a - 2, 0] if a > 1 else 0.0)
            for f in range(1, p.nF):
                for a in range(p.nE):
                    t[a, f] = (D * t[a, f - 1] + ((f - 1) * B01 * t[a, f - 2] if f > 1 else 0.0)
                               + (a * B00 * t[a - 1, f - 1] if a else 0.0))
            for a in range(p.nE):
                for f in range(p.nF):
                    tab[ax * ts + (a * rf + f) * gen_rys.KS + r] = t[a, f]
    return tab


def _execute(cls, tab, kcp, nfs, ne):
    """ACC from the emitted code: every warp's matrix products and stores."""
    p = gen_rys.plan(cls)
    code, words = gen_rys.emit_class(cls, "X", 0)
    cut = code.index("void store(")
    parts = [re.split(r"case \d+: \{|default: \{", t) for t in (code[:cut], code[cut:])]
    if p.warps > 1:
        parts = [t[1:] for t in parts]
    assert [len(t) for t in parts] == [p.warps] * 2

    def rows(at, shift, mask=0xffff):
        out = []
        for v in words[at:at + 8]:
            off = v >> shift & mask
            assert off % 8 == 0
            out.append(tab[off // 8:off // 8 + kcp])
        return np.array(out)
    acc_out = np.full(ne * nfs, np.nan)
    for gemm, store in zip(*parts):
        at = {m[1]: int(m[2]) for m in
              re.finditer(r"unsigned (z\d+_\d+|c\d+) = __ldg\(X \+ (\d+) \+ r\)", gemm)}
        acc = {}
        for m in re.finditer(r"rys_mma\(acc\[(\d+)\], acc\[\d+\], v(\d+), b(\d+_\d+)\)", gemm):
            c = at["c" + m[2]]
            acc[m[1]] = (rows(c, 0) * rows(c, 16)) @ rows(at["z" + m[3]], 0, 0xffffffff).T
        for m in re.finditer(r"rys_put\(__ldg\(X \+ (\d+) \+ lane\), acc\[(\d+)\]", store):
            for lane in range(32):
                v = words[int(m[1]) + lane]
                for h, place in enumerate((v & 0xffff, v >> 16)):
                    if place != 0xffff:
                        assert math.isnan(acc_out[place])  # every target once
                        acc_out[place] = acc[m[2]][lane >> 2, 2 * (lane & 3) + h]
    return acc_out


@pytest.mark.parametrize("cls", HEAVY, ids=lambda c: "%d%d%d%d" % c)
def test_generated_products_match_recursion(cls):
    rng = random.Random(sum(v * 4 ** i for i, v in enumerate(cls)))
    z, e = rng.uniform(0.5, 5.0), rng.uniform(0.5, 5.0)
    PQ, PA, QC = ([rng.uniform(-0.8, 0.8) for _ in range(3)] for _ in range(3))
    rz = e / (z + e)
    T = z * rz * sum(v * v for v in PQ)
    S = gen_lines.Schedule(*cls)
    ref = _reference(S, z, e, PA, QC, PQ)
    p, n = gen_rys.plan(cls), gen_rys.n_points(cls)
    x, w = (v[0].astype(float) for v in gen_rys.rys_points(n, [T]))
    tab = _tables(p, x, w, PA, QC, PQ, z, e)
    nfs = S.NF | 1
    got = _execute(cls, tab, (n + 3) & ~3, nfs, S.NE).reshape(S.NE, nfs)[:, :S.NF].reshape(-1)
    assert not np.isnan(got).any()
    assert np.max(np.abs(got - ref)) < 1e-13 * max(1.0, np.max(np.abs(ref)))
