"""Generate class-specialised recursion code for the ERI kernels (writes ``eri_gen.cuh``).

For every class (la, lb | lc, ld) — ordered pair types, the bra pair type not below the ket
pair type in the order (la + lb, max(la, lb), la) — this emits straight-line device code for

* ``prim``: one primitive quartet of the Obara-Saika vertical recursion on centre A
  ([e0|00]^(m), e <= L) followed by the electron-transfer recursion onto centre C
  ([e0|f0], la <= |e| <= la+lb, lc <= |f| <= lc+ld), accumulated into ``acc``;
* ``hrr``: the horizontal recursions (ket first, then bra) that turn the contracted
  [e0|f0] into the Cartesian block (ab|cd).

Only the intermediates the targets depend on are emitted (dependency closure), and the
recursion direction at every node is chosen per class to minimise the operation count.
The mathematics is that of gbasis (``gbasis/integrals/_two_elec_int.py:350-526`` for
VRR/ETR, ``:549-788`` for HRR); the code organisation is this project's.

Usage: ``python gen_eri.py [LMAX] > eri_gen.cuh`` (default LMAX = 3).
"""
from __future__ import annotations

import itertools
import sys

DIRS = "xyz"


def ncart(l):
    return (l + 1) * (l + 2) // 2


def comps(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def comps_range(lo, hi):
    return [c for n in range(lo, hi + 1) for c in comps(n)]


def add(t, i, k=1):
    u = list(t)
    u[i] += k
    return tuple(u)


def tname(t):
    return "".join(str(v) for v in t)


def pair_types(lmax):
    """Ordered pair types (lA, lB) sorted by (lA + lB, max, lA): the engine's pair classes."""
    return sorted(((a, b) for a in range(lmax + 1) for b in range(lmax + 1)),
                  key=lambda t: (t[0] + t[1], max(t), t[0]))


def canonical_classes(lmax):
    """(lA, lB, lC, lD) with the bra pair class not below the ket pair class."""
    pts = pair_types(lmax)
    return [bra + ket for i, bra in enumerate(pts) for ket in pts[: i + 1]]


# --------------------------------------------------------------------------- VRR/ETR
class PrimGen:
    """Dependency closure and code for one class's primitive recursion."""

    def __init__(self, la, lb, lc, ld, vrr_pick, etr_pick):
        self.la, self.lb, self.lc, self.ld = la, lb, lc, ld
        self.L = la + lb + lc + ld
        self.E = comps_range(la, la + lb)
        self.F = comps_range(lc, lc + ld)
        self.vrr_pick, self.etr_pick = vrr_pick, etr_pick
        self.vrr = {}  # (e, m) -> (i, deps)
        self.etr = {}  # (e, f) -> (i, deps)
        for e in self.E:
            for f in self.F:
                self._need_etr(e, f)

    def _need_vrr(self, e, m):
        key = (e, m)
        if key in self.vrr:
            return
        if sum(e) == 0:
            self.vrr[key] = None
            return
        i = self.vrr_pick(e)
        e1 = add(e, i, -1)
        self.vrr[key] = i
        self._need_vrr(e1, m)
        self._need_vrr(e1, m + 1)
        if e1[i] > 0:
            e2 = add(e1, i, -1)
            self._need_vrr(e2, m)
            self._need_vrr(e2, m + 1)

    def _need_etr(self, e, f):
        key = (e, f)
        if key in self.etr:
            return
        if sum(f) == 0:
            self.etr[key] = None
            self._need_vrr(e, 0)
            return
        i = self.etr_pick(e, f)
        f1 = add(f, i, -1)
        self.etr[key] = i
        self._need_etr(e, f1)
        self._need_etr(add(e, i), f1)
        if e[i] > 0:
            self._need_etr(add(e, i, -1), f1)
        if f1[i] > 0:
            self._need_etr(e, add(f1, i, -1))

    def op_count(self):
        n = 0
        for (e, m), i in self.vrr.items():
            if i is None:
                continue
            e1 = add(e, i, -1)
            n += 2 + (2 if e1[i] > 0 else 0)
        for (e, f), i in self.etr.items():
            if i is None:
                continue
            f1 = add(f, i, -1)
            n += 2 + (1 if e[i] > 0 else 0) + (1 if f1[i] > 0 else 0)
        return n

    @staticmethod
    def vname(e, m):
        return f"v{tname(e)}_{m}"

    @staticmethod
    def ename(e, f):
        if sum(f) == 0:
            return PrimGen.vname(e, 0)
        return f"t{tname(e)}_{tname(f)}"

    def emit(self, out):
        """Emit the body; inputs F[m], PA*, WP*, o2z, rz, CE*, ze, o2e; output acc[]."""
        order = sorted(self.vrr.items(), key=lambda kv: (sum(kv[0][0]), -kv[0][1]))
        for (e, m), i in order:
            nm = self.vname(e, m)
            if i is None:
                out.append(f"const R {nm} = F[{m}];")
                continue
            e1 = add(e, i, -1)
            d = DIRS[i]
            expr = f"fma(PA{d}, {self.vname(e1, m)}, WP{d} * {self.vname(e1, m + 1)})"
            if e1[i] > 0:
                e2 = add(e1, i, -1)
                k = e1[i]
                expr = (f"fma(R({k}) * o2z, fma(-rz, {self.vname(e2, m + 1)}, {self.vname(e2, m)}), "
                        f"{expr})")
            out.append(f"const R {nm} = {expr};")
        order = sorted(((k, v) for k, v in self.etr.items() if v is not None),
                       key=lambda kv: sum(kv[0][1]))
        for (e, f), i in order:
            f1 = add(f, i, -1)
            d = DIRS[i]
            expr = (f"fma(CE{d}, {self.ename(e, f1)}, -ze * {self.ename(add(e, i), f1)})")
            if e[i] > 0:
                expr = f"fma(R({e[i]}) * o2e, {self.ename(add(e, i, -1), f1)}, {expr})"
            if f1[i] > 0:
                expr = f"fma(R({f1[i]}) * o2e, {self.ename(e, add(f1, i, -1))}, {expr})"
            out.append(f"const R {self.ename(e, f)} = {expr};")
        nf = len(self.F)
        for ie, e in enumerate(self.E):
            for jf, f in enumerate(self.F):
                out.append(f"acc[{ie * nf + jf}] += {self.ename(e, f)};")


def pick_first(t, *_):
    return next(i for i in range(3) if t[i] > 0)


def pick_last(t, *_):
    return next(i for i in (2, 1, 0) if t[i] > 0)


def pick_max(t, *_):
    return max(range(3), key=lambda i: (t[i], -i))


def pick_etr_first(e, f):
    return pick_first(f)


def pick_etr_last(e, f):
    return pick_last(f)


def pick_etr_max(e, f):
    return pick_max(f)


def pick_etr_min_e(e, f):
    # prefer the direction where e is small (fewer [e-1] terms)
    cands = [i for i in range(3) if f[i] > 0]
    return min(cands, key=lambda i: (e[i], -f[i], i))


def best_prim(la, lb, lc, ld):
    best = None
    for vp in (pick_first, pick_last, pick_max):
        for ep in (pick_etr_first, pick_etr_last, pick_etr_max, pick_etr_min_e):
            g = PrimGen(la, lb, lc, ld, vp, ep)
            n = g.op_count()
            if best is None or n < best[0]:
                best = (n, g)
    return best[1]


class VerticalGen:
    """Primitive recursion of the register kernels: the Obara-Saika vertical recursion on both sides,
        [e+1_i|f]^(m) = PA_i [e|f]^(m) + WP_i [e|f]^(m+1) + e_i/(2 zeta) ([e-1_i|f]^(m)
                        - rho/zeta [e-1_i|f]^(m+1)) + f_i/(2 (zeta + eta)) [e|f-1_i]^(m+1)
    and the same for f with QC, WQ, eta.  Against the transfer recursion from [e+f|0] it needs
    20 to 35 % fewer operations and no [e|0] beyond the bra's own range, and none of its terms is
    multiplied by zeta/eta: the recursion centre may be the shell far from P."""

    def __init__(self, la, lb, lc, ld, pick):
        self.E = comps_range(la, la + lb)
        self.F = comps_range(lc, lc + ld)
        self.pick = pick
        self.nodes = {}  # (e, f, m) -> (side lowered, direction)
        for e in self.E:
            for f in self.F:
                self._need(e, f, 0)

    @staticmethod
    def terms(e, f, m, side, i):
        """The five operands (None where its factor is zero) and the two factors."""
        low, other = (e, f) if side == "bra" else (f, e)
        low1 = add(low, i, -1)

        def key(a, b, mm):
            return (a, b, mm) if side == "bra" else (b, a, mm)
        t = [key(low1, other, m), key(low1, other, m + 1)]
        t += [key(add(low1, i, -1), other, m), key(add(low1, i, -1), other, m + 1)] if low1[i] \
            else [None, None]
        t.append(key(low1, add(other, i, -1), m + 1) if other[i] else None)
        return t, low1[i], other[i]

    def _need(self, e, f, m):
        if (e, f, m) in self.nodes:
            return
        if sum(e) + sum(f) == 0:
            self.nodes[e, f, m] = None
            return
        side, i = self.pick(e, f)
        self.nodes[e, f, m] = (side, i)
        for t in self.terms(e, f, m, side, i)[0]:
            if t is not None:
                self._need(*t)

    def op_count(self):
        n = 0
        for (e, f, m), v in self.nodes.items():
            if v is not None:
                _, k, j = self.terms(e, f, m, *v)
                n += 2 + (2 if k else 0) + (1 if j else 0)
        return n

    @staticmethod
    def name(e, f, m):
        return f"v{tname(e)}_{tname(f)}_{m}"

    def emit(self, out):
        """Emit the body; inputs F[m], PA*, WP*, o2z, rz, QC*, WQ*, o2e, re, o2s; output acc[]."""
        order = sorted(self.nodes.items(), key=lambda kv: (sum(kv[0][0]) + sum(kv[0][1]), -kv[0][2]))
        for (e, f, m), v in order:
            if v is None:
                out.append(f"const R {self.name(e, f, m)} = F[{m}];")
                continue
            side, i = v
            t, k, j = self.terms(e, f, m, side, i)
            x, wx, o2, r = (("PA", "WP", "o2z", "rz") if side == "bra" else ("QC", "WQ", "o2e", "re"))
            d = DIRS[i]
            expr = f"fma({x}{d}, {self.name(*t[0])}, {wx}{d} * {self.name(*t[1])})"
            if k:
                expr = (f"fma(R({k}) * {o2}, fma(-{r}, {self.name(*t[3])}, {self.name(*t[2])}), "
                        f"{expr})")
            if j:
                expr = f"fma(R({j}) * o2s, {self.name(*t[4])}, {expr})"
            out.append(f"const R {self.name(e, f, m)} = {expr};")
        nf = len(self.F)
        for ie, e in enumerate(self.E):
            for jf, f in enumerate(self.F):
                out.append(f"acc[{ie * nf + jf}] += {self.name(e, f, 0)};")


def _vertical_picks():
    """Choices of (side, direction): a side first, and per side the direction of the fewest terms."""
    rules = [lambda t, o: min(i for i in range(3) if t[i]),
             lambda t, o: max(i for i in range(3) if t[i]),
             lambda t, o: max(range(3), key=lambda i: (t[i], -i)),
             lambda t, o: min((i for i in range(3) if t[i]), key=lambda i: (t[i], i)),
             lambda t, o: min((i for i in range(3) if t[i]), key=lambda i: (o[i] > 0, t[i] > 1, i)),
             lambda t, o: min((i for i in range(3) if t[i]), key=lambda i: (t[i] > 1, o[i] > 0, i))]
    for rb in rules:
        for rk in rules:
            for ket_first in (True, False):
                def pick(e, f, rb=rb, rk=rk, ket_first=ket_first):
                    if sum(f) and (ket_first or not sum(e)):
                        return "ket", rk(f, e)
                    return "bra", rb(e, f)
                yield pick


def best_vertical(la, lb, lc, ld):
    """The cheapest recursion of the class over the rules above."""
    gens = [VerticalGen(la, lb, lc, ld, p) for p in _vertical_picks()]
    return min(gens, key=lambda g: g.op_count())


def kernel_class(c):
    """(class whose kernel runs class c, flip bits: 1 bra, 2 ket).  A pair whose first shell is an
    s shell (the one with the larger exponent) and whose second is not runs with the second shell as
    the recursion centre: (s l| needs [e0| for e = 0 .. l and the horizontal recursion,
    (l s| = [l0| neither.  The s shell has one function, so the values' places are the same."""
    flip = [int(a == 0 and b > 0) for a, b in (c[:2], c[2:])]
    bra, ket = (p[::-1] if f else p for p, f in zip((tuple(c[:2]), tuple(c[2:])), flip))
    return bra + ket, flip[0] + 2 * flip[1]


# ---------------------------------------------------------------------------- HRR
class HrrGen:
    """(ab|cd) from contracted [e0|f0]: ket HRR with CD, then bra HRR with AB."""

    def __init__(self, la, lb, lc, ld):
        self.la, self.lb, self.lc, self.ld = la, lb, lc, ld
        self.E = comps_range(la, la + lb)
        self.F = comps_range(lc, lc + ld)

    @staticmethod
    def closure(lo, tgt_a, tgt_b, pick):
        nodes = {}

        def need(a, b):
            if (a, b) in nodes:
                return
            if sum(b) == 0:
                nodes[(a, b)] = None
                return
            i = pick(b)
            b1 = add(b, i, -1)
            nodes[(a, b)] = i
            need(add(a, i), b1)
            need(a, b1)

        for a in tgt_a:
            for b in tgt_b:
                need(a, b)
        return nodes

    def emit(self, out):
        la, lb, lc, ld = self.la, self.lb, self.lc, self.ld
        NF = len(self.F)
        Fidx = {f: j for j, f in enumerate(self.F)}
        Eidx = {e: j for j, e in enumerate(self.E)}
        cd_t = [(c, d) for c in comps(lc) for d in comps(ld)]
        ab_t = [(a, b) for a in comps(la) for b in comps(lb)]
        NCD = len(cd_t)
        best = None
        for pk in (pick_first, pick_last, pick_max):
            kn = self.closure(lc, comps(lc), comps(ld), pk)
            bn = self.closure(la, comps(la), comps(lb), pk)
            n = len(self.E) * sum(1 for v in kn.values() if v is not None) + \
                NCD * sum(1 for v in bn.values() if v is not None)
            if best is None or n < best[0]:
                best = (n, kn, bn)
        _, kn, bn = best
        korder = sorted(((k, v) for k, v in kn.items() if v is not None), key=lambda kv: sum(kv[0][1]))
        border = sorted(((k, v) for k, v in bn.items() if v is not None), key=lambda kv: sum(kv[0][1]))
        # ket side: for every e, h[e][cd]
        for ie, e in enumerate(self.E):
            def kname(c, d):
                if sum(d) == 0:
                    return f"acc[{ie * NF + Fidx[c]}]"
                return f"k{ie}_{tname(c)}_{tname(d)}"
            for (c, d), i in korder:
                dd = DIRS[i]
                d1 = add(d, i, -1)
                out.append(f"const double {kname(c, d)} = fma(CD{dd}, {kname(c, d1)}, "
                           f"{kname(add(c, i), d1)});")
            for icd, (c, d) in enumerate(cd_t):
                out.append(f"double h{ie}_{icd} = {kname(c, d)};")
        # bra side: for every cd, (ab|cd)
        NB = ncart(lb)
        for icd in range(NCD):
            def bname(a, b):
                if sum(b) == 0:
                    return f"h{Eidx[a]}_{icd}"
                return f"b{icd}_{tname(a)}_{tname(b)}"
            for (a, b), i in border:
                dd = DIRS[i]
                b1 = add(b, i, -1)
                out.append(f"const double {bname(a, b)} = fma(AB{dd}, {bname(a, b1)}, "
                           f"{bname(add(a, i), b1)});")
            for iab, (a, b) in enumerate(ab_t):
                out.append(f"out[{iab * NCD + icd}] = {bname(a, b)};")
        del NB


def _dfact(n):
    r = 1
    while n > 1:
        r *= n
        n -= 2
    return r


def emit_sph_and_norms(w, lmax):
    """Constant Cartesian->spherical code per l (engine_sph_matrix) and the Cartesian
    component norms 1/sqrt(prod (2a_i-1)!!) in canonical order."""
    import math
    import os
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__)))))
    from gbasis_b200.spherical import engine_sph_matrix
    w("template <int L> struct Sph;")
    for l in range(2, lmax + 1):
        K = engine_sph_matrix(l)
        w(f"template <> struct Sph<{l}> {{")
        w(f"  static __device__ __forceinline__ void apply(const double* x, double* y) {{")
        for u in range(K.shape[0]):
            terms = [(c, float(K[u, c])) for c in range(K.shape[1]) if K[u, c] != 0.0]
            expr = f"{terms[0][1]!r} * x[{terms[0][0]}]"
            for c, v in terms[1:]:
                expr = f"fma({v!r}, x[{c}], {expr})"
            w(f"    y[{u}] = {expr};")
        w("  }")
        w("};")
    w("template <int L> __device__ __forceinline__ double cnorm(int c);")
    for l in range(lmax + 1):
        vals = [1.0 / math.sqrt(_dfact(2 * a - 1) * _dfact(2 * b - 1) * _dfact(2 * c - 1))
                for a, b, c in comps(l)]
        w(f"template <> __device__ __forceinline__ double cnorm<{l}>(int c) {{")
        w(f"  constexpr double v[{len(vals)}] = {{{', '.join(repr(v) for v in vals)}}};")
        w("  return v[c];")
        w("}")


LIGHT_LIMIT = 170  # doubles of [e0|f0] + (ab|cd) one thread may hold


def is_light(c):
    """Classes evaluated by one thread in registers; the rest run on the cooperative kernel."""
    la, lb, lc, ld = c
    ne = sum(ncart(e) for e in range(la, la + lb + 1))
    nf = sum(ncart(f) for f in range(lc, lc + ld + 1))
    return ne * nf + ncart(la) * ncart(lb) * ncart(lc) * ncart(ld) <= LIGHT_LIMIT


def is_register(c):
    """Classes the register kernel runs: the light ones, and those whose kernel class holds up to
    102 accumulators raised by up to 600 operations ((fs|ds), (fp|ps), (fs|pp), (dd|ps), (pf|ps),
    (ff|ss) and the classes that flip to them).  Register against quadrature kernel on 8,000 to
    160,000 quartets: (sf|sd) 0.51 against 1.20 ms, (sf|pp) 0.46 and 1.18, (dd|sp) 0.68 and 1.33,
    (pf|sp) 0.85 and 1.41.  Beyond, the recursion's values spill at every primitive quartet: (pd|ds)
    (114, 723) 3.0 and 2.4 ms, (dp|ds) (96, 723) 0.36 and 0.28, (fs|fs) (100, 1296) 0.59 and 0.40,
    (dd|ds) (186, 1446) 3.7 and 1.1.  Lists of a hundred quartets lose 0.01 to 0.02 ms; the rule
    does not look at the list, on which a quartet's value must not depend."""
    if is_light(c):
        return True
    k = kernel_class(c)[0]
    acc = len(comps_range(k[0], k[0] + k[1])) * len(comps_range(k[2], k[2] + k[3]))
    return acc <= 102 and sum(k) <= 6 and best_vertical(*k).op_count() <= 600


# Largest total angular momentum for which the straight-line register code is emitted: the CPU
# tests execute it against the oracle for every class up to L = 8, and the device compiles it
# for classes up to L = 6 only (light classes and the (ab|ss) structs).  Executed on the CPU, the
# VRR/transfer code emitted for the L >= 11 heavy f classes disagrees with a direct recursion.
MAX_EMIT_L = 8


def emit_all(lmax, classes=None):
    if classes is None:
        classes = sorted({kernel_class(c)[0] for c in canonical_classes(lmax) if is_light(c)})
    lines = []
    w = lines.append
    w("// Generated by gen_eri.py — class-specialised ERI recursions. Do not edit by hand.")
    w("#pragma once")
    w(f"#define GBX_GEN_LMAX {lmax}")
    w("namespace gbx { namespace gen {")
    emit_sph_and_norms(w, lmax)
    w("template <int LA, int LB, int LC, int LD> struct Cls;")
    for la, lb, lc, ld in classes:
        if la + lb + lc + ld > MAX_EMIT_L:
            raise ValueError(f"straight-line register code is emitted up to L = {MAX_EMIT_L}; "
                             f"class {(la, lb, lc, ld)} runs the line, split or cooperative kernel")
        g = best_vertical(la, lb, lc, ld)
        h = HrrGen(la, lb, lc, ld)
        NE, NF = len(g.E), len(g.F)
        NAB, NCD = ncart(la) * ncart(lb), ncart(lc) * ncart(ld)
        w(f"template <> struct Cls<{la},{lb},{lc},{ld}> {{")
        w(f"  static constexpr int L = {la + lb + lc + ld}, NE = {NE}, NF = {NF}, "
          f"NAB = {NAB}, NCD = {NCD}, PRIM_OPS = {g.op_count()};")
        w("  template <typename R>")
        w("  static __device__ __forceinline__ void prim(const R* __restrict__ F, R PAx, R PAy, R PAz,")
        w("      R WPx, R WPy, R WPz, R o2z, R rz, R QCx, R QCy, R QCz, R WQx, R WQy, R WQz, R o2e,")
        w("      R re, R o2s, R* __restrict__ acc) {")
        body = []
        g.emit(body)
        for b in body:
            w("    " + b)
        w("    (void)PAx; (void)PAy; (void)PAz; (void)WPx; (void)WPy; (void)WPz; (void)o2z; (void)rz;")
        w("    (void)QCx; (void)QCy; (void)QCz; (void)WQx; (void)WQy; (void)WQz; (void)o2e; (void)re;")
        w("    (void)o2s;")
        w("  }")
        w("  static __device__ __forceinline__ void hrr(const double* __restrict__ acc,")
        w("      double ABx, double ABy, double ABz, double CDx, double CDy, double CDz,")
        w("      double* __restrict__ out) {")
        body = []
        h.emit(body)
        for b in body:
            w("    " + b)
        w("    (void)ABx; (void)ABy; (void)ABz; (void)CDx; (void)CDy; (void)CDz;")
        w("  }")
        w("};")
    w("}}  // namespace gbx::gen")
    return "\n".join(lines) + "\n"


def emit_sources(outdir, lmax):
    """Write eri_gen.cuh (register classes), their instantiation files, the cooperative programs
    of the heavy classes (coop_programs.cuh) and the class dispatch."""
    import os
    import gen_coop
    os.makedirs(outdir, exist_ok=True)

    def put(name, text):
        path = os.path.join(outdir, name)
        if not (os.path.exists(path) and open(path).read() == text):
            with open(path, "w") as f:
                f.write(text)

    every = canonical_classes(lmax)
    light = [c for c in every if is_light(c)]
    heavy = [c for c in every if not is_light(c)]
    reg_k = sorted({kernel_class(c)[0] for c in every if is_register(c)})
    rys_k = sorted({kernel_class(c)[0] for c in every if not is_register(c)})
    # the point-charge kernel uses the (ab|ss) structs of every pair class, heavy ones included
    one_e = [(la, lb, 0, 0) for la in range(lmax + 1) for lb in range(lmax + 1)]
    put("eri_gen.cuh", emit_all(lmax, reg_k + [c for c in one_e if c not in reg_k]))
    # heavy classes first (their cooperative kernels index the table by position), then the
    # light classes, whose programs only the multi-class queue kernel runs
    gen_coop.emit(heavy + light, os.path.join(outdir, "coop_programs.cuh"), n_heavy=len(heavy))
    files = []
    # spread the register classes over translation units of similar compile cost (code size)
    nbins = 12
    bins = [[] for _ in range(nbins)]
    load = [0] * nbins
    cost = {c: best_vertical(*c).op_count() + 4 * ncart(c[0]) * ncart(c[1]) * ncart(c[2]) * ncart(c[3])
            for c in reg_k}
    for c in sorted(reg_k, key=lambda c: -cost[c]):
        k = load.index(min(load))
        bins[k].append(c)
        load[k] += cost[c]
    for k, mine in enumerate(b for b in bins if b):
        lines = ["// Generated by gen_eri.py: explicit instantiations of the class kernels.",
                 '#include "../eri_kernels.cuh"',
                 '#include "../errors.h"',
                 "namespace gbx {",
                 "template <int LA, int LB, int LC, int LD>",
                 "int launch_t(const EriLaunch& a, int grid, cudaStream_t st) {",
                 "  if (a.fp32) eri_block<LA, LB, LC, LD, float><<<grid, kEriThreads, 0, st>>>(a);",
                 "  else if (a.potential)",
                 "    eri_block<LA, LB, LC, LD, double, true><<<grid, kEriThreads, 0, st>>>(a);",
                 "  else eri_block<LA, LB, LC, LD, double><<<grid, kEriThreads, 0, st>>>(a);",
                 '  return cuda_status(cudaGetLastError(), "eri class kernel launch");',
                 "}"]
        for c in mine:
            lines.append(f"template int launch_t<{c[0]}, {c[1]}, {c[2]}, {c[3]}>(const EriLaunch&, "
                         "int, cudaStream_t);")
        lines.append("}  // namespace gbx")
        name = f"eri_cls_{k:02d}.cu"
        put(name, "\n".join(lines) + "\n")
        files.append(name)
    import gen_lines
    lfiles, launchers = gen_lines.emit_sources(outdir, heavy)
    files += lfiles
    import gen_rys
    rfiles, rlaunchers = gen_rys.emit_sources(outdir, rys_k)
    files += rfiles
    lines = ["// Generated by gen_eri.py: (la,lb,lc,ld) -> class kernel launcher.",
             "#include <cstdlib>",
             "#include <cstring>",
             '#include "../coop.cuh"',
             '#include "../runtime.h"',
             "namespace gbx {",
             "template <int LA, int LB, int LC, int LD>",
             "int launch_t(const EriLaunch& a, int grid, cudaStream_t st);"]
    for c in reg_k:
        lines.append(f"extern template int launch_t<{c[0]}, {c[1]}, {c[2]}, {c[3]}>(const EriLaunch&, "
                     "int, cudaStream_t);")
    for c in heavy:
        lines.append(f"int {launchers[c]}(const EriLaunch& a, cudaStream_t st);")
    for c in rys_k:
        lines.append(f"int {rlaunchers[c]}(const EriLaunch& a, cudaStream_t st);")
    lines.append("// Heavy classes run the quadrature kernel (eri_rys) or, the smallest of them, the register kernel")
    lines.append("// (is_register in gen_eri.py); for both the block's variant knob selects the")
    lines.append("// line kernel (1) or (2) its group form or, for the classes that have one, the split kernel.")
    lines.append("// The split kernel, a thread per quartet, is faster on long lists of quartets with equal")
    lines.append("// primitive counts and slower on short or uneven ones.  Its time over the quadrature kernel's")
    lines.append("// on (pd|pp), (pd|sd), (pd|ds), (dp|pp), (dp|sd) and (dp|ds): 80,000 quartets 0.4 to 0.55 at")
    lines.append("// one primitive quartet each and 0.6 to 0.7 at 81, 16,000 quartets 0.5 to 0.8 and 0.7 to 1.0,")
    lines.append("// 700 quartets 1.7 and 1.7 to 2.6; of 1 to 256 primitive quartets, 16,000 quartets 1.3 to 1.8.")
    lines.append("// It is the default on none: its recursion loses digits (error of these classes' values")
    lines.append("// against 64-bit ones, split and quadrature: five atoms of s, p, d shells of one primitive")
    lines.append("// 7.2e-16 and 2.5e-16, of four 1.8e-14 and 4.0e-15; a 5-atom batch molecule 2.6e-14 and 1.5e-14).")
    lines.append("// GBX_HEAVY_KERNEL=interp selects the")
    lines.append("// program-interpreting cooperative kernel instead (read once per process).")
    lines.append("static bool heavy_interp() {")
    lines.append('  static const bool v = [] { const char* e = std::getenv("GBX_HEAVY_KERNEL");')
    lines.append('                             return e && std::strcmp(e, "interp") == 0; }();')
    lines.append("  return v;")
    lines.append("}")
    lines.append(f"int compiled_lmax() {{ return {lmax}; }}")
    lines.append("// Register and quadrature kernels: a pair of an s shell and another runs with the other")
    lines.append("// shell as the recursion centre (`flip`), so (sl| and (ls| share the kernels of (ls|.")
    lines.append("int launch_class(int la, int lb, int lc, int ld, const EriLaunch& args, int grid, "
                 "cudaStream_t st) {")
    lines.append("  EriLaunch a = args;")
    lines.append("  a.flip = (la == 0 && lb > 0 ? 1 : 0) + (lc == 0 && ld > 0 ? 2 : 0);")
    lines.append("  switch (((la * 8 + lb) * 8 + lc) * 8 + ld) {")

    def main(c):
        k = kernel_class(c)[0]
        return "launch_t<%d, %d, %d, %d>(a, grid, st)" % k if is_register(c) \
            else f"{rlaunchers[k]}(a, st)"
    for c in light:
        key = ((c[0] * 8 + c[1]) * 8 + c[2]) * 8 + c[3]
        lines.append(f"    case {key}: return {main(c)};")
    for j, c in enumerate(heavy):
        key = ((c[0] * 8 + c[1]) * 8 + c[2]) * 8 + c[3]
        lines.append(f"    case {key}: return heavy_interp() ? launch_coop({j}, a, st) : "
                     f"a.variant == 0 ? {main(c)} : {launchers[c]}(a, st);")
    lines.append("    default: break;")
    lines.append("  }")
    lines.append('  return set_error(GBX_ERR_UNSUPPORTED, "no kernel for class (%d %d|%d %d)", '
                 "la, lb, lc, ld);")
    lines.append("}")
    lines.append("}  // namespace gbx")
    put("eri_dispatch.cu", "\n".join(lines) + "\n")
    files.append("eri_dispatch.cu")
    return files


if __name__ == "__main__":
    if len(sys.argv) > 1 and sys.argv[1] == "--emit-dir":
        lmax = int(sys.argv[3]) if len(sys.argv) > 3 else 2
        print("\n".join(emit_sources(sys.argv[2], lmax)))
    else:
        lmax = int(sys.argv[1]) if len(sys.argv) > 1 else 3
        sys.stdout.write(emit_all(lmax))
