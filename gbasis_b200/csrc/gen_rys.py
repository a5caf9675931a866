"""Plans and tables of the quadrature kernel for heavy classes (``rys_kernel.cuh``).

Rys quadrature (Dupuis, Rys and King, J. Chem. Phys. 65, 111 (1976); King and Dupuis, J. Comput.
Phys. 21, 144 (1976)) writes one primitive quartet's [e0|f0] as a sum over n = L/2 + 1 points,

    [e0|f0] = sum_r Ix(ex, fx; r) Iy(ey, fy; r) Iz(ez, fz; r),

with 1-D tables I from a two-index recursion.  Over a contracted quartet the points of all its
primitive quartets form one contraction index k = (primitive quartet, point): a matrix product of
the "columns" XY[c][k] = Ix Iy, c = (ex, fx, ey, fy), with Iz[k][(ez, fz)], which the FP64 matrix
instruction m8n8k4 runs.  A column with s = ex + ey and t = fx + fy needs only the (ez, fz) with
la <= s + ez <= la + lb and lc <= t + fz <= lc + ld, so the columns are grouped by the z indices
they share.

``Plan`` groups a class's columns, orders each group's z indices by how many columns need them,
cuts columns and z indices into tiles of 8 and keeps, per tile of columns, the z tiles that it
needs; the grouping that takes the fewest matrix instructions wins.  The column tiles go to the
warps of a CTA.  ``root_tables`` makes the points and weights as piecewise polynomials of T.
"""
from __future__ import annotations

import functools
import hashlib
import itertools
import math
import os

from gen_lines import ncart, tet

KC = 32          # quadrature points per chunk: a lane each
KS = KC + 4      # row stride of the 1-D tables: 4 rows x 4 points cover the banks once
DEG = 11         # degree of the root polynomials on unit intervals of T
# above these T the Hermite limit x = h^2 / T, w = v / sqrt(T) holds to 4e-15 relative (measured
# against the discretised Stieltjes procedure below)
TMAX = {3: 56, 4: 60, 5: 65, 6: 70, 7: 76}


def n_points(cls):
    return sum(cls) // 2 + 1


def _partitions(l, top):
    """Consecutive classes of s = 0..top; s >= l share a class (their z ranges start at 0)."""
    for mask in range(1 << l):
        out = [[0]]
        for i in range(1, l + 1):
            if mask >> (i - 1) & 1:
                out.append([i])
            else:
                out[-1].append(i)
        out[-1] += list(range(l + 1, top + 1))
        yield out


class Plan:
    """tiles: per warp a list of (group, columns, z tiles): up to 8 columns (ex, fx, ey, fy) and the
    indices of the group's z tiles they need; ztiles: per group its z tiles, up to 8 (ez, fz) each.

    A column tile's operand is the product of 8 table rows of x and 8 of y, a lane per (row, point).
    Shared-memory bandwidth bounds the kernel, so the rows of one half tile (a 16-lane wavefront)
    are chosen from different banks where possible: table rows that differ modulo 4."""

    def __init__(self, la, lb, lc, ld, warps=None):
        self.cls = (la, lb, lc, ld)
        self.nE, self.nF = la + lb + 1, lc + ld + 1
        self.rf = self.nF | 1  # table rows per e (odd: neighbours in e and in f differ modulo 4)
        best = None
        for pe in _partitions(la, la + lb):
            for pf in _partitions(lc, lc + ld):
                groups = [self._group(S, T) for S in pe for T in pf]
                cost = self._cost(groups)
                if best is None or cost < best[0]:
                    best = (cost, groups)
        self.ztiles = [[self._order_z(z) for z in zt] for zt, _ in best[1]]
        tiles = []
        for g, (_, sets) in enumerate(best[1]):
            tiles += [(g, cols, zs) for cols, zs in self._sequence(sets)]
        self.n_mma = sum(len(t[2]) for t in tiles)
        self.warps = warps or (1 if self.n_mma <= 8 else 2 if self.n_mma <= 20 else
                               4 if self.n_mma <= 48 else 8)
        # contiguous shares of about the same number of matrix instructions
        self.tiles, done, total = [[] for _ in range(self.warps)], 0, self.n_mma
        for t in tiles:
            w = min(self.warps - 1, int((done + len(t[2]) / 2.0) * self.warps / total))
            self.tiles[w].append(t)
            done += len(t[2])
        self.load = [sum(len(t[2]) for t in ts) for ts in self.tiles]

    def row(self, e, f):
        return e * self.rf + f

    def needs(self, col):
        """The (ez, fz) a column is summed over."""
        la, lb, lc, ld = self.cls
        s, t = col[0] + col[2], col[1] + col[3]
        return [(ez, fz) for ez in range(max(0, la - s), la + lb - s + 1)
                for fz in range(max(0, lc - t), lc + ld - t + 1)]

    def _group(self, S, T):
        """z tiles of the columns with s in S and t in T, and {z tiles needed: columns}."""
        cols = [(ex, fx, s - ex, t - fx) for s in S for t in T
                for ex in range(s, -1, -1) for fx in range(t, -1, -1)]
        use = {}
        for c in cols:
            for z in self.needs(c):
                use[z] = use.get(z, 0) + 1
        zs = sorted(use, key=lambda z: (-use[z], z))
        tile_of = {z: i // 8 for i, z in enumerate(zs)}
        sets = {}
        for c in cols:
            sets.setdefault(tuple(sorted({tile_of[z] for z in self.needs(c)})), []).append(c)
        return [zs[i:i + 8] for i in range(0, len(zs), 8)], sets

    @staticmethod
    def _tiles_of(sets):
        """(number of column tiles, matrix instructions) when the sets are cut one after another,
        those of the most z tiles first."""
        order = [m for m in sorted(sets, key=lambda m: (len(m), m), reverse=True) for _ in sets[m]]
        parts = [order[i:i + 8] for i in range(0, len(order), 8)]
        return len(parts), sum(len(set().union(*p)) for p in parts)

    @classmethod
    def _cost(cls, groups):
        """About the SM cycles of a quadrature point: matrix instructions (4 cycles per 4 points)
        or shared-memory wavefronts (2 loads per column tile, 1 per z tile, 2 wavefronts each)."""
        n = [cls._tiles_of(sets) for _, sets in groups]
        mma = sum(m for _, m in n)
        loads = sum(4 * t + 2 * len(z) for (t, _), (z, _) in zip(n, groups)) / 4.0
        return max(1.2 * loads, mma) + 0.3 * min(1.2 * loads, mma)

    def _wavefronts(self, rows):
        """Wavefronts of a load of 8 table rows x 4 points: per half tile, the most different rows
        in one bank group."""
        n = 0
        for half in (rows[:4], rows[4:]):
            d = set(half)
            n += max([sum(1 for r in d if r % 4 == m) for m in range(4)] + [1])
        return n

    def _order_z(self, zt):
        """The z indices of a tile in the order of the fewest wavefronts."""
        rows = {z: self.row(*z) for z in zt}
        best = None
        for half in itertools.combinations(zt, min(4, len(zt))):
            order = list(half) + [z for z in zt if z not in half]
            n = self._wavefronts([rows[z] for z in order])
            if best is None or n < best[0]:
                best = (n, order)
        return best[1]

    def _sequence(self, sets):
        """The group's columns cut into tiles, the sets of the most z tiles first; a tile takes, of
        the next columns, those whose table rows clash least within its half tiles."""
        left = [(m, c) for m in sorted(sets, key=lambda m: (len(m), m), reverse=True)
                for c in sets[m]]
        tiles = []
        while left:
            zs = set().union(*(m for m, _ in left[:8]))
            pick = []
            for r in range(min(8, len(left))):
                half = pick[4 * (r // 4):]

                def clash(c):
                    return sum((h[a], h[a + 1]) != (c[a], c[a + 1]) and
                               (self.row(*h[a:a + 2]) - self.row(*c[a:a + 2])) % 4 == 0
                               for a in (0, 2) for h in half)
                cand = [mc for mc in left[:32] if zs.issuperset(mc[0])]
                m, c = min(cand, key=lambda mc: clash(mc[1]))
                pick.append(c)
                left.remove((m, c))
            tiles.append((pick, sorted(zs)))
        return tiles

    def wavefronts(self):
        """Shared-memory wavefronts of the matrix products per quadrature point."""
        n = 0
        for ts in self.tiles:
            n += sum(self._wavefronts([self.row(*v) for v in self.ztiles[g][z]])
                     for g, z in {(g, z) for g, _, zs in ts for z in zs})
            n += sum(self._wavefronts([self.row(*c[a:a + 2]) for c in cols])
                     for _, cols, _ in ts for a in (0, 2))
        return n / 4.0

    def acc_index(self, col, z, nfs):
        """Place of a target in ACC (row stride nfs), or -1 when the column does not need z."""
        if z not in self.needs(col):
            return -1
        (ex, fx, ey, fy), (ez, fz) = col, z

        def comp(lo, x, y, z_):
            return tet(x + y + z_) - tet(lo) + (y + z_) * (y + z_ + 1) // 2 + z_
        return comp(self.cls[0], ex, ey, ez) * nfs + comp(self.cls[2], fx, fy, fz)


@functools.lru_cache(maxsize=None)
def plan(cls):
    return Plan(*cls)


# ------------------------------------------------------------------------------ points
def _legendre(n):
    """Gauss-Legendre points and weights on [0, 1] in extended precision."""
    import numpy as np
    ld = np.longdouble
    x = np.polynomial.legendre.leggauss(n)[0].astype(ld)
    for last in (0, 0, 0, 1):
        p0, p1 = np.ones_like(x), x.copy()
        for k in range(2, n + 1):
            p0, p1 = p1, ((2 * k - 1) * x * p1 - (k - 1) * p0) / ld(k)
        dp = n * (x * p1 - p0) / (x * x - 1)
        if not last:
            x = x - p1 / dp
    return (x + 1) / 2, 1 / ((1 - x * x) * dp * dp)


def rys_points(n, T):
    """Points x_r (in t^2) and weights of the n-point rule for exp(-T t^2) on [0, 1], for an array
    of T, in extended precision: discretised Stieltjes procedure on 100 Gauss-Legendre points,
    eigenvalues of the Jacobi matrix polished by Newton steps, Christoffel weights."""
    import numpy as np
    ld = np.longdouble
    T = np.asarray(T, dtype=ld).reshape(-1)
    t, tw = _legendre(100)
    s = t * t
    W = tw[None, :] * np.exp(-T[:, None] * s[None, :])
    p0, p1 = np.zeros_like(W), np.ones_like(W)
    al, be, norm = [], [], None
    for k in range(n):
        q = (W * p1 * p1).sum(1)
        a = (W * p1 * p1 * s).sum(1) / q
        b = q if norm is None else q / norm
        norm = q
        al.append(a)
        be.append(b)
        p0, p1 = p1, (s - a[:, None]) * p1 - (b[:, None] * p0 if k else 0)
    J = np.zeros((len(T), n, n))
    for k in range(n):
        J[:, k, k] = al[k]
        if k:
            J[:, k, k - 1] = J[:, k - 1, k] = np.sqrt(be[k])
    x = np.linalg.eigvalsh(J).astype(ld)

    def polys(x):
        q0, q1, d0, d1 = np.zeros_like(x), np.ones_like(x), np.zeros_like(x), np.zeros_like(x)
        total, h = np.zeros_like(x), np.ones(len(T), dtype=ld)
        for k in range(n):
            h = h * be[k]
            total = total + q1 * q1 / h[:, None]
            b = be[k][:, None] if k else 0
            q0, q1, d0, d1 = q1, (x - al[k][:, None]) * q1 - b * q0, d1, \
                q1 + (x - al[k][:, None]) * d1 - b * d0
        return q1, d1, total
    for _ in range(4):
        q, d, _t = polys(x)
        x = x - q / d
    return x, 1 / polys(x)[2]


def root_table(n):
    """Doubles of the n-point table: per unit interval [i, i + 1) of T the coefficients of the
    polynomials in u = 2 (T - i) - 1, two degrees at a time (x, w of degree 2d, x, w of degree
    2d + 1: one 32-byte load) for each point; then the Hermite limit (x T, w sqrt(T), 0, 0) of each
    point."""
    import numpy as np
    ld = np.longdouble
    k = np.arange(DEG + 1)
    u = np.cos((k.astype(ld) + ld(0.5)) / (DEG + 1) * np.arccos(ld(-1)))
    T = (np.arange(TMAX[n], dtype=ld)[:, None] + (u[None, :] + 1) / 2).reshape(-1)
    x, w = rys_points(n, T)
    y = np.stack([x, w], -1).reshape(TMAX[n], DEG + 1, n, 2)
    # interpolation at the Chebyshev points: Newton's divided differences, expanded to powers
    coef = np.zeros_like(y)
    dd = y.copy()
    for j in range(1, DEG + 1):
        dd[:, j:] = (dd[:, j:] - dd[:, j - 1:-1]) / (u[j:] - u[:-j])[None, :, None, None]
    for j in range(DEG, -1, -1):  # coef <- coef * (u - u_j) + dd_j
        up = np.zeros_like(coef)
        up[:, 1:] = coef[:, :-1]
        coef = up - u[j] * coef
        coef[:, 0] += dd[:, j]
    big = ld(400)
    hx, hw = rys_points(n, [big])
    tail = np.stack([hx[0] * big, hw[0] * np.sqrt(big), 0 * big * hx[0], 0 * big * hx[0]], -1)
    pairs = coef.reshape(TMAX[n], (DEG + 1) // 2, 2, n, 2).transpose(0, 1, 3, 2, 4)
    return [float(v) for v in np.concatenate([pairs.reshape(-1), tail.reshape(-1)])]


def table_offset(n):
    return sum((TMAX[m] * (DEG + 1) + 2) * m * 2 for m in TMAX if m < n)


# ------------------------------------------------------------------------------ code
def _tag(cls):
    return "".join(str(v) for v in cls)


def emit_class(cls, tab_name, tab_off):
    """Struct RysCls_<tag> (the plan's matrix products); returns (code, table words).

    Table words: per column tile 8 rows (byte offsets of the x row, and of the y row << 16, in the
    tables), per z tile 8 offsets, per matrix instruction 32 lanes x two 16-bit ACC places."""
    p = plan(cls)
    la, lb, lc, ld = cls
    nfs = (tet(lc + ld + 1) - tet(lc)) | 1
    ts = p.nE * p.rf * KS
    words, gemm, store = [], [], []

    def put(vals):
        at = tab_off + len(words)
        words.extend(vals)
        return at

    def z_words(zt):
        rows = [8 * (2 * ts + p.row(*z) * KS) for z in zt]
        return rows + [rows[0]] * (8 - len(rows))

    def col_words(rows):
        return [8 * p.row(ex, fx) * KS | 8 * (ts + p.row(ey, fy) * KS) << 16 for ex, fx, ey, fy in rows]
    z_at = {}
    for tiles in p.tiles:
        decl, zload, body, st, n = [], [], [], [], 0
        for g, z in sorted({(g, z) for g, _, zs in tiles for z in zs}):
            if (g, z) not in z_at:
                z_at[g, z] = put(z_words(p.ztiles[g][z]))
            decl.append(f"const unsigned z{g}_{z} = __ldg({tab_name} + {z_at[g, z]} + r);")
            zload.append(f"const double b{g}_{z} = rys_ld(t, z{g}_{z});")
        for i, (g, cols, zs) in enumerate(tiles):
            rows = cols + [cols[-1]] * (8 - len(cols))
            decl.append(f"const unsigned c{i} = __ldg({tab_name} + {put(col_words(rows))} + r);")
            body.append(f"const double v{i} = rys_ld(t, c{i} & 0xffffu) * rys_ld(t, c{i} >> 16);")
            for z in zs:
                zt = p.ztiles[g][z]
                vals = []
                for lane in range(32):
                    at = []
                    for h in range(2):
                        row, k = lane >> 2, 2 * (lane & 3) + h
                        a = p.acc_index(cols[row], zt[k], nfs) if row < len(cols) and k < len(zt) else -1
                        at.append(a & 0xffff)
                    vals.append(at[0] | at[1] << 16)
                body.append(f"rys_mma(acc[{n}], acc[{n + 1}], v{i}, b{g}_{z});")
                st.append(f"rys_put(__ldg({tab_name} + {put(vals)} + lane), acc[{n}], acc[{n + 1}], ACC);")
                n += 2
        gemm.append(decl + ["#pragma unroll 2", "for (int k = 0; k < kcp; k += 4, t += 32) {"]
                    + ["  " + ln for ln in zload + body] + ["}"])
        store.append(st)

    def switch(parts):
        if p.warps == 1:
            return ["    " + ln for ln in parts[0]]
        out = ["    switch (wq) {"]
        for w, part in enumerate(parts):
            out.append(f"      {'default' if w == p.warps - 1 else f'case {w}'}: {{")
            out += ["        " + ln for ln in part] + ["        break;", "      }"]
        return out + ["    }"]
    kacc = 2 * max(p.load)
    code = [f"struct RysCls_{_tag(cls)} {{",
            f"  static constexpr int LA = {la}, LB = {lb}, LC = {lc}, LD = {ld}, L = {sum(cls)};",
            f"  static constexpr int kN = {n_points(cls)}, kW = {p.warps}, kAcc = {kacc};",
            "  static __device__ __forceinline__ void gemm(int wq, int lane, const double* T, int kcp,",
            "                                              double* acc) {",
            "    const int r = lane >> 2;",
            "    const char* t = reinterpret_cast<const char*>(T + (lane & 3));",
            *switch(gemm),
            "  }",
            "  static __device__ __forceinline__ void store(int wq, int lane, const double* acc,",
            "                                               double* ACC) {",
            *switch(store),
            "  }",
            "};"]
    return "\n".join(code), words


def _put(path, text):
    if not (os.path.exists(path) and open(path).read() == text):
        with open(path, "w") as f:
            f.write(text)


def emit_sources(outdir, classes, nfiles=12):
    """Write rys_XX.cu (instantiations) and rys_tables.cu (points and weights); returns the file
    names and {class: launcher name}."""
    cost = {c: plan(c).n_mma + sum(ncart(v) for v in c) for c in classes}
    bins, load = [[] for _ in range(nfiles)], [0.0] * nfiles
    for c in sorted(classes, key=lambda c: -cost[c]):
        k = load.index(min(load))
        bins[k].append(c)
        load[k] += cost[c]
    files, launchers = [], {}
    for k, mine in enumerate(b for b in bins if b):
        words, structs = [], []
        for c in sorted(mine):
            code, w = emit_class(c, "kRysDesc", len(words))
            structs.append(code)
            words += w
        out = ["// Generated by gen_rys.py: quadrature kernels of heavy classes.",
               '#include "../rys_kernel.cuh"',
               "namespace gbx {",
               f"__device__ const unsigned kRysDesc[{len(words)}] = {{"
               + ", ".join(f"{v}u" for v in words) + "};"]
        out += structs
        for c in sorted(mine):
            launchers[c] = f"launch_rys_{_tag(c)}"
            out.append(f"int {launchers[c]}(const EriLaunch& a, cudaStream_t st) "
                       f"{{ return launch_rys_t<RysCls_{_tag(c)}>(a, st); }}")
        out.append("}  // namespace gbx")
        name = f"rys_{k:02d}.cu"
        _put(os.path.join(outdir, name), "\n".join(out) + "\n")
        files.append(name)
    path = os.path.join(outdir, "rys_tables.cu")
    # making the table takes seconds: kept while this generator is the one that made it
    with open(__file__, "rb") as f:
        made_by = hashlib.sha256(f.read()).hexdigest()[:16]
    head = (f"// Generated by gen_rys.py ({made_by}): points and weights, degree {DEG} on unit intervals, "
            f"two degrees a row, ranges {TMAX}.")
    if not (os.path.exists(path) and open(path).readline().rstrip("\n") == head):
        vals = [v for n in TMAX for v in root_table(n)]
        text = "\n".join([
            head, '#include "../rys_kernel.cuh"', "namespace gbx {",
            f"__device__ __align__(32) const double kRysTable[{len(vals)}] = {{",
            ",\n".join(", ".join(v.hex() for v in vals[i:i + 6]) for i in range(0, len(vals), 6)),
            "};",
            "// Address of the table on the current device (resolved once per device).",
            "int rys_table(const double** out) {",
            "  static std::atomic<const double*> at[64];",
            "  int dev = 0;",
            '  int s = cuda_status(cudaGetDevice(&dev), "cudaGetDevice");',
            "  if (s) return s;",
            "  if (dev < 0 || dev >= 64) return set_error(GBX_ERR_INVALID, \"bad device %d\", dev);",
            "  const double* p = at[dev].load();",
            "  if (!p) {",
            "    void* q = nullptr;",
            '    if ((s = cuda_status(cudaGetSymbolAddress(&q, kRysTable), "quadrature table"))) return s;',
            "    p = static_cast<const double*>(q);",
            "    at[dev].store(p);",
            "  }",
            "  *out = p;",
            "  return GBX_OK;",
            "}",
            "}  // namespace gbx"]) + "\n"
        _put(path, text)
    files.append("rys_tables.cu")
    return files, launchers
