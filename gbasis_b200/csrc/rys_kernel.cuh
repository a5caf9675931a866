// Quadrature kernel for heavy classes: a CTA of C::kW warps per contracted quartet.
//
// [e0|f0] of a primitive quartet is a sum over n = L/2 + 1 Rys points of Ix Iy Iz (plan and
// tables: gen_rys.py), so the points of all primitive quartets of a contracted quartet form one
// long contraction index k.  Per chunk of up to kRysKC points:
//   points: a warp per chunk, lane k its point's abscissa and weight (piecewise polynomials of T)
//           and the recursion coefficients PR[.][k];
//   tables: threads (axis, k) run the two-index recursion and write I[axis][(e, f)][k];
//   sums:   the warps run the columns' matrix products X Y * Z over the chunk on the FP64 matrix
//           instruction, sums in registers (C::gemm), beside the next chunk's tables where two
//           table buffers fit.
// The tables have k innermost: a matrix operand is 8 table rows x 4 points.  After the last chunk
// the sums go to shared memory ACC[e][f] once and the whole CTA runs the tail: horizontal
// recursions, transforms, store / Schwarz maximum / Coulomb contributions.
//
// What bounds it: shared memory and the matrix pipe together (l1tex data pipe 73 to 85 %, FP64
// matrix pipe 53 to 58 % busy on 3,000 quartets of (dd|dd) and (df|fs) of 81 primitive quartets;
// (ff|ff) 52 and 49 %), with the barriers between the phases.  The matrix instruction is there for its operand reuse:
// the same sums with a lane per column and FMAs read 8 shared values for every 9 FMAs and took 1.4
// to 2 times longer.  Measured on the 20-atom chain's first 10 atoms (spherical, unique integrals,
// blocks one after another), the line or split kernel before against this one: all heavy classes
// 97.6 -> 17.9 ms; (pf|sf) 5.05 -> 0.89, (df|pf) 5.24 -> 0.50, (ff|ff) 2.03 -> 0.14, (pd|pd) 2.38
// -> 0.32 ms (12.3 TF/s of algorithmic work, 36 % of the FP64 rate).  The points of kW chunks at a
// time (their latency once, not per chunk), the second table buffer, 32-byte table loads and the
// element offsets of the store kept per row and column then took 3,000 to 20,000 quartets per class
// of 81 primitive quartets from 33,400 to 29,200 SM cycles a quartet on (dd|dd), 30,400 to 27,500
// on (df|sf), 6,640 to 6,140 on (pd|sd) (all classes: 8 % less; of 16 primitive quartets 6 % less,
// of one 2 % more).  Error against 64-bit
// reference values: tensors of the 60-molecule batch 2.0e-13 before, 2.8e-14 now.
//
// Mathematics: [e0|f0] as gbasis/integrals/_two_elec_int.py:293-547 defines it (the engine's other
// kernels build the same values by vertical recursions), :549-812 (horizontal
// recursion, component norm), gbasis/base_four_symm.py:195-349 (norm_cont, spherical transform).
#pragma once
#include <algorithm>
#include <atomic>

#include "eri_kernels.cuh"  // gen::Sph, gen::cnorm
#include "errors.h"
#include "gbx_common.cuh"

namespace gbx {

constexpr int kRysKC = 32;           // quadrature points per chunk
constexpr int kRysKS = kRysKC + 4;   // row stride of the tables: 4 rows x 4 points cover the banks
constexpr int kRysDeg = 11;          // degree of the point polynomials (unit intervals of T)
constexpr long long kRysMaxSmem = 227 * 1024;

__host__ __device__ constexpr int rys_tmax(int n) {
  return n == 3 ? 56 : n == 4 ? 60 : n == 5 ? 65 : n == 6 ? 70 : 76;
}
// Doubles before the n-point table.
__host__ __device__ constexpr int rys_table_offset(int n) {
  int o = 0;
  for (int m = 3; m < n; ++m) o += (rys_tmax(m) * (kRysDeg + 1) + 2) * m * 2;
  return o;
}
int rys_table(const double** out);

__host__ __device__ constexpr int rys_tet(int k) { return k * (k + 1) * (k + 2) / 6; }
// Components of total angular momentum lo..hi.
__host__ __device__ constexpr int rys_ncomp(int lo, int hi) { return rys_tet(hi + 1) - rys_tet(lo); }

// A 32-byte load of a table row (the address a multiple of 32 bytes).
struct RysRow4 {
  double x0, w0, x1, w1;
};
__device__ __forceinline__ RysRow4 rys_row(const double* p) {
  RysRow4 r;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(r.x0), "=d"(r.w0), "=d"(r.x1), "=d"(r.w1)
      : "l"(p));
  return r;
}

// Abscissa (in t^2) and weight of point r of the N-point rule for exp(-T t^2) on [0, 1].  A chunk's
// lanes gather from as many intervals as it has primitive quartets, so the loads cost wavefronts by
// count: two degrees of a point's pair of polynomials come in one 32-byte load.
template <int N>
__device__ __forceinline__ double2 rys_point(double T, int r, const double* __restrict__ tab) {
  constexpr int TM = rys_tmax(N), ND = (kRysDeg + 1) / 2;
  if (T < (double)TM) {
    const int i = (int)T;
    const double u = fma(2.0, T - (double)i, -1.0);
    const double* __restrict__ c = tab + ((size_t)i * ND * N + r) * 4;
    RysRow4 g = rys_row(c + (ND - 1) * N * 4);
    double x = fma(g.x1, u, g.x0), w = fma(g.w1, u, g.w0);
#pragma unroll
    for (int d = ND - 2; d >= 0; --d) {
      g = rys_row(c + d * N * 4);
      x = fma(fma(x, u, g.x1), u, g.x0);
      w = fma(fma(w, u, g.w1), u, g.w0);
    }
    return make_double2(x, w);
  }
  const RysRow4 h = rys_row(tab + ((size_t)TM * ND * N + r) * 4);
  const double q = rsqrt(T);
  return make_double2(h.x0 * (q * q), h.w0 * q);
}

// Rows of the per-point coefficients.
enum RysRow { kB00, kB10, kB01, kC0, kD0 = kC0 + 3, kWt = kD0 + 3, kRysRows };

// One axis of one point: I(0,0) = scale, I(e+1,0) = C I(e,0) + e B10 I(e-1,0),
// I(e,f+1) = D I(e,f) + f B01 I(e,f-1) + e B00 I(e-1,f), into out[(e * RF + f) * kRysKS].
template <int NE1, int NF1, int RF>
__device__ __forceinline__ void rys_axis(double C, double D, double B00, double B10, double B01,
                                         double scale, double* __restrict__ out) {
  double a0[NE1], a1[NE1];
  a1[0] = scale;
#pragma unroll
  for (int e = 1; e < NE1; ++e)
    a1[e] = e == 1 ? C * a1[0] : fma((double)(e - 1) * B10, a1[e - 2], C * a1[e - 1]);
#pragma unroll
  for (int e = 0; e < NE1; ++e) {
    out[e * RF * kRysKS] = a1[e];
    a0[e] = 0.0;
  }
#pragma unroll
  for (int f = 1; f < NF1; ++f) {
    double nw[NE1];
#pragma unroll
    for (int e = 0; e < NE1; ++e) {
      double v = D * a1[e];
      if (f > 1) v = fma((double)(f - 1) * B01, a0[e], v);
      if (e > 0) v = fma((double)e * B00, a1[e - 1], v);
      nw[e] = v;
    }
#pragma unroll
    for (int e = 0; e < NE1; ++e) {
      out[(e * RF + f) * kRysKS] = nw[e];
      a0[e] = a1[e];
      a1[e] = nw[e];
    }
  }
}

// FP64 matrix instruction m8n8k4: C[row][col] += sum_k A[row][k] B[k][col]; lane l holds A[l / 4]
// [l % 4], B[l % 4][l / 4] and C[l / 4][2 (l % 4) + (0, 1)].
__device__ __forceinline__ void rys_mma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// A table value at a byte offset.
__device__ __forceinline__ double rys_ld(const char* t, unsigned off) {
  return *reinterpret_cast<const double*>(t + off);
}

// A matrix instruction's two sums to their places in ACC (0xffff: not a target).
__device__ __forceinline__ void rys_put(unsigned at, double c0, double c1, double* __restrict__ ACC) {
  if ((at & 0xffffu) != 0xffffu) ACC[at & 0xffffu] = c0;
  if ((at >> 16) != 0xffffu) ACC[at >> 16] = c1;
}

// Sizes of a class's kernel.
template <class C>
struct RysDims {
  static constexpr int NE1 = C::LA + C::LB + 1, NF1 = C::LC + C::LD + 1;
  static constexpr int NE = rys_ncomp(C::LA, C::LA + C::LB), NF = rys_ncomp(C::LC, C::LC + C::LD);
  static constexpr int NFs = NF | 1;  // row stride of ACC (odd: lanes on consecutive rows)
  static constexpr int NCA = ncart(C::LA), NCB = ncart(C::LB), NCC = ncart(C::LC), NCD = ncart(C::LD);
  static constexpr int NAB = NCA * NCB, NKET = NCC * NCD;
  static constexpr int HS = C::LD == 0 ? NFs : (NKET | 1);  // row stride of [e0|cd]
  static constexpr int NT = 32 * C::kW;
  // registers for 16 resident warps per SM where the sums leave room, else 12 or 8
  static constexpr int kMinCtas = (C::kAcc <= 24 ? 16 : C::kAcc <= 36 ? 12 : 8) / C::kW;
  static constexpr int RF = NF1 | 1;             // table rows per e
  static constexpr int TS = NE1 * RF * kRysKS;   // one axis's table
  // shared memory (doubles): ACC, overlaid after the ket recursion by the bra step's block of
  // columns; then the tables and coefficients, overlaid by [e0|cd]
  static constexpr int kAccSize = NE * NFs > 3 * NAB ? NE * NFs : 3 * NAB;
  static constexpr int kAccEven = (kAccSize + 1) & ~1;
  static constexpr int kHf = C::LD == 0 ? 0 : NE * HS;
  static constexpr int smem_of(int buffers) {
    const int t = buffers * 3 * TS + C::kW * kRysRows * kRysKS;
    return kAccEven + (t > kHf ? t : kHf);
  }
  // two table buffers where the CTAs that the registers allow still fit (228 KB per SM; 1 KB and
  // the shell data of each CTA beside it)
  static constexpr int kBuf =
      (long long)kMinCtas * (smem_of(2) * 8 + 16 * (NAB + NKET) + 2 * 1024) <= 228 * 1024 && C::kW > 1 ? 2 : 1;
  static constexpr int kSmem = smem_of(kBuf);
  // [e0|cd] of classes whose ket pair has no second angular momentum is ACC itself: the bra
  // step's block then sits in the tables' place
  static constexpr int kBlkSize = C::LD == 0 ? kSmem - kAccEven : kAccSize;
};

// Horizontal recursion onto a shell of angular momentum L for one component c of the first shell
// (angular momentum L0): values [c + j], |j| <= L, read at in[index * stride] (components of total
// L0.. in order), shifted along each axis in turn, in place:
// (c, b) = sum_k binom(b, k) AB^(b-k) [c + k].  out: the ncart(L) components (c, b).
template <int L0, int L>
__device__ __forceinline__ void rys_hrr(const double* __restrict__ in, int stride, int c, double ABx,
                                        double ABy, double ABz, double* __restrict__ out) {
  const int u = (c >= 1) + (c >= 3) + (c >= 6);  // y + z of component c (at most 10 components)
  const int zc = c - u * (u + 1) / 2;
  double v[L + 1][L + 1][L + 1];
#pragma unroll
  for (int jx = 0; jx <= L; ++jx)
#pragma unroll
    for (int jy = 0; jy <= L - jx; ++jy)
#pragma unroll
      for (int jz = 0; jz <= L - jx - jy; ++jz) {
        const int a = u + jy + jz;
        v[jx][jy][jz] =
            in[(rys_tet(L0 + jx + jy + jz) - rys_tet(L0) + a * (a + 1) / 2 + zc + jz) * stride];
      }
#pragma unroll
  for (int jy = 0; jy <= L; ++jy)
#pragma unroll
    for (int jz = 0; jz <= L - jy; ++jz)
#pragma unroll
      for (int s = 1; s <= L - jy - jz; ++s)
#pragma unroll
        for (int j = L - jy - jz; j >= s; --j) v[j][jy][jz] = fma(ABx, v[j - 1][jy][jz], v[j][jy][jz]);
#pragma unroll
  for (int bx = 0; bx <= L; ++bx)
#pragma unroll
    for (int jz = 0; jz <= L - bx; ++jz)
#pragma unroll
      for (int s = 1; s <= L - bx - jz; ++s)
#pragma unroll
        for (int j = L - bx - jz; j >= s; --j) v[bx][j][jz] = fma(ABy, v[bx][j - 1][jz], v[bx][j][jz]);
#pragma unroll
  for (int bx = 0; bx <= L; ++bx)
#pragma unroll
    for (int by = 0; by <= L - bx; ++by)
#pragma unroll
      for (int s = 1; s <= L - bx - by; ++s)
#pragma unroll
        for (int j = L - bx - by; j >= s; --j) v[bx][by][j] = fma(ABz, v[bx][by][j - 1], v[bx][by][j]);
  int k = 0;
#pragma unroll
  for (int bx = L; bx >= 0; --bx)
#pragma unroll
    for (int by = L - bx; by >= 0; --by) out[k++] = v[bx][by][L - bx - by];
}

struct RysArgs {
  EriLaunch a;
  const double* tab;  // rys_table()
};

// Per-quartet shell data in shared memory: A, B, C, D.
struct RysShells {
  double scl[4][kMaxCart];
  int pos[4][kMaxCart];
  int func[4], nint[4], nout[4];
};

template <int NW>
__device__ __forceinline__ void rys_sync() {
  if constexpr (NW == 1) __syncwarp();
  else __syncthreads();
}

// Points of primitive quartets p0, p0 + 1, ... of a quartet with nk ket primitive pairs (kc points,
// kpp per primitive quartet): lane k writes its point's recursion coefficients PR[.][k], zeros up to a
// multiple of 4 points.
template <class C>
__device__ __forceinline__ void rys_points(const EriLaunch& a, const PairDev& P, const PairDev& Q,
                                           const double* __restrict__ tab, int p0, int kc, int kpp,
                                           int lane, double* __restrict__ PR) {
  constexpr int N = C::kN;
  if (lane >= ((kc + 3) & ~3)) return;
  double* const pr = PR + lane;
  if (lane >= kc) {
#pragma unroll
    for (int i = 0; i < kRysRows; ++i) pr[i * kRysKS] = 0.0;
    return;
  }
  const int pi = kpp == N ? lane / N : lane / (2 * N), r2 = lane - pi * kpp, r = r2 < N ? r2 : r2 - N;
  const int nk = Q.nprim, ip = (p0 + pi) / nk, jq = p0 + pi - ip * nk;
  PrimPair bp = a.prims[P.prim_off + ip], kp = a.prims[Q.prim_off + jq];
  // a flipped pair's recursion centre is its second shell: P - B = (P - A) + (A - B)
  if constexpr (C::LB == 0 && C::LA > 0) {
    if (a.flip & 1) { bp.Xx += P.ABx; bp.Xy += P.ABy; bp.Xz += P.ABz; }
  }
  if constexpr (C::LD == 0 && C::LC > 0) {
    if (a.flip & 2) { kp.Xx += Q.ABx; kp.Xy += Q.ABy; kp.Xz += Q.ABz; }
  }
  const double rs = rsqrt(bp.zeta + kp.zeta), inv = rs * rs;
  const double PQx = bp.Px - kp.Px, PQy = bp.Py - kp.Py, PQz = bp.Pz - kp.Pz;
  const double rz = kp.zeta * inv, re = bp.zeta * inv;  // rho / zeta, rho / eta
  const double rho = bp.zeta * rz;
  double T = fmax(rho * fma(PQx, PQx, fma(PQy, PQy, PQz * PQz)), 0.0);
  double pref = bp.C * kp.C * rs, sx = 1.0;
  if (a.potential == 1 || r2 >= N) {
    // erf(omega r)/r: points and weights at s T, scaled by s and sqrt(s); erfc: subtracted
    const double w2 = a.omega * a.omega;
    sx = w2 / (w2 + rho);
    T *= sx;
    pref *= a.potential == 1 ? sqrt(sx) : -sqrt(sx);
  }
  const double2 xw = rys_point<N>(T, r, tab);
  const double x = xw.x * sx;
  const double o2z = 0.5 * bp.izeta, o2e = 0.5 * kp.izeta, xz = x * rz, xe = x * re;
  pr[kB00 * kRysKS] = 0.5 * x * inv;
  pr[kB10 * kRysKS] = fma(-xz, o2z, o2z);
  pr[kB01 * kRysKS] = fma(-xe, o2e, o2e);
  pr[kC0 * kRysKS] = fma(-xz, PQx, bp.Xx);
  pr[(kC0 + 1) * kRysKS] = fma(-xz, PQy, bp.Xy);
  pr[(kC0 + 2) * kRysKS] = fma(-xz, PQz, bp.Xz);
  pr[kD0 * kRysKS] = fma(xe, PQx, kp.Xx);
  pr[(kD0 + 1) * kRysKS] = fma(xe, PQy, kp.Xy);
  pr[(kD0 + 2) * kRysKS] = fma(xe, PQz, kp.Xz);
  pr[kWt * kRysKS] = pref * xw.y;
}

template <class C>
__global__ void __launch_bounds__(32 * C::kW, RysDims<C>::kMinCtas) eri_rys(const RysArgs A) {
  using D = RysDims<C>;
  constexpr int N = C::kN, NT = D::NT, NW = C::kW, LA = C::LA, LB = C::LB, LC = C::LC, LD = C::LD;
  extern __shared__ __align__(16) double smem[];
  __shared__ RysShells S;
  __shared__ long long s_next[2];
  // mode 0: element offsets and scales of the block's rows (a, b) and columns (c, d)
  __shared__ long long s_ro[D::NAB], s_co[D::NKET];
  __shared__ double s_rs[D::NAB], s_cs[D::NKET];
  const EriLaunch& a = A.a;
  const int tid = threadIdx.x, lane = tid & 31, wq = tid >> 5;
  double* const ACC = smem;
  double* const T = smem + D::kAccEven;
  double* const PR = T + D::kBuf * 3 * D::TS;
  double* const HF = LD == 0 ? ACC : T;
  double* const BLK = LD == 0 ? T : ACC;
  const double* __restrict__ tab = A.tab + rys_table_offset(N);
  const long long count = a.work_count ? (long long)(*a.work_count) : a.nwork;
  const bool schwarz = a.mode == 1, coulomb = a.mode == 2;
  double* const DCD = smem + D::kSmem;   // Coulomb mode: D[c][d] of the ket block,
  double* const DAB = DCD + D::NKET;     // D[a][b] of the bra block,
  double* const VAB = DAB + D::NAB;      // sum_cd (ab|cd) D[c][d]
  long long w = blockIdx.x;
  int turn = 0;
  if (a.ticket) {  // quartets from the launch's counter; the next draw overlaps the quartet
    if (tid == 0) s_next[0] = (long long)atomicAdd(a.ticket, 1ull);
    rys_sync<NW>();
    w = s_next[0];
  }
  while (w < count) {  // w is the same for all threads of the CTA
    if (a.ticket && tid == 0) s_next[turn ^ 1] = (long long)atomicAdd(a.ticket, 1ull);
    const int2 pq = a.work[a.reverse ? a.work_off + a.nwork - 1 - w : a.work_off + w];
    const PairDev& P = a.pairs[pq.x];
    const PairDev& Q = a.pairs[pq.y];
    for (int i = tid; i < 4 * kMaxCart; i += NT) {
      const int q = i / kMaxCart, c = i - q * kMaxCart;
      const bool second = (q & 1) ^ ((a.flip >> (q >> 1)) & 1);
      const PairDev& pr = q < 2 ? P : Q;
      const ShellDev& s = a.shells[second ? pr.shB : pr.shA];
      S.scl[q][c] = s.scl[c];
      S.pos[q][c] = s.pos[c];
      if (c == 0) {
        S.func[q] = s.func_off;
        S.nout[q] = s.nout;
        S.nint[q] = schwarz ? ncart(s.l) : internal_count(s);
      }
    }
    const int np = P.nprim * Q.nprim;
    double acc[C::kAcc];
#pragma unroll
    for (int i = 0; i < C::kAcc; ++i) acc[i] = 0.0;
    // points per primitive quartet: erfc(omega r)/r is 1/r minus erf(omega r)/r
    const int kpp = a.potential == 2 ? 2 * N : N;
    const int per_chunk = a.potential == 2 ? kRysKC / (2 * N) : kRysKC / N;
    // tables of chunk c (points PR[c]) into buffer b
    auto tables = [&](int c, int kcp, int b) {
      for (int i = tid; i < 3 * kcp; i += NT) {
        const int ax = i / kcp, k = i - ax * kcp;
        const double* const pr = PR + c * kRysRows * kRysKS + k;
        rys_axis<D::NE1, D::NF1, D::RF>(pr[(kC0 + ax) * kRysKS], pr[(kD0 + ax) * kRysKS],
                                        pr[kB00 * kRysKS], pr[kB10 * kRysKS], pr[kB01 * kRysKS],
                                        ax == 2 ? pr[kWt * kRysKS] : 1.0,
                                        T + (b * 3 + ax) * D::TS + k);
      }
    };
    for (int s0 = 0; s0 < np; s0 += NW * per_chunk) {
      // a chunk per warp, the last warp first (its share of the sums is the lightest): the points'
      // latency (pair data, then table rows at T) is paid once per NW chunks
      const int mine = NW - 1 - wq, p0 = s0 + mine * per_chunk;
      rys_points<C>(a, P, Q, tab, p0, min(max(np - p0, 0), per_chunk) * kpp, kpp, lane,
                    PR + mine * kRysRows * kRysKS);
      const int nc = min(NW, (np - s0 + per_chunk - 1) / per_chunk);
      auto padded = [&](int c) {
        return (min(np - s0 - c * per_chunk, per_chunk) * kpp + 3) & ~3;
      };
      rys_sync<NW>();  // points written; the previous chunk's tables are read
      if constexpr (D::kBuf == 2) {  // a chunk's tables beside the sums of the one before
        for (int c = 0; c <= nc; ++c) {
          if (c < nc) tables(c, padded(c), c & 1);
          if (c > 0) C::gemm(wq, lane, T + ((c - 1) & 1) * 3 * D::TS, padded(c - 1), acc);
          if (c < nc) rys_sync<NW>();
        }
      } else {
        for (int c = 0; c < nc; ++c) {
          if (c > 0) rys_sync<NW>();
          tables(c, padded(c), 0);
          rys_sync<NW>();
          C::gemm(wq, lane, T, padded(c), acc);
        }
      }
    }
    C::store(wq, lane, acc, ACC);
    rys_sync<NW>();  // ACC complete, tables read
    // ------------------------------------------------------------------------------ tail
    const int nA = S.nint[0], nB = S.nint[1], nC = S.nint[2], nD = S.nint[3];
    const int ncol = nC * nD;
    if (coulomb) {
      for (int i = tid; i < ncol; i += NT) {
        const int uc = i / nD, ud = i - uc * nD;
        DCD[i] = a.D[(S.func[2] + S.pos[2][uc]) * a.nbf + S.func[3] + S.pos[3][ud]] * S.scl[2][uc] *
                 S.scl[3][ud];
      }
      for (int i = tid; i < nA * nB; i += NT) {
        const int ua = i / nB, ub = i - ua * nB;
        DAB[i] = a.D[(S.func[0] + S.pos[0][ua]) * a.nbf + S.func[1] + S.pos[1][ub]] * S.scl[0][ua] *
                 S.scl[1][ub];
        VAB[i] = 0.0;
      }
    }
    if (a.mode == 0) {  // read after the barriers below
      long long bbase, bcols;
      block_dest(a, P, bbase, bcols);
      const bool tr = quartet_transposed(P, Q);
      const long long sbra = tr ? 1 : bcols, sket = tr ? bcols : 1;
      for (int i = tid; i < nA * nB; i += NT) {
        const int ua = i / nB, ub = i - ua * nB;
        s_ro[i] = bbase + ((long long)P.fo + S.pos[0][ua] * S.nout[1] + S.pos[1][ub]) * sbra;
        s_rs[i] = S.scl[0][ua] * S.scl[1][ub];
      }
      for (int i = NT - 1 - tid; i < ncol; i += NT) {
        const int uc = i / nD, ud = i - uc * nD;
        s_co[i] = ((long long)Q.fo + S.pos[2][uc] * S.nout[3] + S.pos[3][ud]) * sket;
        s_cs[i] = S.scl[2][uc] * S.scl[3][ud];
      }
      if constexpr (LD == 0) rys_sync<NW>();  // the ket step's barrier otherwise
    }
    // ket recursion and transform on D: tasks (row e, component c) -> HF[e][c][ud]
    if constexpr (LD > 0) {
      const double CDx = Q.ABx, CDy = Q.ABy, CDz = Q.ABz;
      for (int t = tid; t < D::NE * D::NCC; t += NT) {
        const int c = t / D::NE, e = t - c * D::NE;
        double o[D::NCD];
        rys_hrr<LC, LD>(ACC + e * D::NFs, 1, c, CDx, CDy, CDz, o);
        if constexpr (LD >= 2) {
          if (nD != D::NCD) {
            double y[2 * LD + 1];
            gen::Sph<LD>::apply(o, y);
#pragma unroll
            for (int i = 0; i < 2 * LD + 1; ++i) HF[e * D::HS + c * (2 * LD + 1) + i] = y[i];
            continue;
          }
        }
#pragma unroll
        for (int i = 0; i < D::NCD; ++i) HF[e * D::HS + c * D::NCD + i] = o[i];
      }
      rys_sync<NW>();
    }
    // transform on C, in place: tasks (row e, ud)
    if constexpr (LC >= 2) {
      if (nC != D::NCC) {
        for (int t = tid; t < D::NE * nD; t += NT) {
          const int ud = t / D::NE, e = t - ud * D::NE;
          double* const row = HF + e * D::HS + ud;
          double x[D::NCC], y[2 * LC + 1];
#pragma unroll
          for (int c = 0; c < D::NCC; ++c) x[c] = row[c * nD];
          gen::Sph<LC>::apply(x, y);
#pragma unroll
          for (int c = 0; c < 2 * LC + 1; ++c) row[c * nD] = y[c];
        }
        rys_sync<NW>();
      }
    }
    // bra recursion, transforms and output, a block of columns at a time
    const double ABx = P.ABx, ABy = P.ABy, ABz = P.ABz;
    const bool sphA = LA >= 2 && nA != D::NCA;
    const bool block = sphA || coulomb;  // the columns' values meet in BLK[(a, ub)][column]
    const int rowlen = D::NCA * nB;
    const int cap = block ? D::kBlkSize / rowlen : ncol;
    const int cmax = block ? min(ncol, (cap & 1) ? cap : cap - 1) : ncol;  // odd row stride
    const int CS = cmax | 1;
    double mx = 0.0;
    auto put = [&](int row, int col, double v) {
      out_store(a, s_ro[row] + s_co[col], v * s_rs[row] * s_cs[col]);
    };
    for (int c0 = 0; c0 < ncol; c0 += cmax) {
      const int cc = min(cmax, ncol - c0);
      for (int t = tid; t < cc * D::NCA; t += NT) {
        const int ca = t / cc, cl = t - ca * cc, col = c0 + cl;
        double o[D::NCB];
        rys_hrr<LA, LB>(HF + col, D::HS, ca, ABx, ABy, ABz, o);
        if (schwarz) {
          const int uc = col / nD, ud = col - uc * nD;
          const double wcd = gen::cnorm<LC>(uc) * gen::cnorm<LD>(ud) * gen::cnorm<LA>(ca);
#pragma unroll
          for (int i = 0; i < D::NCB; ++i) mx = fmax(mx, fabs(o[i]) * (gen::cnorm<LB>(i) * wcd));
          continue;
        }
        if constexpr (LB >= 2) {
          if (nB != D::NCB) {
            double y[2 * LB + 1];
            gen::Sph<LB>::apply(o, y);
#pragma unroll
            for (int i = 0; i < 2 * LB + 1; ++i) o[i] = y[i];
          }
        }
#pragma unroll
        for (int i = 0; i < D::NCB; ++i) {
          if (i >= nB) break;
          if (block) BLK[(ca * nB + i) * CS + cl] = o[i];
          else put(ca * nB + i, col, o[i]);
        }
      }
      if (!block) continue;
      rys_sync<NW>();
      if constexpr (LA >= 2) {
        if (sphA) {  // transform on A: tasks (ub, column), stored or put back in place
          for (int t = tid; t < cc * nB; t += NT) {
            const int ub = t / cc, cl = t - ub * cc;
            double x[D::NCA], y[2 * LA + 1];
#pragma unroll
            for (int i = 0; i < D::NCA; ++i) x[i] = BLK[(i * nB + ub) * CS + cl];
            gen::Sph<LA>::apply(x, y);
#pragma unroll
            for (int i = 0; i < 2 * LA + 1; ++i) {
              if (coulomb) BLK[(i * nB + ub) * CS + cl] = y[i];
              else put(i * nB + ub, c0 + cl, y[i]);
            }
          }
          rys_sync<NW>();
        }
      }
      if (coulomb) {
        // J[a][b] sums over the block's columns; J[c][d] of each column
        const int nab = nA * nB;
        for (int t = tid; t < nab + cc; t += NT) {
          if (t < nab) {
            double s = VAB[t];
            for (int cl = 0; cl < cc; ++cl) s = fma(BLK[t * CS + cl], DCD[c0 + cl], s);
            VAB[t] = s;
          } else if (pq.x != pq.y) {
            const int cl = t - nab, col = c0 + cl, uc = col / nD, ud = col - uc * nD;
            double s = 0.0;
            for (int i = 0; i < nab; ++i) s = fma(BLK[i * CS + cl], DAB[i], s);
            s *= ((P.shA != P.shB) ? 2.0 : 1.0) * S.scl[2][uc] * S.scl[3][ud];
            const long long fc = S.func[2] + S.pos[2][uc], fd = S.func[3] + S.pos[3][ud];
            j_add(a, fc * a.nbf + fd, s);
            if (Q.shA != Q.shB) j_add(a, fd * a.nbf + fc, s);
          }
        }
        rys_sync<NW>();
      }
    }
    if (schwarz) {
      for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      rys_sync<NW>();  // HF is read
      if (lane == 0) smem[wq] = mx;
      rys_sync<NW>();
      if (tid == 0) {
        for (int i = 1; i < C::kW; ++i) mx = fmax(mx, smem[i]);
        a.qout[pq.x] = sqrt(mx);
      }
    }
    if (coulomb) {
      const double fk = (Q.shA != Q.shB) ? 2.0 : 1.0;
      for (int i = tid; i < nA * nB; i += NT) {
        const int ua = i / nB, ub = i - ua * nB;
        const long long fa = S.func[0] + S.pos[0][ua], fb = S.func[1] + S.pos[1][ub];
        const double s = VAB[i] * fk * S.scl[0][ua] * S.scl[1][ub];
        j_add(a, fa * a.nbf + fb, s);
        if (P.shA != P.shB) j_add(a, fb * a.nbf + fa, s);
      }
    }
    rys_sync<NW>();  // shared memory free for the next quartet; the next draw is visible
    turn ^= 1;
    w = a.ticket ? s_next[turn] : w + gridDim.x;
  }
}

template <class C>
int launch_rys_t(const EriLaunch& a, cudaStream_t st) {
  using D = RysDims<C>;
  RysArgs A;
  A.a = a;
  int s = rys_table(&A.tab);
  if (s) return s;
  int dev = 0;
  cudaGetDevice(&dev);
  const int cm = a.mode == 2 ? 1 : 0;
  const int smem = (D::kSmem + (cm ? D::NKET + 2 * D::NAB : 0)) * (int)sizeof(double);
  static_assert((D::kSmem + 3 * D::NKET + 4 * D::NAB) * 8 + 1024 <= kRysMaxSmem, "shared memory");
  // CTAs the device keeps resident in this mode, found once per device and mode
  static std::atomic<int> resident[64][2];
  int r = dev >= 0 && dev < 64 ? resident[dev][cm].load() : 0;
  if (!r) {
    int per_sm = 0, nsm = 1;
    const int most = (D::kSmem + D::NKET + 2 * D::NAB) * (int)sizeof(double);
    s = cuda_status(cudaFuncSetAttribute(eri_rys<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, most),
                    "eri_rys shared memory attribute");
    if (s) return s;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, eri_rys<C>, D::NT, smem);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    r = std::max(1, per_sm) * nsm;
    if (dev >= 0 && dev < 64) resident[dev][cm].store(r);
  }
  const int grid = (int)std::max<long long>(1, std::min<long long>(a.nwork, r));
  eri_rys<C><<<grid, D::NT, smem, st>>>(A);
  return cuda_status(cudaGetLastError(), "eri_rys launch");
}

}  // namespace gbx
