// K1: per-quartet screening and set-up on the device (FP64).
//
// Restates the per-quartet part of calculate_intracule (src/mod_intracule.f90:282-343) and
// its helpers JA8 / polycoef / gauherm (src/mod_intrastuff.f90:32-341): normalisation,
// screen 1 |v| sqrt(J_ik J_jl) >= lim, Gaussian products, the three per-dimension
// polynomials (Gauss-Hermite right-hand side, Vandermonde system solved by LU with partial
// pivoting, zeroed on a singular matrix or |C| > 1e3) and screen 2 |A Ux Uy Uz| >= lim.
//
// The arithmetic is spelled out operation by operation (integer powers by repeated
// multiplication, half-integer powers through sqrt, a Cody-Waite/Taylor exponential) and this
// translation unit is compiled with -fmad=false, so every screening value is bit-identical to the
// CPU oracle's and the screening decisions are identical.
//
// Quartets whose four primitives lie in the same shells (same exponent and centre) share everything
// but their powers and DM2 value: one Gaussian exp(-sqe^2 |r + d|^2), and in each dimension one of
// at most prod (t_max + 1) polynomials. So the work goes by groups of such quartets:
//   1. screen 1 of every quartet (a thread each: two table entries and a square root);
//   2. the quartets that pass are sorted by group (stable radix sort: input order within a group);
//   3. each (group, dimension, powers) polynomial that some quartet needs is solved once (k_poly, a
//      thread each) into a table;
//   4. k_groups, eight lanes to four warps per group: screen 2 of its quartets from table entries, and
//      their sum: the shared Gaussian times one trivariate polynomial, at most 35 coefficients for four p shells
//      where the quartets are 81 products (CH4: 5.2 quartets per record; molecules with d shells: 9
//      to 14), summed in FP64 in a fixed order;
//   5. the records are sorted by the shape of their polynomial and written (k_write) as
//      class-segmented FP64 records (the FP64 evaluation) and FP32 records (the mixed evaluation).
// A group keeps one product record per quartet where that is cheaper to evaluate (a few quartets of
// incomplete shells with high powers) or its total degree exceeds kMaxTotal.
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include <algorithm>
#include <thread>
#include <cmath>
#include <cstring>

#define INCA_GH_TABLE static __constant__ const
#include "hermite_table.h"
#include "inca_internal.h"

namespace inca {
namespace {


// Constants and arguments of a preparation, passed to every kernel by value: contexts on several host
// threads prepare and read back at the same time, so nothing of a call lives in a module-wide symbol. (The
// quadrature's tables are initialised with the code and never written.)
struct PrepConst {
  double wm[kMaxCoef];
  double pi15;
  double thresh;
  double c_u;  // sqrt(1/ln 2): u = c_u r' turns e^(-r'^2) into 2^(-u^2)
  double cu_inv_pow[kMaxTotal + 1];  // c_u^-k
  float fact[kMaxTotal + 1];         // k!
  int nprim;
  int normalize;
  int merge;  // 0: every quartet is a group of its own
};

__device__ __forceinline__ double ipow(double x, int n) {
  if (n <= 0) return 1.0;
  double r = x;
  for (int i = 1; i < n; ++i) r = r * x;
  return r;
}

// Cody-Waite reduction x = k ln2 + r (ln2 with a 32-bit head), Taylor degree 13 by Horner.
__device__ double pexp(double x) {
  if (x != x) return x;
  if (x > 709.0) return HUGE_VAL;
  if (x < -708.0) return 0.0;
  const double kInvLn2 = 1.4426950408889634;
  const double kLn2Hi = 0.6931471803691238;
  const double kLn2Lo = 1.9082149292705877e-10;
  const double k = rint(x * kInvLn2);
  const double r = (x - k * kLn2Hi) - k * kLn2Lo;
  const double c[14] = {1.6059043836821613e-10, 2.08767569878681e-09, 2.505210838544172e-08,
                        2.755731922398589e-07, 2.7557319223985893e-06, 2.48015873015873e-05,
                        0.0001984126984126984, 0.001388888888888889, 0.008333333333333333,
                        0.041666666666666664, 0.16666666666666666, 0.5, 1.0, 1.0};
  double p = c[0];
#pragma unroll
  for (int i = 1; i < 14; ++i) p = p * r + c[i];
  return ldexp(p, static_cast<int>(k));
}

__device__ __forceinline__ double xmax(int n) { return inca_gh::kNode[n][n - 1]; }

// JA8 (src/mod_intrastuff.f90:32-123).
__device__ __forceinline__ double ja8(const PrepConst& cP, const PrimD& a, const PrimD& b, double R2, double aik, double eik) {
  const int sumt = a.t[0] + b.t[0] + a.t[1] + b.t[1] + a.t[2] + b.t[2];
  const double s2a = sqrt(2.0 / aik);
  const double two_a = 2.0 * aik;
  double v = cP.pi15 / (ipow(two_a, sumt + 1) * sqrt(two_a));
  v = v * pexp((-2.0 * eik) * R2);
  const double ax[3] = {a.x, a.y, a.z}, bx[3] = {b.x, b.y, b.z};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double xm = xmax(a.t[d] + b.t[d] + 1);
    const double dx = fabs(bx[d] - ax[d]);
    v = v * ipow(xm + (b.alpha * s2a) * dx, 2 * a.t[d]);
    v = v * ipow(xm + (a.alpha * s2a) * dx, 2 * b.t[d]);
  }
  return v;
}

// LU with partial pivoting (first maximum), reciprocal pivot scaling, then the two
// triangular solves: LAPACK dgesv semantics (dgetf2 + dgetrs). Returns info.
__device__ int lu_solve(int n, double* M, double* b) {
  int info = 0;
  int piv[kMaxCoef];
  for (int j = 0; j < n; ++j) {
    int p = j;
    double big = fabs(M[j * n + j]);
    for (int i = j + 1; i < n; ++i) {
      const double a = fabs(M[i * n + j]);
      if (a > big) { big = a; p = i; }
    }
    piv[j] = p;
    if (M[p * n + j] != 0.0) {
      if (p != j)
        for (int c = 0; c < n; ++c) {
          const double t = M[j * n + c];
          M[j * n + c] = M[p * n + c];
          M[p * n + c] = t;
        }
      const double inv = 1.0 / M[j * n + j];
      for (int i = j + 1; i < n; ++i) M[i * n + j] = M[i * n + j] * inv;
    } else if (info == 0) {
      info = j + 1;
    }
    for (int i = j + 1; i < n; ++i) {
      const double l = M[i * n + j];
      for (int c = j + 1; c < n; ++c) M[i * n + c] = M[i * n + c] - l * M[j * n + c];
    }
  }
  if (info) return info;
  for (int j = 0; j < n; ++j)
    if (piv[j] != j) {
      const double t = b[j];
      b[j] = b[piv[j]];
      b[piv[j]] = t;
    }
  for (int i = 0; i < n; ++i)
    for (int c = 0; c < i; ++c) b[i] = b[i] - M[i * n + c] * b[c];
  for (int i = n - 1; i >= 0; --i) {
    for (int c = i + 1; c < n; ++c) b[i] = b[i] - M[i * n + c] * b[c];
    b[i] = b[i] / M[i * n + i];
  }
  return 0;
}

// polycoef (src/mod_intrastuff.f90:127-194); C highest degree first.
__device__ __forceinline__ void polycoef(const PrepConst& cP, const double R[4], double Pik, double Pjl, double Pijkl,
                                         const int t[4], double sqe, double invz, double alf, double* C) {
  const int L = t[0] + t[1] + t[2] + t[3];
  const int np = L + 1;
  const int nn = L / 2 + 1;
  if (np == 1) {
    C[0] = inca_gh::kWeight[1][0];
    return;
  }
  double M[kMaxCoef * kMaxCoef];
  for (int i = 0; i < np; ++i) {
    const double xx = -0.5 + double(i + 1);
    const double base = sqe * ((xx + Pik) - Pjl);
    for (int j = 0; j < np; ++j) M[i * np + j] = ipow(base, L - j);
    const double am = (alf - 0.5) * xx, ap = (alf + 0.5) * xx;
    double rhs = 0.0;
    for (int h = 0; h < nn; ++h) {
      const double zr = invz * inca_gh::kNode[nn][h];
      double W = ipow((zr + am) + (Pijkl - R[0]), t[0]) * ipow((zr + ap) + (Pijkl - R[1]), t[1]);
      W = W * ipow((zr + am) + (Pijkl - R[2]), t[2]);
      W = W * ipow((zr + ap) + (Pijkl - R[3]), t[3]);
      rhs = rhs + inca_gh::kWeight[nn][h] * W;
    }
    C[i] = rhs;
  }
  const int info = lu_solve(np, M, C);
  bool blow = false;
  for (int i = 0; i < np; ++i)
    if (fabs(C[i]) > 1e3) blow = true;
  if (info != 0 || blow)
    for (int i = 0; i < np; ++i) C[i] = 0.0;
}

// polycoef for a compile-time number of coefficients, everything in registers: the same operations
// in the same order (rows are exchanged by selection), so the same bits. The loops over the powers
// are unrolled selections too; with the matrix in local memory the small systems, most of all
// solved, waited on it.
template <int kT>  // powers up to kT: a product that no lane needs would still be computed and selected away
__device__ __forceinline__ double ipow_up_to(double x, int n) {
  double r = n > 0 ? x : 1.0;
  if (kT > 1 && n > 1) r = r * x;
  if (kT > 2 && n > 2) r = r * x;
  if (kT > 3 && n > 3) r = r * x;
  return r;
}
// |x| as an integer: in the order of the numbers (NaN above infinity), compared outside the FP64 pipe.
constexpr uint64_t kInfinity = 0x7FF0000000000000ull;
__device__ __forceinline__ uint64_t magnitude(double x) {
  return static_cast<uint64_t>(__double_as_longlong(x)) & 0x7FFFFFFFFFFFFFFFull;
}
template <int NP, int kT>
__device__ __forceinline__ void polycoef_n(const PrepConst& cP, const double R[4], double Pik, double Pjl,
                                           double Pijkl, const int t[4], double sqe, double invz, double alf,
                                           double* C) {
  constexpr int L = NP - 1, NN = L / 2 + 1;
  double M[NP][NP], b[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const double xx = -0.5 + double(i + 1);
    const double base = sqe * ((xx + Pik) - Pjl);
#pragma unroll
    for (int j = L; j >= 0; --j) M[i][j] = L - j == 0 ? 1.0 : L - j == 1 ? base : M[i][j + 1] * base;
    const double am = (alf - 0.5) * xx, ap = (alf + 0.5) * xx;
    double rhs = 0.0;
#pragma unroll
    for (int h = 0; h < NN; ++h) {
      const double zr = invz * inca_gh::kNode[NN][h];
      double W = ipow_up_to<kT>((zr + am) + (Pijkl - R[0]), t[0]) * ipow_up_to<kT>((zr + ap) + (Pijkl - R[1]), t[1]);
      W = W * ipow_up_to<kT>((zr + am) + (Pijkl - R[2]), t[2]);
      W = W * ipow_up_to<kT>((zr + ap) + (Pijkl - R[3]), t[3]);
      rhs = rhs + inca_gh::kWeight[NN][h] * W;
    }
    b[i] = rhs;
  }
  bool singular = false;
  int piv[NP];
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    int p = j;
    uint64_t big = magnitude(M[j][j]);
#pragma unroll
    for (int i = j + 1; i < NP; ++i) {
      const uint64_t a = magnitude(M[i][j]);
      if (a > big && a <= kInfinity) { big = a; p = i; }
    }
    piv[j] = p;
#pragma unroll
    for (int i = j + 1; i < NP; ++i)
#pragma unroll
      for (int c = 0; c < NP; ++c) {
        const double x = M[j][c], y = M[i][c];
        M[j][c] = p == i ? y : x;
        M[i][c] = p == i ? x : y;
      }
    if (magnitude(M[j][j]) != 0) {
      const double inv = 1.0 / M[j][j];
#pragma unroll
      for (int i = j + 1; i < NP; ++i) M[i][j] = M[i][j] * inv;
    } else {
      singular = true;
    }
#pragma unroll
    for (int i = j + 1; i < NP; ++i)
#pragma unroll
      for (int c = j + 1; c < NP; ++c) M[i][c] = M[i][c] - M[i][j] * M[j][c];
  }
#pragma unroll
  for (int j = 0; j < NP; ++j)
#pragma unroll
    for (int i = j + 1; i < NP; ++i) {
      const double x = b[j], y = b[i];
      b[j] = piv[j] == i ? y : x;
      b[i] = piv[j] == i ? x : y;
    }
#pragma unroll
  for (int i = 0; i < NP; ++i)
#pragma unroll
    for (int c = 0; c < i; ++c) b[i] = b[i] - M[i][c] * b[c];
#pragma unroll
  for (int i = NP - 1; i >= 0; --i) {
#pragma unroll
    for (int c = i + 1; c < NP; ++c) b[i] = b[i] - M[i][c] * b[c];
    b[i] = b[i] / M[i][i];
  }
  bool blow = singular;
#pragma unroll
  for (int i = 0; i < NP; ++i)
    blow |= magnitude(b[i]) > 0x408F400000000000ull && magnitude(b[i]) <= kInfinity;  // |b| > 1e3
#pragma unroll
  for (int i = 0; i < NP; ++i) C[i] = blow ? 0.0 : b[i];
}

struct QRec {
  double A, sqe, d[3];
  int L[3];
  double C[3][kMaxCoef];
};

// JA8 of a primitive pair.
__device__ __forceinline__ double pair_ja8(const PrepConst& cP, const PrimD& Pi, const PrimD& Pk) {
  const double aik = Pi.alpha + Pk.alpha;
  const double eik = (Pi.alpha * Pk.alpha) * (1.0 / aik);
  const double Xi[3] = {Pi.x, Pi.y, Pi.z}, Xk[3] = {Pk.x, Pk.y, Pk.z};
  double Rik2 = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) Rik2 = Rik2 + (Xi[d] - Xk[d]) * (Xi[d] - Xk[d]);
  return ja8(cP, Pi, Pk, Rik2, aik, eik);
}

// JA8 of every ordered primitive pair (i, k): a quartet's screen-1 value reads two table entries
// instead of evaluating JA8 twice, and the values are the same bits.
__global__ void k_pair_ja8(const __grid_constant__ PrepConst cP, int nprim, const PrimD* __restrict__ prims,
                           double* __restrict__ J) {
  const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (t < static_cast<int64_t>(nprim) * nprim) J[t] = pair_ja8(cP, prims[t / nprim], prims[t % nprim]);
}

constexpr int kPairTableMax = 4096;
// inca_prepare keeps its scratch in the context up to this many bytes in all (by what was reserved: 40 B per
// quartet and the radix sort's storage of 16 more, 112 B per subgroup, and the largest slab's table)
constexpr size_t kPrepKeepBytes = size_t(1) << 32;
// What a subgroup's quartets share: the same shells i, j, k, l in this order.
struct SubConst {
  double R[4][3];  // centres of i, j, k, l
  double sqe, invz, alf, c1, c2, lim;  // c1 c2 DMval is the quartet's amplitude A
  double Pik[3], Pjl[3], Pijkl[3];
  int m[4];  // largest power of i, j, k, l among its quartets, any dimension
  int mol, total;  // total: the largest sum of a quartet's powers can be (at most kMaxTotal)
  // The table has an entry for each combination of powers up to m and dimension. A subgroup of one quartet
  // (shells with one function each) has its own three entries alone: 20 g functions on shells of their own filled 6 slabs
  // of 1875 entries a subgroup, one after the other: preparation 5.5 ms, 1.1 so.
  uint32_t single[3];  // 0, or kSingle and the one quartet's powers of i, j, k, l in each dimension, 3 bits each
  static constexpr uint32_t kSingle = 1u << 31;
  __device__ __forceinline__ int combos() const {
    return single[0] ? 1 : (m[0] + 1) * (m[1] + 1) * (m[2] + 1) * (m[3] + 1);
  }
  __device__ __forceinline__ int entry() const { return m[0] + m[1] + m[2] + m[3] + 2; }  // U and the coefficients
  __device__ __forceinline__ int combo(int ti, int tj, int tk, int tl) const {
    return single[0] ? 0 : ((ti * (m[1] + 1) + tj) * (m[2] + 1) + tk) * (m[3] + 1) + tl;
  }
};

// Exponents, product centres and factors of four primitives (src/mod_intracule.f90:301-330).
__device__ __forceinline__ void shared_of(const PrimD& Pi, const PrimD& Pj, const PrimD& Pk, const PrimD& Pl,
                                          SubConst* c) {
  const double aik = Pi.alpha + Pk.alpha, ajl = Pj.alpha + Pl.alpha;
  const double eik = (Pi.alpha * Pk.alpha) * (1.0 / aik);
  const double ejl = (Pj.alpha * Pl.alpha) * (1.0 / ajl);
  const double Xi[3] = {Pi.x, Pi.y, Pi.z}, Xj[3] = {Pj.x, Pj.y, Pj.z};
  const double Xk[3] = {Pk.x, Pk.y, Pk.z}, Xl[3] = {Pl.x, Pl.y, Pl.z};
  double Rik2 = 0.0, Rjl2 = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    Rik2 = Rik2 + (Xi[d] - Xk[d]) * (Xi[d] - Xk[d]);
    Rjl2 = Rjl2 + (Xj[d] - Xl[d]) * (Xj[d] - Xl[d]);
  }
  const double zeta = aik + ajl;
  const double eijkl = (aik * ajl) * (1.0 / zeta);
  c->sqe = sqrt(eijkl);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    c->R[0][d] = Xi[d];
    c->R[1][d] = Xj[d];
    c->R[2][d] = Xk[d];
    c->R[3][d] = Xl[d];
    c->Pik[d] = (Pi.alpha * Xi[d] + Pk.alpha * Xk[d]) * (1.0 / aik);
    c->Pjl[d] = (Pj.alpha * Xj[d] + Pl.alpha * Xl[d]) * (1.0 / ajl);
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) c->Pijkl[d] = (aik * c->Pik[d] + ajl * c->Pjl[d]) * (1.0 / zeta);
  c->invz = 1.0 / sqrt(zeta);
  c->alf = (0.5 * (aik - ajl)) * (1.0 / zeta);
  c->c1 = 1.0 / (zeta * sqrt(zeta));
  c->c2 = pexp((-eik) * Rik2 - ejl * Rjl2);
}

__device__ __forceinline__ double dm_value(const PrepConst& cP, const PrimD& Pi, const PrimD& Pj, const PrimD& Pk,
                                           const PrimD& Pl, double v) {
  return cP.normalize ? v * (((Pi.norm * Pj.norm) * Pk.norm) * Pl.norm) : v;
}

// Screen 1 (src/mod_intracule.f90:282-300) of a quartet. Jtab (optional): the table of k_pair_ja8.
__device__ __forceinline__ bool screen1_of(const PrepConst& cP, const PrimD& Pi, const PrimD& Pj, const PrimD& Pk,
                                           const PrimD& Pl, int4 q, double v, const double* __restrict__ Jtab,
                                           double* value) {
  const double DMval = dm_value(cP, Pi, Pj, Pk, Pl, v);
  double Jik, Jjl;
  if (Jtab) {
    Jik = Jtab[static_cast<int64_t>(q.x - 1) * cP.nprim + (q.z - 1)];
    Jjl = Jtab[static_cast<int64_t>(q.y - 1) * cP.nprim + (q.w - 1)];
  } else {
    Jik = pair_ja8(cP, Pi, Pk);
    Jjl = pair_ja8(cP, Pj, Pl);
  }
  const double lim = cP.thresh * Pi.lim_scale;
  *value = fabs(DMval) * sqrt(Jik * Jjl);
  return *value >= lim;
}

// The record of one surviving quartet (src/mod_intracule.f90:301-343).
__device__ __forceinline__ void restate(const PrepConst& cP, const PrimD* __restrict__ prims, int4 q, double v,
                                        QRec* out) {
  const PrimD &Pi = prims[q.x - 1], &Pj = prims[q.y - 1], &Pk = prims[q.z - 1], &Pl = prims[q.w - 1];
  SubConst c;
  shared_of(Pi, Pj, Pk, Pl, &c);
  out->A = (dm_value(cP, Pi, Pj, Pk, Pl, v) * c.c1) * c.c2;
  out->sqe = c.sqe;
  for (int d = 0; d < 3; ++d) {
    const double R[4] = {c.R[0][d], c.R[1][d], c.R[2][d], c.R[3][d]};
    const int t[4] = {Pi.t[d], Pj.t[d], Pk.t[d], Pl.t[d]};
    out->L[d] = t[0] + t[1] + t[2] + t[3];
    polycoef(cP, R, c.Pik[d], c.Pjl[d], c.Pijkl[d], t, c.sqe, c.invz, c.alf, out->C[d]);
    out->d[d] = c.Pik[d] - c.Pjl[d];
  }
}

// Sort key of a quartet: its molecule's first group key plus (pair of shells i, k; pair of shells
// j, l), times four, plus which way round the two pairs are written (the polynomials' operation
// sequence follows the order i, j, k, l; the Gaussian and its centre do not).
__device__ __forceinline__ uint64_t quartet_key(const PrimD& i, const PrimD& j, const PrimD& k, const PrimD& l) {
  const int64_t np = static_cast<int64_t>(i.nshell) * (i.nshell + 1) / 2;
  const int64_t hi = max(i.shell, k.shell), lo = min(i.shell, k.shell);
  const int64_t hj = max(j.shell, l.shell), lj = min(j.shell, l.shell);
  const int64_t group = i.gbase + (hi * (hi + 1) / 2 + lo) * np + hj * (hj + 1) / 2 + lj;
  return static_cast<uint64_t>(group) * 4 + (i.shell > k.shell ? 1 : 0) + (j.shell > l.shell ? 2 : 0);
}

// Counters of a preparation, read back together.
enum PrepCount { kNScreen1 = 0, kNBad, kNSub, kNEntry, kNTable, kNCoef, kNGroup, kNSurv, kNRec, kNProduct,
                 kNUsed, kNClass,
                 kNSmall, kNMedium, kNLarge, kNSingle, kNTask,  // of a slab: groups by size, and
                 kNCounts = kNTask + kMaxCoef };  // kNTask + L: polynomials of degree L to solve

// Screen 1 of every quartet, and the sort key of those that pass (the others get fail_key and sort
// last).
__global__ void k_screen1(const __grid_constant__ PrepConst cP, int64_t n, const int4* __restrict__ ijkl, const double* __restrict__ v,
                          const PrimD* __restrict__ prims, uint8_t* flags, double* s1, double* s2, uint64_t* key,
                          int64_t* idx, uint64_t fail_key, unsigned long long* count,
                          const double* __restrict__ Jtab) {
  const int64_t q = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  bool pass = false;
  if (q < n) {
    const int4 r = ijkl[q];
    uint64_t kq = fail_key;
    double value = 0.0;
    if (r.x < 1 || r.y < 1 || r.z < 1 || r.w < 1 || r.x > cP.nprim || r.y > cP.nprim || r.z > cP.nprim ||
        r.w > cP.nprim) {
      count[kNBad] = 1;
    } else {
      const PrimD &Pi = prims[r.x - 1], &Pj = prims[r.y - 1], &Pk = prims[r.z - 1], &Pl = prims[r.w - 1];
      pass = screen1_of(cP, Pi, Pj, Pk, Pl, r, v[q], Jtab, &value);
      if (pass) kq = cP.merge ? quartet_key(Pi, Pj, Pk, Pl) : 4 * static_cast<uint64_t>(q);
    }
    idx[q] = q;
    key[q] = kq;
    flags[q] = pass ? 1 : 0;
    if (s1) s1[q] = value;
    if (s2) s2[q] = 0.0;
  }
  const unsigned b = __ballot_sync(0xffffffffu, pass);
  if ((threadIdx.x & 31) == 0 && b) atomicAdd(&count[kNScreen1], static_cast<unsigned long long>(__popc(b)));
}

// Quartets of one sort key (a subgroup): the same shells in the same order.
struct SubHead {
  const uint64_t* key;
  uint64_t fail_key;
  __device__ bool operator()(int64_t i) const {
    return key[i] != fail_key && (i == 0 || key[i] != key[i - 1]);
  }
};
// First subgroup of a group.
struct GroupHead {
  const uint64_t* key;
  const int64_t* sub_off;
  __device__ bool operator()(int64_t s) const {
    return s == 0 || (key[sub_off[s]] >> 2) != (key[sub_off[s - 1]] >> 2);
  }
};
struct Survivor {
  const uint8_t* flags;
  __device__ bool operator()(int64_t i) const { return flags[i] == 3; }
};

// Doubles of a merged record before it has its place: FP64 coefficients, FP32 hi and lo, S.
__host__ __device__ inline int64_t record_scratch(int nc, int total) {
  return nc + (2 * nc + total + 1 + 1) / 2;
}

// A subgroup's polynomials (3 per combination of powers) and their table entries in doubles; summed, the
// places of the subgroups after it.
struct SubSize {
  int64_t ent, tab;
  __host__ __device__ SubSize operator+(const SubSize& o) const { return SubSize{ent + o.ent, tab + o.tab}; }
};

// Instructions a term costs at a point in the FP32 evaluation, counted in mixed_eval.cu's terms32:
// what decides between one merged record and a product record per quartet.
__device__ __forceinline__ int product_cost(int sum_l) { return 50 + 2 * sum_l; }
__device__ __forceinline__ int merged_cost(int total) { return 44 + merged_coefs(total) + 2 * total; }

// Largest powers of a subgroup's four shells in any dimension, and the largest sum of its quartets' powers.
struct SubPowers {
  uint8_t m[4];
  int total;
};

// Table entries of a subgroup of n quartets (SubConst::combos in three dimensions).
__device__ __forceinline__ int sub_entries(const SubPowers& P, int64_t n) {
  return n == 1 ? 3 : 3 * (P.m[0] + 1) * (P.m[1] + 1) * (P.m[2] + 1) * (P.m[3] + 1);
}

// Powers and sizes of every subgroup, kTeam lanes each (a warp, or eight lanes where subgroups have up to eight
// quartets on average: 108 000 of one, 53 us with a warp, 28 so). The totals go to count, with what the groups' records can
// need at most: a group is merged only where that is cheaper than its quartets' products, so a record has no
// more coefficients than these cost (a bound by the shells alone held 16 KB for each quartet of shells with one
// component of a g shell, 8.2 KB a quartet held after a preparation of such shells, 1.1 KB now).
template <int kTeam>
__global__ void k_sub(int64_t nsub, const int64_t* __restrict__ sub_off, int64_t npass, const uint64_t* __restrict__ key,
                      const int64_t* __restrict__ idx, const int4* __restrict__ ijkl, const PrimD* __restrict__ prims,
                      SubPowers* sub, SubSize* size, unsigned long long* count) {
  const int lane = threadIdx.x % kTeam;
  const unsigned team = kTeam == 32 ? 0xffffffffu : ((1u << (kTeam % 32)) - 1u) << ((threadIdx.x & 31) & ~(kTeam - 1));
  __shared__ unsigned long long sh[3];
  if (threadIdx.x < 3) sh[threadIdx.x] = 0;
  __syncthreads();
  const int64_t s = blockIdx.x * static_cast<int64_t>(blockDim.x / kTeam) + threadIdx.x / kTeam;
  auto first = [&](int64_t t) { return t < nsub ? sub_off[t] : npass; };
  int m[4];
  auto scan = [&](int64_t m0, int64_t m1) {  // m, and the sum of the powers
    int sums[4] = {0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 4; ++k) m[k] = 0;
    for (int64_t p = m0 + lane; p < m1; p += kTeam) {
      const int4 q = ijkl[idx[p]];
      const int at[4] = {q.x - 1, q.y - 1, q.z - 1, q.w - 1};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const PrimD& P = prims[at[k]];
        m[k] = max(m[k], max(P.t[0], max(P.t[1], P.t[2])));
        sums[k] = max(sums[k], P.t[0] + P.t[1] + P.t[2]);
      }
    }
    int total = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      m[k] = __reduce_max_sync(team, m[k]);
      total += __reduce_max_sync(team, sums[k]);
    }
    return total;
  };
  unsigned long long need[3] = {0, 0, 0};
  if (s < nsub) {
    int64_t m0 = first(s), m1 = first(s + 1);
    int total = scan(m0, m1);
    if (lane == 0) {
      const int powers = m[0] + m[1] + m[2] + m[3];
      SubPowers P;
      for (int k = 0; k < 4; ++k) P.m[k] = static_cast<uint8_t>(m[k]);
      P.total = min(total, kMaxTotal);
      const int ent = sub_entries(P, m1 - m0);
      sub[s] = P;
      size[s] = SubSize{ent, static_cast<int64_t>(ent) * (powers + 2)};
      need[0] = static_cast<unsigned long long>(ent);
      need[1] = need[0] * (powers + 2);
    }
    const uint64_t group = key[m0] >> 2;
    if (s == 0 || key[m0 - 1] >> 2 != group) {  // a group's first subgroup: the others (at most three) too
      int64_t cost = (m1 - m0) * product_cost(total);
      for (int64_t t = s + 1; t < nsub; ++t) {
        m0 = m1;
        m1 = first(t + 1);
        if (key[m0] >> 2 != group) break;
        const int sum = scan(m0, m1);
        total = max(total, sum);
        cost += (m1 - m0) * product_cost(sum);
      }
      int most = min(total, kMaxTotal);
      while (most > 0 && merged_cost(most) > cost) --most;
      if (lane == 0) need[2] = static_cast<unsigned long long>(record_scratch(merged_coefs(most), most));
    }
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    for (int o = kTeam; o < 32; o *= 2) need[k] += __shfl_xor_sync(0xffffffffu, need[k], o);  // (lane 0 of each team)
    if ((threadIdx.x & 31) == 0) atomicAdd(&sh[k], need[k]);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(&count[kNEntry], sh[0]);
    atomicAdd(&count[kNTable], sh[1]);
    atomicAdd(&count[kNCoef], sh[2]);
  }
}

// Lists of up to kSmallList quartets: what sorts, selections and scans over the list do in some ten launches and
// two read-backs for grouping, and six and one for the records' classes, done by one block each, kSmallItems consecutive
// items a thread. Such lists are all launch latency: a preparation of 6, 231 and 3 081 quartets took 165, 233 and 284
// us, so 122, 178 and 228. (14 706 quartets, 16 items a thread: 343 us against 299.)
constexpr int kSmallThreads = 1024, kSmallItems = 4;
constexpr int64_t kSmallList = kSmallThreads * kSmallItems;
struct SmallBlock {
  using Sort = cub::BlockRadixSort<uint32_t, kSmallThreads, kSmallItems, int>;
  // (scans by warps: raking ones keep 32 values a thread in registers)
  using Scan = cub::BlockScan<int, kSmallThreads, cub::BLOCK_SCAN_WARP_SCANS>;
  using SizeScan = cub::BlockScan<SubSize, kSmallThreads, cub::BLOCK_SCAN_WARP_SCANS>;
  union {
    Sort::TempStorage sort;
    Scan::TempStorage scan;
    SizeScan::TempStorage size;
  } u;
  uint32_t last[kSmallThreads];  // each thread's last key
  unsigned long long coef;
  // Flags of a thread's items (a bit each) to the number flagged before the thread; the number of all in *all.
  __device__ __forceinline__ int before(uint32_t flags, int* all) {
    int n = __popc(flags);
    Scan(u.scan).ExclusiveSum(n, n, *all);
    __syncthreads();
    return n;
  }
  // Sorts the first n of the block's items by the low bits (stable; the others carry 0xFFFFFFFF and go last) and
  // flags the first of each run of equal keys below `end`.
  __device__ __forceinline__ uint32_t sort_runs(uint32_t (&k)[kSmallItems], int (&v)[kSmallItems], int bits, int n,
                                                uint32_t end) {
    Sort(u.sort).Sort(k, v, 0, bits);
    __syncthreads();
    last[threadIdx.x] = k[kSmallItems - 1];
    __syncthreads();
    uint32_t heads = 0, prev = threadIdx.x > 0 ? last[threadIdx.x - 1] : 0u;
#pragma unroll
    for (int i = 0; i < kSmallItems; ++i) {
      const int at = threadIdx.x * kSmallItems + i;
      heads |= at < n && k[i] < end && (at == 0 || k[i] != prev) ? 1u << i : 0u;
      prev = k[i];
    }
    return heads;
  }
};

// Scratch of the two, by subgroup (sums: the sums of the quartets' powers that occur, a bit each, 13 for each of
// the four primitives; pows: the largest powers that occur, 5 bits each; total: the largest sum) and by place in the
// sorted list.
struct SmallScratch {
  unsigned long long* sums;
  uint32_t *pows, *sub_key;
  int *sub_grp, *total, *place_sub;
};

// The quartets that passed, sorted by subgroup, and everything that k_sub and the passes around it give: subgroups,
// their powers, sizes and places, groups, and the counters.
__global__ void __launch_bounds__(kSmallThreads)
k_small_groups(int n, int key_bits, const uint64_t* __restrict__ key, uint32_t fail_key, const int4* __restrict__ ijkl,
               const PrimD* __restrict__ prims, int64_t* idx, int64_t* sub_off, SubPowers* powers, SubSize* sub_at,
               int64_t* grp_sub, SmallScratch x, unsigned long long* count) {
  __shared__ SmallBlock B;
  const int t0 = threadIdx.x * kSmallItems;
  const int npass = static_cast<int>(count[kNScreen1]);
  int nsub = 0, ngroup = 0;
  if (threadIdx.x == 0) B.coef = 0;
  {
    uint32_t k[kSmallItems];
    int v[kSmallItems];
#pragma unroll
    for (int i = 0; i < kSmallItems; ++i) {
      k[i] = t0 + i < n ? static_cast<uint32_t>(key[t0 + i]) : 0xFFFFFFFFu;
      v[i] = t0 + i;
    }
    const uint32_t heads = B.sort_runs(k, v, key_bits, n, fail_key);
    int s = B.before(heads, &nsub) - 1;
#pragma unroll
    for (int i = 0; i < kSmallItems; ++i) {
      if (t0 + i < n) idx[t0 + i] = v[i];
      if ((heads >> i) & 1u) {
        ++s;
        sub_off[s] = t0 + i;
        x.sub_key[s] = k[i];
        x.sums[s] = 0;
        x.pows[s] = 0;
      }
      if (t0 + i < npass) x.place_sub[t0 + i] = s;
    }
  }
  __syncthreads();
  for (int p = threadIdx.x; p < npass; p += kSmallThreads) {
    const int4 q = ijkl[idx[p]];
    const int at[4] = {q.x - 1, q.y - 1, q.z - 1, q.w - 1}, s = x.place_sub[p];
    uint32_t pows = 0;
    unsigned long long sums = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const PrimD& P = prims[at[j]];
      pows |= 1u << (5 * j + max(P.t[0], max(P.t[1], P.t[2])));
      sums |= 1ull << (13 * j + P.t[0] + P.t[1] + P.t[2]);
    }
    atomicOr(&x.pows[s], pows);
    atomicOr(&x.sums[s], sums);
  }
  __syncthreads();
  for (int s = threadIdx.x; s < nsub; s += kSmallThreads) {
    // (the masks were changed by atomics, which leave the first-level cache alone)
    const uint32_t pows = __ldcg(&x.pows[s]);
    const unsigned long long sums = __ldcg(&x.sums[s]);
    SubPowers P;
    int total = 0, m = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      P.m[j] = static_cast<uint8_t>(31 - __clz(static_cast<int>((pows >> (5 * j)) & 31u)));
      m += P.m[j];
      total += 31 - __clz(static_cast<int>((sums >> (13 * j)) & 8191u));
    }
    P.total = min(total, kMaxTotal);
    powers[s] = P;
    x.total[s] = total;
    const int ent = sub_entries(P, (s + 1 < nsub ? sub_off[s + 1] : npass) - sub_off[s]);
    sub_at[s] = SubSize{ent, static_cast<int64_t>(ent) * (m + 2)};
  }
  __syncthreads();
  // places of the subgroups, and the groups: kSmallItems subgroups a thread
  SubSize at{0, 0}, all;
  uint32_t heads = 0;
#pragma unroll 4
  for (int i = 0; i < kSmallItems; ++i) {
    const int s = t0 + i;
    if (s >= nsub) break;
    at = at + sub_at[s];
    heads |= s == 0 || (x.sub_key[s] ^ x.sub_key[s - 1]) >> 2 != 0 ? 1u << i : 0u;
  }
  SmallBlock::SizeScan(B.u.size).ExclusiveScan(at, at, SubSize{0, 0}, cuda::std::plus<>(), all);
  __syncthreads();
  int g = B.before(heads, &ngroup) - 1;
  unsigned need = 0;  // added up by warps: an addition to shared memory for every group took 90 us of 3 081
#pragma unroll 1
  for (int i = 0; i < kSmallItems; ++i) {
    const int s = t0 + i;
    if (s >= nsub) break;
    const SubSize mine = sub_at[s];
    sub_at[s] = at;
    at = at + mine;
    if ((heads >> i) & 1u) {
      grp_sub[++g] = s;
      const uint32_t group = x.sub_key[s] >> 2;  // the most that the group's record can need, as in k_sub
      int total = 0;
      int64_t cost = 0;
      for (int t = s; t < nsub && x.sub_key[t] >> 2 == group; ++t) {
        cost += ((t + 1 < nsub ? sub_off[t + 1] : npass) - sub_off[t]) * product_cost(x.total[t]);
        total = max(total, x.total[t]);
      }
      int most = min(total, kMaxTotal);
      while (most > 0 && merged_cost(most) > cost) --most;
      need += static_cast<unsigned>(record_scratch(merged_coefs(most), most));
    }
    x.sub_grp[s] = g;
  }
  need = __reduce_add_sync(0xffffffffu, need);
  if ((threadIdx.x & 31) == 0) atomicAdd(&B.coef, static_cast<unsigned long long>(need));
  __syncthreads();
  if (threadIdx.x == 0) {
    count[kNSub] = static_cast<unsigned long long>(nsub);
    count[kNGroup] = static_cast<unsigned long long>(ngroup);
    count[kNEntry] = static_cast<unsigned long long>(all.ent);
    count[kNTable] = static_cast<unsigned long long>(all.tab);
    count[kNCoef] = B.coef;
  }
}

// The shared values of the subgroups s0 to s1 (a slab's), a thread each.
__global__ void k_sub_const(const __grid_constant__ PrepConst cP, int64_t s0, int64_t s1, int64_t nsub, int64_t npass,
                            const int64_t* __restrict__ sub_off, const int64_t* __restrict__ idx,
                            const int4* __restrict__ ijkl, const PrimD* __restrict__ prims,
                            const SubPowers* __restrict__ powers, SubConst* sub) {
  const int64_t s = s0 + blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (s >= s1) return;
  const int4 q = ijkl[idx[sub_off[s]]];
  const PrimD &Pi = prims[q.x - 1], &Pj = prims[q.y - 1], &Pk = prims[q.z - 1], &Pl = prims[q.w - 1];
  SubConst c;
  shared_of(Pi, Pj, Pk, Pl, &c);
  const SubPowers P = powers[s];
  for (int k = 0; k < 4; ++k) c.m[k] = P.m[k];
  c.lim = cP.thresh * Pi.lim_scale;
  c.mol = Pi.mol;
  c.total = P.total;
  const bool one = (s + 1 < nsub ? sub_off[s + 1] : npass) - sub_off[s] == 1;
#pragma unroll
  for (int d = 0; d < 3; ++d)
    c.single[d] = one ? SubConst::kSingle | static_cast<uint32_t>(Pi.t[d] | Pj.t[d] << 3 | Pk.t[d] << 6 | Pl.t[d] << 9) : 0u;
  sub[s] = c;
}

// First group, subgroup, quartet, entry and table place of each slab: the first group that starts at or
// after the slab's share of the table (and the end of the last slab).
__global__ void k_slabs(int nslab, int64_t ngroup, int64_t nsub, int64_t npass, int64_t nentry, int64_t ntable,
                        const int64_t* __restrict__ grp_sub, const int64_t* __restrict__ sub_off,
                        const SubSize* __restrict__ off, int64_t* bound) {
  for (int k = threadIdx.x; k <= nslab; k += blockDim.x) {
    const int64_t want = ntable / nslab * k;
    int64_t lo = 0, hi = ngroup;
    while (lo < hi) {
      const int64_t mid = (lo + hi) / 2;
      if (off[grp_sub[mid]].tab < want) lo = mid + 1; else hi = mid;
    }
    if (k == nslab) lo = ngroup;
    bound[5 * k] = lo;
    bound[5 * k + 1] = lo < ngroup ? grp_sub[lo] : nsub;
    bound[5 * k + 2] = lo < ngroup ? sub_off[grp_sub[lo]] : npass;
    bound[5 * k + 3] = lo < ngroup ? off[grp_sub[lo]].ent : nentry;
    bound[5 * k + 4] = lo < ngroup ? off[grp_sub[lo]].tab : ntable;
  }
}

// What k_group needs of a quartet, in sorted order (its loads are then consecutive, not a chain
// through indices and primitives): the combination of powers (10 bits) and their sum (5 bits) in each
// dimension.
struct QuartetDesc {
  uint64_t w;
  __device__ __forceinline__ int combo(int d) const { return static_cast<int>(w >> (10 * d)) & 1023; }
  __device__ __forceinline__ int degree(int d) const { return static_cast<int>(w >> (30 + 5 * d)) & 31; }
};

// The powers of a table entry's polynomial, in dimension d.
__device__ __forceinline__ void entry_powers(const SubConst& c, int d, int combo, int t[4]) {
  const uint32_t own = c.single[d];
#pragma unroll
  for (int j = 3; j >= 0; --j) {
    t[j] = own ? static_cast<int>(own >> (3 * j)) & 7 : combo % (c.m[j] + 1);
    combo /= c.m[j] + 1;
  }
}

// A subgroup by bisection (s0 to s1 - 1): the last that starts at or before place p.
__device__ __forceinline__ int64_t subgroup_of(const int64_t* __restrict__ sub_off, int64_t s0, int64_t s1, int64_t p) {
  int64_t lo = s0, hi = s1 - 1;
  while (lo < hi) {
    const int64_t mid = (lo + hi + 1) / 2;
    if (sub_off[mid] <= p) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// The quartets in sorted order, a thread each (its subgroup by bisection: a warp per subgroup left most
// lanes idle where shells have one to nine quartets, 44 us on CH4 against 15): descriptor and amplitude
// A, a mark at the polynomials that it uses (a byte per table entry), and how many of each degree there
// are. Constants are written at once. s0, s1, p0, p1, e0, t0: the slab's subgroups, quartets, first table
// entry and its place in the table.
__global__ void __launch_bounds__(256)
k_mark(const __grid_constant__ PrepConst cP, int64_t s0, int64_t s1, int64_t p0, int64_t p1,
       const int64_t* __restrict__ sub_off,
       const int64_t* __restrict__ idx, const int4* __restrict__ ijkl, const double* __restrict__ v,
       const PrimD* __restrict__ prims, const SubConst* __restrict__ sub, const SubSize* __restrict__ off, int64_t e0,
       int64_t t0, QuartetDesc* desc, double* amp, uint8_t* mark, double* table, unsigned long long* count) {
  __shared__ unsigned int sh[kMaxCoef];
  if (threadIdx.x < kMaxCoef) sh[threadIdx.x] = 0;
  __syncthreads();
  const int64_t p = p0 + blockIdx.x * 256LL + threadIdx.x;
  if (p < p1) {
    const int64_t from = idx[p];
    const int4 q = ijkl[from];
    const PrimD &Pi = prims[q.x - 1], &Pj = prims[q.y - 1], &Pk = prims[q.z - 1], &Pl = prims[q.w - 1];
    const int64_t lo = subgroup_of(sub_off, s0, s1, p);
    const SubConst& c = sub[lo];
    const int combos = c.combos();
    const int64_t first = off[lo].ent - e0;
    amp[p] = (dm_value(cP, Pi, Pj, Pk, Pl, v[from]) * c.c1) * c.c2;
    uint64_t w = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int combo = c.combo(Pi.t[d], Pj.t[d], Pk.t[d], Pl.t[d]), L = Pi.t[d] + Pj.t[d] + Pk.t[d] + Pl.t[d];
      const int64_t at = first + d * combos + combo;
      const unsigned bit = 1u << (8 * (at & 3));
      if (!mark[at] && !(atomicOr(reinterpret_cast<unsigned*>(mark + (at & ~int64_t(3))), bit) & bit)) {
        if (L > 0) {
          atomicAdd(&sh[L], 1u);
        } else {
          double* out = table + (off[lo].tab - t0) + static_cast<int64_t>(d * combos + combo) * c.entry();
          out[0] = inca_gh::kWeight[1][0] * cP.wm[0];
          out[1] = inca_gh::kWeight[1][0];
        }
      }
      w |= static_cast<uint64_t>(combo) << (10 * d);
      w |= static_cast<uint64_t>(L) << (30 + 5 * d);
    }
    desc[p].w = w;
  }
  __syncthreads();
  if (threadIdx.x < kMaxCoef && sh[threadIdx.x])
    atomicAdd(&count[kNTask + threadIdx.x], static_cast<unsigned long long>(sh[threadIdx.x]));
}

struct PolyTask {
  uint32_t sub, entry;  // within the slab
};

// The marked polynomials, those of one degree together (a warp then solves systems of one size), 16
// lanes per subgroup, or four where a subgroup has up to four entries on average (108 000 of three: 60 us with 16 lanes,
// 14 with four; CH4: 13 and 28). next: how many of each degree are listed so far (their order differs from run to
// run; each is solved by itself).
__device__ __forceinline__ void list_polynomials(
    int64_t s0, int64_t s1, const SubConst* __restrict__ sub, const SubSize* __restrict__ off, int64_t e0,
    const uint8_t* __restrict__ mark, const unsigned long long* __restrict__ count, unsigned int* next,
    PolyTask* task, int team) {
  __shared__ unsigned int need[kMaxCoef], base[kMaxCoef];
  for (int i = threadIdx.x; i < kMaxCoef; i += blockDim.x) need[i] = 0;
  __syncthreads();
  const int64_t s = s0 + blockIdx.x * static_cast<int64_t>(blockDim.x / team) + threadIdx.x / team;
  const uint8_t* at = s < s1 ? mark + (off[s].ent - e0) : mark;
  const int combos = s < s1 ? sub[s].combos() : 0;
  for (int pass = 0; pass < 2; ++pass) {
    for (int e = threadIdx.x % team; e < 3 * combos; e += team) {
      if (!at[e]) continue;
      int t[4];
      entry_powers(sub[s], e / combos, e % combos, t);
      const int L = t[0] + t[1] + t[2] + t[3];
      if (L == 0) continue;
      const unsigned place = atomicAdd(&need[L], 1u);
      if (pass == 1) task[base[L] + place] = PolyTask{static_cast<uint32_t>(s - s0), static_cast<uint32_t>(e)};
    }
    __syncthreads();
    if (pass == 0) {
      const int L = threadIdx.x;
      if (L < kMaxCoef) {
        unsigned before = 0;
        for (int k = 1; k < L; ++k) before += static_cast<unsigned>(count[kNTask + k]);
        base[L] = need[L] ? before + atomicAdd(&next[L], need[L]) : 0;
        need[L] = 0;
      }
      __syncthreads();
    }
  }
}

// The listed polynomials, a thread each: U = sum C_m wm_m, then C highest degree first. kT: the largest
// power of the basis.
template <int kT>
__global__ void __launch_bounds__(128)
k_poly(const __grid_constant__ PrepConst cP, const PolyTask* __restrict__ task,
       const unsigned long long* __restrict__ count, int64_t s0,
       const SubConst* __restrict__ sub, const SubSize* __restrict__ off, int64_t t0, double* table) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  unsigned long long ntask = 0;
#pragma unroll
  for (int k = 1; k < kMaxCoef; ++k) ntask += count[kNTask + k];
  if (i >= static_cast<int64_t>(ntask)) return;
  const PolyTask T = task[i];
  const SubConst& c = sub[s0 + T.sub];
  const int combos = c.combos(), d = static_cast<int>(T.entry) / combos;
  int t[4];
  entry_powers(c, d, static_cast<int>(T.entry) - d * combos, t);
  const double R[4] = {c.R[0][d], c.R[1][d], c.R[2][d], c.R[3][d]};
  const double Pik = c.Pik[d], Pjl = c.Pjl[d], Pijkl = c.Pijkl[d], sqe = c.sqe, invz = c.invz, alf = c.alf;
  const int L = t[0] + t[1] + t[2] + t[3];
  double* out = table + (off[s0 + T.sub].tab - t0) + static_cast<int64_t>(T.entry) * c.entry();
  auto finish = [&](const double* C, int n) {
    double U = 0.0;
    for (int m = 0; m < n; ++m) U = U + C[m] * cP.wm[m];
    out[0] = U;
    for (int m = 0; m < n; ++m) out[1 + m] = C[m];
  };
#define INCA_POLY(NP)                                               \
  case NP - 1: {                                                    \
    double C[NP];                                                   \
    polycoef_n<NP, kT>(cP, R, Pik, Pjl, Pijkl, t, sqe, invz, alf, C);   \
    double U = 0.0;                                                 \
    _Pragma("unroll") for (int m = 0; m < NP; ++m) U = U + C[m] * cP.wm[m]; \
    out[0] = U;                                                     \
    _Pragma("unroll") for (int m = 0; m < NP; ++m) out[1 + m] = C[m]; \
    break;                                                          \
  }
  switch (L) {
    INCA_POLY(2)
    INCA_POLY(3)
    INCA_POLY(4)
    INCA_POLY(5)
    default:
      if (kT > 1) {
        double C[kMaxCoef];
        polycoef(cP, R, Pik, Pjl, Pijkl, t, sqe, invz, alf, C);
        finish(C, L + 1);
      }
  }
#undef INCA_POLY
}

// Class key of a record: molecule, kind, degrees (w bits each: enough for the basis's powers, so
// the class sort runs over few bits).
__device__ __forceinline__ uint32_t class_key(int mol, int shape, int w) {
  uint32_t k = static_cast<uint32_t>(mol) * 2 + ((shape & kMergedBit) ? 1 : 0);
#pragma unroll
  for (int f = 0; f < 4; ++f) k = (k << w) | static_cast<uint32_t>((shape >> (5 * f)) & 31);
  return k;
}

// A group: where its coefficients are, what it holds and what its quartets share.
struct GroupRec {
  double sqe, d[3];
  int64_t scratch;  // place of its numbers (merged)
  int64_t first;    // its first quartet in the sorted list
  int shape, mol;
  int quartets, ks;
};

__device__ __forceinline__ void hi_lo(double x, float* hi, float* lo) {
  *hi = static_cast<float>(x);
  *lo = static_cast<float>(x - static_cast<double>(*hi));
}

// Screen 2 (src/mod_intracule.f90:301-343) of a group's quartets and their merged polynomial. amp: A of
// each surviving quartet (0 for the others), in sorted order. Threads first take a quartet each (A, three
// table values U), then a coefficient each, over the quartets in sorted order: two FP64 instructions a
// quartet and coefficient. FP64 issue bounds the work (a warp's FP64 instruction takes 16 cycles of its
// SM however many lanes it has), so a group gets the threads that it fills: eight lanes up to kTinyGroup
// quartets of total degree up to kTinyTotal, a warp up to kSmallGroup quartets, four warps beyond; a thread
// for one quartet of total degree up to 1 (108 000 of s shells of one function each: 102 us with eight lanes, 34 so).
// One launch takes the four lists, large groups first. (A warp for every group up to 64 quartets and a
// second launch for the others: 117 + 44 us on CH4, 79 so.)
// The merged record's numbers (see k_write) go to the next free place of scratch (which place differs
// from run to run; what is stored does not).
constexpr int kSmallGroup = 64, kTinyGroup = 16, kTinyTotal = 4;
constexpr int kTinyTeam = 8, kTinyD = kTinyTotal + 1, kTinyPer = 5;  // lanes, coefficients a dimension, a lane
static_assert(kTinyTeam * kTinyPer >= (kTinyD * (kTinyD + 1) * (kTinyD + 2)) / 6, "a tiny group's coefficients");
constexpr int kGroupThreads = 128;

struct GroupArgs {
  const int64_t* grp_sub;
  const int64_t* sub_off;
  int64_t nsub, npass, ngroup;
  const SubConst* sub;
  const SubSize* off;
  int64_t t0;
  const double* table;
  const int64_t* idx;
  const QuartetDesc* desc;
  double* amp;
  uint8_t* flags;
  double* s2;
  int D, nc_max, smem;  // smem: bytes of a warp's group
  double* scratch;
  GroupRec* grp;
  // of the slab's nlist groups; list: tiny ones from the front, a warp's from the back; large: single ones from the back
  int64_t *gcount, *list, *large;
  int64_t nlist;
  unsigned long long* count;
};

// The groups of a slab by size.
__device__ __forceinline__ void list_groups(int64_t g0, int64_t g1, int64_t block, const GroupArgs& a) {
  const int64_t g = g0 + block * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int cls = -1;
  if (g < g1) {
    const int64_t sub0 = a.grp_sub[g], sub1 = g + 1 < a.ngroup ? a.grp_sub[g + 1] : a.nsub;
    const int64_t size = (sub1 < a.nsub ? a.sub_off[sub1] : a.npass) - a.sub_off[sub0];
    int total = 0;
    for (int64_t s = sub0; s < sub1; ++s) total = max(total, a.sub[s].total);
    cls = size > kSmallGroup ? 2 : size == 1 && total <= 1 ? 3 : size <= kTinyGroup && total <= kTinyTotal && sub1 - sub0 <= 4 ? 0 : 1;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const unsigned on = __ballot_sync(0xffffffffu, cls == k);
    if (!on) continue;
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(&a.count[kNSmall + k], static_cast<unsigned long long>(__popc(on)));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(on & ((1u << lane) - 1u));
    if (cls == k) (k >= 2 ? a.large : a.list)[k & 1 ? a.nlist - 1 - at : at] = g;
  }
}

// Both lists of a slab in one launch: the first poly_blocks blocks the polynomials, the others the groups.
constexpr int kListThreads = 128;
__global__ void __launch_bounds__(kListThreads)
k_list(unsigned poly_blocks, int team, int64_t s0, int64_t s1, int64_t g0, int64_t g1, int64_t e0, const uint8_t* __restrict__ mark,
       unsigned int* next, PolyTask* task, GroupArgs a) {
  if (blockIdx.x < poly_blocks)
    list_polynomials(s0, s1, a.sub, a.off, e0, mark, a.count, next, task, team);
  else
    list_groups(g0, g1, blockIdx.x - poly_blocks, a);
}

// The numbers of a preparation that a thread has seen.
struct GroupSums {
  unsigned long long nsurv, nrec, nprod;
};

// Shared memory of a warp of group_body: its sums of the coefficients, the polynomials of 32 quartets (D
// coefficients a dimension), the powers of each coefficient and the place of x^a y^b z^0 (a D + b).
__host__ __device__ inline int group_smem(int nc_max, int D) {
  return static_cast<int>(
      (sizeof(double) * (nc_max + 32 * 3 * D) + sizeof(uint16_t) * (nc_max + D * D) + 15) & ~size_t(15));
}

// One group by a warp (kThreads = 32) or a block. A warp takes 32 quartets of a subgroup at a time, and
// of each the (L_x + 1)(L_y + 1)(L_z + 1) products of its three polynomials, a lane each, into its own
// sums: at most 48 of a d shell's 165 coefficients (a coefficient per lane over all quartets multiplied
// mostly zeros: 1.76 ms for 100 primitives against 1.32).
template <int kThreads>
__device__ __forceinline__ void group_body(const PrepConst& cP, const GroupArgs& a, int64_t g, int tid, unsigned char* dsm, int* sh,
                                           unsigned long long* sh64, GroupSums* sums) {
  constexpr int kWarps = kThreads / 32;
  const int lane = tid & 31, warp = tid >> 5, D = a.D;
  auto sums_of = [&](int w) { return reinterpret_cast<double*>(dsm + w * a.smem); };
  double* acc = sums_of(warp);
  double* pol = acc + a.nc_max;
  uint16_t* xyz = reinterpret_cast<uint16_t*>(pol + 32 * 3 * D);
  uint16_t* pos = xyz + a.nc_max;
  unsigned long long &sh_cost = sh64[0], &sh_at = sh64[1], &sh_big = sh64[2];  // big: bits of the largest |coefficient|
  const SubConst* sub = a.sub;
  const int64_t *sub_off = a.sub_off, nsub = a.nsub, npass = a.npass;
  auto sync = [] {
    if (kThreads == 32) __syncwarp(); else __syncthreads();
  };
  sync();
  if (tid == 0) {
    sh[0] = sh[1] = 0;
    sh_cost = sh_big = 0;
  }
  sync();
  const int64_t sub0 = a.grp_sub[g], sub1 = g + 1 < a.ngroup ? a.grp_sub[g + 1] : nsub;
  const int64_t m0 = sub_off[sub0];
  int total = 0, alive = 0;
  unsigned long long cost = 0;
  for (int64_t s = sub0; s < sub1; ++s) {
    const SubConst& c = sub[s];
    const int64_t p1 = s + 1 < nsub ? sub_off[s + 1] : npass;
    const int combos = c.combos(), len = c.entry();
    const double* tab = a.table + (a.off[s].tab - a.t0);
    for (int64_t p = sub_off[s] + tid; p < p1; p += kThreads) {
      const int64_t q = a.idx[p];
      const QuartetDesc Q = a.desc[p];
      const double A = a.amp[p];
      double U[3];
      int sum = 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        U[d] = tab[(d * combos + Q.combo(d)) * len];
        sum += Q.degree(d);
      }
      const double screen2 = fabs(((A * U[0]) * U[1]) * U[2]);
      const bool ok = screen2 >= c.lim;
      if (a.s2) a.s2[q] = screen2;
      if (ok) a.flags[q] = 3;
      if (!ok) a.amp[p] = 0.0;
      if (ok) {
        ++alive;
        total = max(total, sum);
        cost += product_cost(sum);
      }
    }
  }
  alive = __reduce_add_sync(0xffffffffu, alive);
  total = __reduce_max_sync(0xffffffffu, total);
  for (int o = 16; o > 0; o >>= 1) cost += __shfl_xor_sync(0xffffffffu, cost, o);
  if (kThreads > 32) {
    if (lane == 0) {
      atomicMax(&sh[0], total);
      atomicAdd(&sh[1], alive);
      atomicAdd(&sh_cost, cost);
    }
    sync();
    total = sh[0];
    alive = sh[1];
    cost = sh_cost;
  }
  if (alive == 0) {
    if (tid == 0) a.gcount[g] = 0;
    return;
  }
  const bool merged = total <= kMaxTotal && merged_cost(total) <= cost;
  const int nc = merged ? merged_coefs(total) : 0;
  if (tid == 0) {
    sums->nsurv += alive;
    sums->nrec += merged ? 1 : alive;
    sums->nprod += merged ? 0 : alive;
    sh_at = merged ? atomicAdd(&a.count[kNUsed], static_cast<unsigned long long>(record_scratch(nc, total))) : 0;
  }
  sync();
  double* out = a.scratch + sh_at;
  if (merged) {
    {
      int i = 0;
      for (int x = total; x >= 0; --x)
        for (int y = total - x; y >= 0; --y) {
          const int nz = total - x - y;
          if (lane == 0) pos[x * D + y] = static_cast<uint16_t>(i + nz);
          for (int z = nz - ((lane - i) & 31); z >= 0; z -= 32) {
            xyz[i + nz - z] = static_cast<uint16_t>(x | (y << 5) | (z << 10));
            acc[i + nz - z] = 0.0;
          }
          i += nz + 1;
        }
    }
    for (int64_t s = sub0; s < sub1; ++s) {
      const SubConst& c = sub[s];
      const int64_t p1 = s + 1 < nsub ? sub_off[s + 1] : npass;
      const int combos = c.combos(), len = c.entry();
      const double* tab = a.table + (a.off[s].tab - a.t0);
      for (int64_t b = sub_off[s] + 32 * warp; b < p1; b += 32 * kWarps) {
        __syncwarp();
        double A = 0.0;
        unsigned degrees = 0;
        if (b + lane < p1) {  // A C_x, C_y and C_z of a quartet, ascending powers (A = 0: not a survivor)
          A = a.amp[b + lane];
          const QuartetDesc Q = a.desc[b + lane];
          degrees = static_cast<unsigned>(Q.w >> 30);
          double* to = pol + lane * 3 * D;
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const int l = Q.degree(d);
            const double* C = tab + (d * combos + Q.combo(d)) * len + 1 + l;
            for (int p = 0; p <= l; ++p) to[d * D + p] = d == 0 ? A * C[-p] : C[-p];
          }
        }
        uint32_t on = __ballot_sync(0xffffffffu, A != 0.0);
        while (on) {
          const int q = __ffs(on) - 1;
          on &= on - 1;
          const unsigned L = __shfl_sync(0xffffffffu, degrees, q);
          const int nz = static_cast<int>(L >> 10 & 31) + 1, nyz = (static_cast<int>(L >> 5 & 31) + 1) * nz;
          const int n = (static_cast<int>(L & 31) + 1) * nyz;
          const float rz = __frcp_rn(static_cast<float>(nz)), ryz = __frcp_rn(static_cast<float>(nyz));
          const double* P = pol + q * 3 * D;
          __syncwarp();
          for (int i = lane; i < n; i += 32) {
            const int x = static_cast<int>((static_cast<float>(i) + 0.5f) * ryz), yz = i - x * nyz;
            const int y = static_cast<int>((static_cast<float>(yz) + 0.5f) * rz), z = yz - y * nz;
            const int at = pos[x * D + y] - z;
            acc[at] = fma(P[x] * P[D + y], P[2 * D + z], acc[at]);
          }
        }
      }
    }
    sync();
    // powers of u, divided by the power of two above the largest coefficient, as FP32 pairs
    double big = 0.0;
    acc = sums_of(0);
    xyz = reinterpret_cast<uint16_t*>(acc + a.nc_max + 32 * 3 * D);
    for (int i = tid; i < nc; i += kThreads) {
      const int deg = (xyz[i] & 31) + ((xyz[i] >> 5) & 31) + (xyz[i] >> 10);
      double t = acc[i];
      for (int w = 1; w < kWarps; ++w) t += sums_of(w)[i];
      out[i] = t * ipow(sub[sub0].sqe, deg);
      t *= cP.cu_inv_pow[deg];
      acc[i] = t;
      big = fmax(big, fabs(t));
    }
    atomicMax(&sh_big, static_cast<unsigned long long>(__double_as_longlong(big)));
    sync();
    big = __longlong_as_double(static_cast<long long>(sh_big));
    int ks = 0;
    if (big > 0.0) frexp(big, &ks);
    float* f = reinterpret_cast<float*>(out + nc);
    for (int i = tid; i < nc; i += kThreads) {
      float h, l;
      hi_lo(ldexp(acc[i], -ks), &h, &l);
      f[i] = h;
      f[nc + i] = l;
      const int x = xyz[i] & 31, y = (xyz[i] >> 5) & 31, z = xyz[i] >> 10;
      float* term = reinterpret_cast<float*>(&acc[i]);  // |c| and its weight a! b! c! / k!
      term[0] = fabsf(h);
      term[1] = cP.fact[x] * cP.fact[y] / cP.fact[x + y + z] * cP.fact[z];
      xyz[i] = static_cast<uint16_t>(x + y + z);
    }
    sync();
    for (int k = warp; k <= total; k += kWarps) {  // S of a degree, in FP32 relative to its largest coefficient
      float top = 0.0f, sum = 0.0f;
      for (int i = lane; i < nc; i += 32)
        if (xyz[i] == k) top = fmaxf(top, reinterpret_cast<const float*>(&acc[i])[0]);
      for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      // (at least 2^-100, so that the reciprocal stays finite and the squares do not vanish)
      const float cmax = fmaxf(top, 7.8886091e-31f), scale = 1.0f / cmax;
      for (int i = lane; i < nc; i += 32)
        if (xyz[i] == k) {
          const float* term = reinterpret_cast<const float*>(&acc[i]);
          const float y = term[0] * scale;
          sum += y * y * term[1];
        }
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      // raised by a margin for its own rounding and that of the evaluation's |u|
      if (lane == 0) f[2 * nc + total - k] = cmax * sqrtf(sum) * (1.0f + 2e-5f + 1e-6f * static_cast<float>(k));
    }
    if (tid == 0) a.grp[g].ks = ks;
  }
  if (tid == 0) {
    const SubConst& c = sub[sub0];
    GroupRec& R = a.grp[g];
    R.sqe = c.sqe;
    for (int d = 0; d < 3; ++d) R.d[d] = c.Pik[d] - c.Pjl[d];
    R.scratch = static_cast<int64_t>(sh_at);
    R.first = m0;
    R.shape = merged ? merged_shape(total) : 0;
    R.mol = c.mol;
    R.quartets = alive;
    a.gcount[g] = merged ? 1 : alive;
  }
}

// kGroupThreads / kTinyTeam groups of the tiny list from `first` on, eight lanes each. The lanes of a warp
// stay together: what differs between its groups is predicated.
__device__ __forceinline__ void tiny_groups(const PrepConst& cP, const GroupArgs& a, int64_t first, int64_t ntiny, unsigned char* dsm,
                                            const uint16_t* powers, GroupSums* sums) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, l = threadIdx.x % kTinyTeam, team = threadIdx.x / kTinyTeam;
  double* pol = reinterpret_cast<double*>(dsm) + team * kTinyTeam * 3 * kTinyD;
  const int64_t item = first + team;
  const bool on = item < ntiny;
  const int64_t g = on ? a.list[item] : 0;
  const int64_t sub0 = on ? a.grp_sub[g] : 0, sub1 = !on ? 0 : g + 1 < a.ngroup ? a.grp_sub[g + 1] : a.nsub;
  const int64_t m0 = on ? a.sub_off[sub0] : 0, m1 = !on ? 0 : sub1 < a.nsub ? a.sub_off[sub1] : a.npass;
  int64_t start[3];  // of the second to fourth subgroup
#pragma unroll
  for (int k = 0; k < 3; ++k) start[k] = sub0 + k + 1 < sub1 ? a.sub_off[sub0 + k + 1] : m1;
  double A[2];
  uint64_t desc[2];
  const double* tab[2];
  int combos[2], len[2];
  int alive = 0, total = 0, cost = 0;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int64_t p = m0 + l + kTinyTeam * r;
    A[r] = 0.0;
    desc[r] = 0;
    tab[r] = a.table;
    combos[r] = len[r] = 0;
    if (p < m1) {
      const int64_t s = sub0 + (p >= start[0]) + (p >= start[1]) + (p >= start[2]);
      const SubConst& c = a.sub[s];
      const int64_t q = a.idx[p];
      const QuartetDesc Q = a.desc[p];
      A[r] = a.amp[p];
      combos[r] = c.combos();
      len[r] = c.entry();
      tab[r] = a.table + (a.off[s].tab - a.t0);
      desc[r] = Q.w;
      double U[3];
      int sum = 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        U[d] = tab[r][(d * combos[r] + Q.combo(d)) * len[r]];
        sum += Q.degree(d);
      }
      const double screen2 = fabs(((A[r] * U[0]) * U[1]) * U[2]);
      const bool ok = screen2 >= c.lim;
      if (a.s2) a.s2[q] = screen2;
      if (ok) {
        a.flags[q] = 3;
        ++alive;
        total = max(total, sum);
        cost += product_cost(sum);
      } else {
        a.amp[p] = A[r] = 0.0;
      }
    }
  }
#pragma unroll
  for (int o = kTinyTeam / 2; o > 0; o >>= 1) {
    alive += __shfl_xor_sync(kAll, alive, o);
    cost += __shfl_xor_sync(kAll, cost, o);
    total = max(total, __shfl_xor_sync(kAll, total, o));
  }
  const bool merged = alive > 0 && merged_cost(total) <= cost;
  const int nc = merged ? merged_coefs(total) : 0;
  // the warp's records take their places together
  const int64_t need = merged ? record_scratch(nc, total) : 0;
  int64_t before = 0, all = 0;
#pragma unroll
  for (int k = 0; k < 32; k += kTinyTeam) {
    const int64_t n = __shfl_sync(kAll, need, k);
    if (k < lane - l) before += n;
    all += n;
  }
  unsigned long long at = 0;
  if (lane == 0 && all) at = atomicAdd(&a.count[kNUsed], static_cast<unsigned long long>(all));
  at = __shfl_sync(kAll, at, 0) + before;
  double acc[kTinyPer];
#pragma unroll
  for (int t = 0; t < kTinyPer; ++t) acc[t] = 0.0;
  const uint16_t* pw = powers + total * kTinyTeam * kTinyPer;
  int xyz[kTinyPer];
#pragma unroll
  for (int t = 0; t < kTinyPer; ++t) xyz[t] = pw[l + kTinyTeam * t];
  const int most = static_cast<int>(__reduce_max_sync(kAll, static_cast<unsigned>(merged ? m1 - m0 : 0)));
  const int ncs = __reduce_max_sync(kAll, nc);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    if (kTinyTeam * r >= most) break;
    __syncwarp();
    const QuartetDesc Q{desc[r]};
#pragma unroll
    for (int d = 0; d < 3; ++d) {  // A C_x, C_y and C_z, ascending powers (A = 0: not a survivor)
      const int deg = Q.degree(d);
      const double* C = tab[r] + (d * combos[r] + Q.combo(d)) * len[r] + 1 + deg;
#pragma unroll
      for (int p = 0; p < kTinyD; ++p)
        pol[l * 3 * kTinyD + d * kTinyD + p] =
            p > deg || len[r] == 0 || !merged ? 0.0 : d == 0 ? A[r] * C[-p] : C[-p];
    }
    __syncwarp();
    const int k = min(kTinyTeam, most - kTinyTeam * r);
    for (int q = 0; q < k; ++q) {
      const double* P = pol + q * 3 * kTinyD;
#pragma unroll
      for (int t = 0; t < kTinyPer; ++t)
        if (kTinyTeam * t < ncs)
          acc[t] = fma(P[xyz[t] & 31] * P[kTinyD + ((xyz[t] >> 5) & 31)], P[2 * kTinyD + (xyz[t] >> 10)], acc[t]);
    }
  }
  const SubConst& c = a.sub[sub0];
  const double sqe = c.sqe;
  double* out = a.scratch + at;
  double big = 0.0;
  int deg[kTinyPer];
#pragma unroll
  for (int t = 0; t < kTinyPer; ++t) {
    deg[t] = (xyz[t] & 31) + ((xyz[t] >> 5) & 31) + (xyz[t] >> 10);
    if (kTinyTeam * t < ncs && l + kTinyTeam * t < nc) {
      out[l + kTinyTeam * t] = acc[t] * ipow(sqe, deg[t]);
      acc[t] = acc[t] * cP.cu_inv_pow[deg[t]];
      big = fmax(big, fabs(acc[t]));
    } else {
      deg[t] = -1;
    }
  }
#pragma unroll
  for (int o = kTinyTeam / 2; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(kAll, big, o));
  int ks = 0;
  if (big > 0.0) frexp(big, &ks);
  float* f = reinterpret_cast<float*>(out + nc);
  float h[kTinyPer];
#pragma unroll
  for (int t = 0; t < kTinyPer; ++t) {
    h[t] = 0.0f;
    if (deg[t] >= 0) {
      float lo;
      hi_lo(ldexp(acc[t], -ks), &h[t], &lo);
      f[l + kTinyTeam * t] = h[t];
      f[nc + l + kTinyTeam * t] = lo;
    }
  }
  const int degrees = __reduce_max_sync(kAll, total);
  for (int k = 0; k <= degrees; ++k) {  // S of each degree, as in group_body
    float top = 0.0f, sum = 0.0f;
#pragma unroll
    for (int t = 0; t < kTinyPer; ++t)
      if (deg[t] == k) top = fmaxf(top, fabsf(h[t]));
#pragma unroll
    for (int o = kTinyTeam / 2; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(kAll, top, o));
    const float cmax = fmaxf(top, 7.8886091e-31f), scale = 1.0f / cmax;
#pragma unroll
    for (int t = 0; t < kTinyPer; ++t)
      if (deg[t] == k) {
        const float y = fabsf(h[t]) * scale;
        sum += y * y *
               (cP.fact[xyz[t] & 31] * cP.fact[(xyz[t] >> 5) & 31] / cP.fact[k] * cP.fact[xyz[t] >> 10]);
      }
#pragma unroll
    for (int o = kTinyTeam / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(kAll, sum, o);
    if (merged && l == 0 && k <= total)
      f[2 * nc + total - k] = cmax * sqrtf(sum) * (1.0f + 2e-5f + 1e-6f * static_cast<float>(k));
  }
  if (on && l == 0) {
    a.gcount[g] = merged ? 1 : alive;
    if (alive > 0) {
      GroupRec& R = a.grp[g];
      R.sqe = sqe;
      for (int d = 0; d < 3; ++d) R.d[d] = c.Pik[d] - c.Pjl[d];
      R.scratch = static_cast<int64_t>(at);
      R.first = m0;
      R.shape = merged ? merged_shape(total) : 0;
      R.mol = c.mol;
      R.quartets = alive;
      R.ks = ks;
      sums->nsurv += alive;
      sums->nrec += merged ? 1 : alive;
      sums->nprod += merged ? 0 : alive;
    }
  }
}

// A group of one quartet of total degree up to 1, a thread each: the arithmetic of tiny_groups.
static_assert(44 + 1 <= 50 && 44 + 4 + 2 <= 50 + 2, "such a quartet is merged: merged_cost is at most product_cost");
__device__ __forceinline__ void single_groups(const PrepConst& cP, const GroupArgs& a, int64_t item, int64_t nsingle,
                                              GroupSums* sums) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int total = 0, need = 0;
  int64_t g = 0, s = 0, p = 0;
  double P[3][2];
  if (item < nsingle) {
    g = a.large[a.nlist - 1 - item];
    s = a.grp_sub[g];
    p = a.sub_off[s];
    const SubConst& c = a.sub[s];
    const QuartetDesc Q = a.desc[p];
    const double A = a.amp[p];
    const int len = c.entry();
    const double* tab = a.table + (a.off[s].tab - a.t0);
    double U[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int deg = Q.degree(d);
      const double* C = tab + d * len;
      U[d] = C[0];
      P[d][0] = C[1 + deg];
      P[d][1] = deg ? C[1] : 0.0;
      total += deg;
    }
    const double screen2 = fabs(((A * U[0]) * U[1]) * U[2]);
    const int64_t q = a.idx[p];
    if (a.s2) a.s2[q] = screen2;
    if (screen2 >= c.lim) {
      a.flags[q] = 3;
      P[0][0] = A * P[0][0];
      P[0][1] = A * P[0][1];
      need = static_cast<int>(record_scratch(total ? 4 : 1, total));
    } else {
      a.amp[p] = 0.0;
      a.gcount[g] = 0;
    }
  }
  // the warp's records take their places together
  int upto = need;
#pragma unroll
  for (int o = 1; o < 32; o *= 2) {
    const int x = __shfl_up_sync(kAll, upto, o);
    if (lane >= o) upto += x;
  }
  unsigned long long at = 0;
  if (lane == 31 && upto) at = atomicAdd(&a.count[kNUsed], static_cast<unsigned long long>(upto));
  at = __shfl_sync(kAll, at, 31) + (upto - need);
  if (!need) return;
  const SubConst& c = a.sub[s];
  const double sqe = c.sqe;
  const int nc = total ? 4 : 1;
  double* out = a.scratch + at;
  // x, y, z, 1
  const double first[4] = {fma(P[0][1] * P[1][0], P[2][0], 0.0), fma(P[0][0] * P[1][1], P[2][0], 0.0),
                           fma(P[0][0] * P[1][0], P[2][1], 0.0), fma(P[0][0] * P[1][0], P[2][0], 0.0)};
  double t[4], big = 0.0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    t[i] = 0.0;
    const int to = i - (4 - nc);
    if (to < 0) continue;
    out[to] = i < 3 ? first[i] * sqe : first[i];
    t[i] = first[i] * cP.cu_inv_pow[i < 3 ? 1 : 0];
    big = fmax(big, fabs(t[i]));
  }
  int ks = 0;
  if (big > 0.0) frexp(big, &ks);
  float* f = reinterpret_cast<float*>(out + nc);
  float h[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    h[i] = 0.0f;
    const int to = i - (4 - nc);
    if (to < 0) continue;
    float lo;
    hi_lo(ldexp(t[i], -ks), &h[i], &lo);
    f[to] = h[i];
    f[nc + to] = lo;
  }
  for (int k = 0; k <= total; ++k) {
    const float b[3] = {fabsf(k ? h[0] : h[3]), k ? fabsf(h[1]) : 0.0f, k ? fabsf(h[2]) : 0.0f};
    const float cmax = fmaxf(fmaxf(b[0], fmaxf(b[1], b[2])), 7.8886091e-31f), scale = 1.0f / cmax;
    float y[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) y[i] = b[i] * scale;
    const float sum = (y[0] * y[0] + y[2] * y[2]) + y[1] * y[1];
    f[2 * nc + total - k] = cmax * sqrtf(sum) * (1.0f + 2e-5f + 1e-6f * static_cast<float>(k));
  }
  a.gcount[g] = 1;
  GroupRec& R = a.grp[g];
  R.sqe = sqe;
  for (int d = 0; d < 3; ++d) R.d[d] = c.Pik[d] - c.Pjl[d];
  R.scratch = static_cast<int64_t>(at);
  R.first = p;
  R.shape = merged_shape(total);
  R.mol = c.mol;
  R.quartets = 1;
  R.ks = ks;
  ++sums->nsurv;
  ++sums->nrec;
}

__global__ void __launch_bounds__(kGroupThreads, 5)
k_groups(const __grid_constant__ PrepConst cP, GroupArgs a) {
  constexpr int kWarps = kGroupThreads / 32, kTeams = kGroupThreads / kTinyTeam;
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ int sh[kWarps][2];  // total degree, survivors
  __shared__ unsigned long long sh64[kWarps][3];
  __shared__ uint16_t powers[(kTinyTotal + 1) * kTinyTeam * kTinyPer];  // of a tiny group's coefficients
  if (threadIdx.x <= kTinyTotal) {
    const int total = threadIdx.x;
    int i = total * kTinyTeam * kTinyPer;
    const int end = i + kTinyTeam * kTinyPer;
    for (int x = total; x >= 0; --x)
      for (int y = total - x; y >= 0; --y)
        for (int z = total - x - y; z >= 0; --z) powers[i++] = static_cast<uint16_t>(x | (y << 5) | (z << 10));
    while (i < end) powers[i++] = 0;
  }
  const int64_t nlarge = static_cast<int64_t>(a.count[kNLarge]), nwarp = static_cast<int64_t>(a.count[kNMedium]),
                ntiny = static_cast<int64_t>(a.count[kNSmall]), nsingle = static_cast<int64_t>(a.count[kNSingle]);
  const int64_t warp_items = (nwarp + kWarps - 1) / kWarps, tiny_items = (ntiny + kTeams - 1) / kTeams;
  const int64_t items = nlarge + warp_items + tiny_items + (nsingle + kGroupThreads - 1) / kGroupThreads;
  const int warp = threadIdx.x >> 5;
  GroupSums sums{0, 0, 0};
  for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
    __syncthreads();
    if (item < nlarge) {
      group_body<kGroupThreads>(cP, a, a.large[item], threadIdx.x, dsm, sh[0], sh64[0], &sums);
    } else if (item < nlarge + warp_items) {
      const int64_t k = (item - nlarge) * kWarps + warp;
      if (k < nwarp)
        group_body<32>(cP, a, a.list[a.nlist - 1 - k], threadIdx.x & 31, dsm + warp * a.smem, sh[warp], sh64[warp],
                        &sums);
    } else if (item < nlarge + warp_items + tiny_items) {
      tiny_groups(cP, a, (item - nlarge - warp_items) * kTeams, ntiny, dsm, powers, &sums);
    } else {
      single_groups(cP, a, (item - nlarge - warp_items - tiny_items) * kGroupThreads + threadIdx.x, nsingle, &sums);
    }
  }
  __syncwarp();
  for (int o = 16; o > 0; o >>= 1) {
    sums.nsurv += __shfl_xor_sync(0xffffffffu, sums.nsurv, o);
    sums.nrec += __shfl_xor_sync(0xffffffffu, sums.nrec, o);
    sums.nprod += __shfl_xor_sync(0xffffffffu, sums.nprod, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (sums.nsurv) atomicAdd(&a.count[kNSurv], sums.nsurv);
    if (sums.nrec) atomicAdd(&a.count[kNRec], sums.nrec);
    if (sums.nprod) atomicAdd(&a.count[kNProduct], sums.nprod);
  }
}

// Place of a record within its class: centre (cells of 1 bohr, Morton order over +-16 bohr), then reach
// (eighths of a bohr up to 8: how far from it the Gaussian stays above 2^-50), so that the records of a
// chunk matter for the same tiles.
constexpr int kPlaceBits = 21;
__device__ __forceinline__ uint64_t record_place(const PrepConst& cP, const GroupRec& R) {
  uint32_t q[3], k = 0;
  for (int d = 0; d < 3; ++d) q[d] = static_cast<uint32_t>(fmin(fmax(R.d[d] + 16.0, 0.0), 31.0));
  for (int b = 4; b >= 0; --b)
    for (int d = 0; d < 3; ++d) k = (k << 1) | ((q[d] >> b) & 1u);
  const float reach = sqrtf(fmaxf(static_cast<float>(R.ks) + 50.0f, 0.0f)) / static_cast<float>(R.sqe * cP.c_u);
  return (static_cast<uint64_t>(k) << 6) | static_cast<uint32_t>(fminf(reach * 8.0f, 63.0f));
}
struct ClassOfKey {
  int place_bits;
  __device__ uint32_t operator()(uint64_t key) const { return static_cast<uint32_t>(key >> place_bits); }
};

// Sort key (class, and with place_bits its place there) and source of every record: merged records point at their group (>= 0), product records
// at their quartet's place in the sorted list (-1 - place). gstart: first record of each group. A
// thread per group, its warp for the products of one with more than kOwnSpan quartets. (A warp for every group took 88
// us for 108 000 merged records, 7 so.)
constexpr int kOwnSpan = 4;
__global__ void k_record_keys(const __grid_constant__ PrepConst cP, int64_t ngroup_max, const unsigned long long* __restrict__ count,
                              const int64_t* __restrict__ grp_sub, int64_t nsub, const int64_t* __restrict__ sub_off,
                              int64_t npass, const GroupRec* __restrict__ grp, const int64_t* __restrict__ gcount,
                              const int64_t* __restrict__ gstart, const uint8_t* __restrict__ flags,
                              const int64_t* __restrict__ idx, const int4* __restrict__ ijkl,
                              const PrimD* __restrict__ prims, int w, int place_bits, uint64_t* rkey, int64_t* rsrc) {
  const int lane = threadIdx.x & 31;
  const int64_t ngroup = min(ngroup_max, static_cast<int64_t>(count[kNGroup]));
  const int64_t g = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  int64_t at = 0, first = 0, m1 = 0;  // of products: first record, quartets
  int mol = 0;
  auto product = [&](int64_t to, int64_t p, int64_t q, int of) {
    const int4 r = ijkl[q];
    const PrimD &Pi = prims[r.x - 1], &Pj = prims[r.y - 1], &Pk = prims[r.z - 1], &Pl = prims[r.w - 1];
    int L[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) L[d] = Pi.t[d] + Pj.t[d] + Pk.t[d] + Pl.t[d];
    rkey[to] = static_cast<uint64_t>(class_key(of, product_shape(L[0], L[1], L[2]), w)) << place_bits;
    rsrc[to] = -1 - p;
  };
  if (g < ngroup && gcount[g] != 0) {
    const GroupRec& R = grp[g];
    at = gstart[g];
    mol = R.mol;
    if (R.shape & kMergedBit) {
      rkey[at] = (static_cast<uint64_t>(class_key(mol, R.shape, w)) << place_bits) | (place_bits ? record_place(cP, R) : 0);
      rsrc[at] = g;
    } else {
      const int64_t sub1 = g + 1 < ngroup ? grp_sub[g + 1] : nsub;
      first = R.first;
      m1 = sub1 < nsub ? sub_off[sub1] : npass;
      if (m1 - first <= kOwnSpan) {
        for (int64_t p = first; p < m1; ++p) {
          const int64_t q = idx[p];
          if (flags[q] == 3) product(at++, p, q, mol);
        }
        m1 = first;
      }
    }
  }
  __syncwarp();
  unsigned todo = __ballot_sync(0xffffffffu, m1 > first);
  while (todo) {
    const int from = __ffs(todo) - 1;
    todo &= todo - 1;
    int64_t next = __shfl_sync(0xffffffffu, at, from);
    const int64_t b0 = __shfl_sync(0xffffffffu, first, from), b1 = __shfl_sync(0xffffffffu, m1, from);
    const int of = __shfl_sync(0xffffffffu, mol, from);
    for (int64_t b = b0; b < b1; b += 32) {
      const int64_t p = b + lane;
      const int64_t q = p < b1 ? idx[p] : 0;
      const bool ok = p < b1 && flags[q] == 3;
      const unsigned on = __ballot_sync(0xffffffffu, ok);
      if (ok) product(next + __popc(on & ((1u << lane) - 1u)), p, q, of);
      next += __popc(on);
    }
  }
}

// The same of a small list in one block: the records of all groups, sorted by class, their sources, and each
// class's key and count behind the counters.
__global__ void __launch_bounds__(kSmallThreads)
k_small_records(int npass, int cls_bits, const GroupRec* __restrict__ grp, const int64_t* __restrict__ gcount,
                const uint8_t* __restrict__ flags, const int64_t* __restrict__ idx, const int4* __restrict__ ijkl,
                const PrimD* __restrict__ prims, int w, SmallScratch x, uint64_t* rkey, int64_t* rsrc,
                unsigned long long* count) {
  __shared__ SmallBlock B;
  const int t0 = threadIdx.x * kSmallItems, nrec = static_cast<int>(count[kNRec]);
  // key of the record that starts at each place (by place: the block reads and writes places and records in turn)
  for (int p = threadIdx.x; p < npass; p += kSmallThreads) {
    uint32_t key = 0xFFFFFFFFu;  // none
    int src = 0;
    const int g = x.sub_grp[x.place_sub[p]];
    if (gcount[g] > 0) {
      const GroupRec& R = grp[g];
      if (R.shape & kMergedBit) {
        if (p == R.first) {
          key = class_key(R.mol, R.shape, w);
          src = g;
        }
      } else if (flags[idx[p]] == 3) {
        const int4 r = ijkl[idx[p]];
        const PrimD &Pi = prims[r.x - 1], &Pj = prims[r.y - 1], &Pk = prims[r.z - 1], &Pl = prims[r.w - 1];
        int L[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) L[d] = Pi.t[d] + Pj.t[d] + Pk.t[d] + Pl.t[d];
        key = class_key(R.mol, product_shape(L[0], L[1], L[2]), w);
        src = -1 - p;
      }
    }
    rkey[p] = static_cast<uint64_t>(key) << 32 | static_cast<uint32_t>(src);
  }
  __syncthreads();
  int nclass = 0;
  unsigned long long* cls = count + kNCounts;  // key and first record of each class, then its count
  {
    uint32_t k[kSmallItems];
    int v[kSmallItems];
#pragma unroll
    for (int i = 0; i < kSmallItems; ++i) {
      const uint64_t r = t0 + i < npass ? rkey[t0 + i] : ~uint64_t(0);
      k[i] = static_cast<uint32_t>(r >> 32);
      v[i] = static_cast<int>(static_cast<uint32_t>(r));
    }
    const uint32_t heads = B.sort_runs(k, v, cls_bits, nrec, 0xFFFFFFFFu);
    int c = B.before(heads, &nclass) - 1;
#pragma unroll
    for (int i = 0; i < kSmallItems; ++i) {
      if (t0 + i < nrec) rsrc[t0 + i] = v[i];
      if ((heads >> i) & 1u) {
        ++c;
        cls[2 * c] = k[i];
        cls[2 * c + 1] = static_cast<unsigned long long>(t0 + i);
      }
    }
  }
  for (int c0 = 0; c0 < nclass; c0 += kSmallThreads) {
    __syncthreads();
    const int c = c0 + threadIdx.x;
    const unsigned long long n =
        c >= nclass ? 0 : (c + 1 < nclass ? cls[2 * c + 3] : static_cast<unsigned long long>(nrec)) - cls[2 * c + 1];
    __syncthreads();
    if (c < nclass) cls[2 * c + 1] = n;
  }
  if (threadIdx.x == 0) count[kNClass] = static_cast<unsigned long long>(nclass);
}

__device__ __forceinline__ int segment_of(const ClassSeg* __restrict__ segs, int nseg, int64_t r) {
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (segs[mid].first <= r) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Merged records into their class's segment, eight lanes each (most are 8 doubles and 16 to 24 floats):
//   FP64 record [sqe^2 / ln 2, sqe, d0, d1, d2, 0, c_abc...] (powers of r + d, of which the Gaussian
//   is 2^-(first number times their square);
//   FP32 record [s_hi, s_lo, b_hi[3], b_lo[3], 0, quartets, ks, ks, c_hi..., c_lo..., S_total..., S_0]
// with s = sqe c_u, b_d = s d_d, u = s (r + d) = c_u r', the polynomial rewritten in u and divided by
// the power of two 2^ks above its largest coefficient (applied exactly by the evaluation's exp2), and
// S_k = sqrt(sum over a + b + c = k of c_abc^2 a! b! c! / k!): by Cauchy-Schwarz
// sum |c_abc u_x^a u_y^b u_z^c| <= sum_k S_k |u|^k, which the error bounds use (one Horner loop over
// the total degree instead of a second one over all coefficients). hi/lo pairs carry the FP64 value
// to about 2^-48.
__global__ void __launch_bounds__(256)
k_write(const __grid_constant__ PrepConst cP, int64_t nrec, const int64_t* __restrict__ rsrc,
        const GroupRec* __restrict__ grp,
        const double* __restrict__ scratch, const ClassSeg* __restrict__ segs, int nseg, double* rec64, float* rec32) {
  const int64_t r = blockIdx.x * 32LL + (threadIdx.x >> 3);
  if (r >= nrec) return;
  const int lane = threadIdx.x & 7;
  const int64_t g = rsrc[r];
  if (g < 0) return;
  const ClassSeg& sg = segs[segment_of(segs, nseg, r)];
  const int nc = sg.nc, nf = 2 * nc + ((sg.shape >> 15) & 31) + 1;
  const GroupRec& G = grp[g];
  const double* c = scratch + G.scratch;
  const float* f = reinterpret_cast<const float*>(c + nc);
  const int64_t local = r - sg.first;
  double* r64 = rec64 + sg.off64 + local * sg.stride;
  float* r32 = rec32 + sg.off32 + local * sg.stride32;
  for (int i = lane; i < sg.stride - kRecHeader; i += 8) r64[kRecHeader + i] = i < nc ? c[i] : 0.0;
  for (int i = lane; i < sg.stride32 - 12; i += 8) r32[12 + i] = i < nf ? f[i] : 0.0f;
  if (lane == 0) {
    const double s = G.sqe * cP.c_u;
    r64[0] = s * s;
    r64[1] = G.sqe;
    hi_lo(s, &r32[0], &r32[1]);
    for (int d = 0; d < 3; ++d) {
      r64[2 + d] = G.d[d];
      hi_lo(s * G.d[d], &r32[2 + d], &r32[5 + d]);
    }
    r64[5] = 0.0;
    r32[8] = 0.0f;
    r32[9] = static_cast<float>(G.quartets);
    r32[10] = r32[11] = static_cast<float>(G.ks);
  }
}

// Bounds of each chunk, a warp each, from its FP32 records (ChunkWalk reads them; the ranges are widened
// so that no record's own bound, FP32 roundings included, exceeds its chunk's).
__global__ void k_chunk_bounds(int nchunks, const WorkChunk* __restrict__ chunks, const ClassSeg* __restrict__ segs,
                               const float* __restrict__ rec32, ChunkBound* out) {
  const int ch = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (ch >= nchunks) return;
  const int lane = threadIdx.x & 31;
  const WorkChunk w = chunks[ch];
  const ClassSeg& sg = segs[w.cls];
  const bool merged = (sg.shape & kMergedBit) != 0;
  const int total = merged ? (sg.shape >> 15) & 31 : (sg.shape & 31) + ((sg.shape >> 5) & 31) + ((sg.shape >> 10) & 31);
  float lo[3], hi[3], smin = HUGE_VALF, smax = 0.0f, la = -HUGE_VALF;
  unsigned quartets = 0;
  for (int d = 0; d < 3; ++d) {
    lo[d] = HUGE_VALF;
    hi[d] = -HUGE_VALF;
  }
  if (lane < w.count) {
    const float* R = rec32 + sg.off32 + (w.rec - sg.first + lane) * sg.stride32;
    smin = smax = R[0];
    la = R[10] + 0.05f;
    quartets = 1;
    if (merged) {
      float sum = 0.0f;
      for (int k = 0; k <= total; ++k) sum += R[12 + 2 * sg.nc + k];
      la += log2f(sum);
      quartets = static_cast<unsigned>(R[9]);
    }
    for (int d = 0; d < 3; ++d) {
      const float x = R[2 + d] / R[0], e = 1e-6f * fabsf(x) + 1e-6f;
      lo[d] = x - e;
      hi[d] = x + e;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    for (int d = 0; d < 3; ++d) {
      lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
    smin = fminf(smin, __shfl_xor_sync(0xffffffffu, smin, o));
    smax = fmaxf(smax, __shfl_xor_sync(0xffffffffu, smax, o));
    la = fmaxf(la, __shfl_xor_sync(0xffffffffu, la, o));
    quartets += __shfl_xor_sync(0xffffffffu, quartets, o);
  }
  if (lane == 0) {
    ChunkBound B;
    for (int d = 0; d < 3; ++d) {
      B.dlo[d] = lo[d];
      B.dhi[d] = hi[d];
    }
    B.smin = smin;
    B.smax = smax;
    B.la = la;
    B.total = static_cast<float>(total);
    B.records = static_cast<uint32_t>(w.count);
    B.quartets = quartets;
    out[ch] = B;
  }
}

// The polynomials of a preparation that went through in one slab (table null: several).
struct BuildTable {
  const double* table;
  const int64_t* sub_off;
  const SubConst* sub;
  const SubSize* off;
  int64_t nsub;
};

// Product records, one thread each: the quartet's values from the polynomial table where it still holds them
// (solving them again took 47 us of a 3 081-quartet list's 240), else restated (identical arithmetic), and its
// records into the class segments:
//   FP64 record [A, sqe, d0, d1, d2, A', Cx.., Cy.., Cz..] (C highest degree first);
//   FP32 record [s_hi, s_lo, b_hi[3], b_lo[3], A'_hi, A'_lo, la, 0, Cn_hi (x,y,z), Cn_lo (x,y,z)]
// with s = sqe c_u, b_d = s d_d, u = s (r + d) = c_u r', the polynomials rewritten in u and
// scaled by kappa_d (largest |coefficient|) so that Cn has max |coefficient| 1, A' = A prod
// kappa_d, and la = log2(|A'| prod_d sum_k |Cn_dk|). hi/lo pairs carry the FP64 value to
// ~2^-48 relative (see mixed_eval.cu).
__global__ void k_build(const __grid_constant__ PrepConst cP, int64_t nrec, const int64_t* __restrict__ rsrc, const int64_t* __restrict__ idx,
                        const int4* __restrict__ ijkl, const double* __restrict__ v,
                        const PrimD* __restrict__ prims, const ClassSeg* __restrict__ segs, int nseg, BuildTable T,
                        double* rec64, float* rec32) {
  const int64_t p = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (p >= nrec) return;
  const ClassSeg sg = segs[segment_of(segs, nseg, p)];
  if (sg.shape & kMergedBit) return;
  const int64_t place = -1 - rsrc[p], src = idx[place];
  QRec rec;
  if (T.table) {
    const int64_t s = subgroup_of(T.sub_off, 0, T.nsub, place);
    const SubConst& c = T.sub[s];
    const int4 q = ijkl[src];
    const PrimD &Pi = prims[q.x - 1], &Pj = prims[q.y - 1], &Pk = prims[q.z - 1], &Pl = prims[q.w - 1];
    rec.A = (dm_value(cP, Pi, Pj, Pk, Pl, v[src]) * c.c1) * c.c2;
    rec.sqe = c.sqe;
    for (int d = 0; d < 3; ++d) {
      const int L = Pi.t[d] + Pj.t[d] + Pk.t[d] + Pl.t[d];
      const int at = d * c.combos() + c.combo(Pi.t[d], Pj.t[d], Pk.t[d], Pl.t[d]);
      const double* C = T.table + T.off[s].tab + static_cast<int64_t>(at) * c.entry() + 1;
      rec.L[d] = L;
      rec.d[d] = c.Pik[d] - c.Pjl[d];
      for (int m = 0; m <= L; ++m) rec.C[d][m] = C[m];
    }
  } else {
    restate(cP, prims, ijkl[src], v[src], &rec);
  }
  const int64_t local = p - sg.first;
  double* r64 = rec64 + sg.off64 + local * sg.stride;
  // u-space polynomials: V_d(r') = sum_k C_k r'^k = sum_k (C_k c^-k) u^k, u = c r'
  double Cu[3][kMaxCoef], kappa[3];
  double Bmax = 1.0;
  for (int d = 0; d < 3; ++d) {
    const int L = rec.L[d];
    double big = 0.0;
    for (int m = 0; m <= L; ++m) {
      const double ck = rec.C[d][m] * ipow(1.0 / cP.c_u, L - m);
      Cu[d][m] = ck;
      big = fmax(big, fabs(ck));
    }
    kappa[d] = big > 0.0 ? big : 1.0;
    Bmax = Bmax * kappa[d];
  }
  // a constant polynomial (L_d = 0) normalises to +-1: fold the sign into A' so the
  // evaluation can skip that dimension (V_d = 1 exactly)
  double sign = 1.0;
  for (int d = 0; d < 3; ++d)
    if (rec.L[d] == 0 && Cu[d][0] < 0.0) {
      sign = -sign;
      Cu[d][0] = -Cu[d][0];
    }
  const double Aprime = sign * rec.A * Bmax;
  r64[0] = rec.A;
  r64[1] = rec.sqe;
  r64[2] = rec.d[0];
  r64[3] = rec.d[1];
  r64[4] = rec.d[2];
  r64[5] = Aprime;
  int o = kRecHeader;
  for (int d = 0; d < 3; ++d)
    for (int m = 0; m <= rec.L[d]; ++m) r64[o++] = rec.C[d][m];
  for (; o < sg.stride; ++o) r64[o] = 0.0;

  float* r32 = rec32 + sg.off32 + local * sg.stride32;
  const double s = rec.sqe * cP.c_u;
  const float s_hi = static_cast<float>(s);
  r32[0] = s_hi;
  r32[1] = static_cast<float>(s - static_cast<double>(s_hi));
  for (int d = 0; d < 3; ++d) {
    const double b = s * rec.d[d];
    const float b_hi = static_cast<float>(b);
    r32[2 + d] = b_hi;
    r32[5 + d] = static_cast<float>(b - static_cast<double>(b_hi));
  }
  // A' = m 2^k with |m| in [0.5, 1): m as an FP32 pair, k applied exactly in the exponent
  // scaling of the evaluation's exp2 (A' itself can exceed the FP32 range for tight d shells)
  int kA = 0;
  const double mA = Aprime != 0.0 ? frexp(Aprime, &kA) : 0.0;
  const float A_hi = static_cast<float>(mA);
  r32[8] = A_hi;
  r32[9] = static_cast<float>(mA - static_cast<double>(A_hi));
  // log2 of |A'| prod_d sum_k |Cn_dk|: the tile bounds of the mixed evaluation start from it
  double la = log2(fabs(Aprime));
  for (int d = 0; d < 3; ++d) {
    double sd = 0.0;
    for (int m = 0; m <= rec.L[d]; ++m) sd += fabs(Cu[d][m] / kappa[d]);
    la += log2(sd);
  }
  r32[10] = static_cast<float>(la);
  r32[11] = static_cast<float>(kA);
  const int nc = rec.L[0] + rec.L[1] + rec.L[2] + 3;
  o = 12;
  for (int d = 0; d < 3; ++d)
    for (int m = 0; m <= rec.L[d]; ++m) {
      const double cn = Cu[d][m] / kappa[d];
      const float hi = static_cast<float>(cn);
      r32[o] = hi;
      r32[o + nc] = static_cast<float>(cn - static_cast<double>(hi));
      ++o;
    }
  for (o += nc; o < sg.stride32; ++o) r32[o] = 0.0f;
}

}  // namespace

// Constants of a preparation (computed on the host with the same expressions as the reference).
static PrepConst prep_constants(const inca_ctx* c, double thresh, int normalize) {
  PrepConst hc;
  std::memset(&hc, 0, sizeof(hc));
  const double pi = 4.0 * std::atan(1.0);
  for (int m = 1; m <= kMaxCoef; ++m)
    hc.wm[m - 1] = (m == 1) ? 1.0 : std::pow(double(m) * 0.5, double(m) * 0.5) * std::exp(-double(m) * 0.5);
  hc.pi15 = pi * std::sqrt(pi);
  hc.thresh = thresh;
  hc.c_u = std::sqrt(1.0 / std::log(2.0));
  hc.cu_inv_pow[0] = 1.0;
  hc.fact[0] = 1.0f;
  for (int k = 1; k <= kMaxTotal; ++k) {
    hc.cu_inv_pow[k] = hc.cu_inv_pow[k - 1] / hc.c_u;
    hc.fact[k] = hc.fact[k - 1] * static_cast<float>(k);
  }
  hc.nprim = c->nprim;
  hc.normalize = normalize ? 1 : 0;
  hc.merge = c->group_keys > 0 ? 1 : 0;
  return hc;
}

// Bytes of each of the two staging buffers that a work chunk may fill: with 16 one-warp CTAs per SM
// the mixed evaluation has 14 KB of shared memory per CTA, 3 KB of it for its tables. (A class whose
// record alone is larger gets chunks of one record.)
constexpr int kStageFloats = 1344;
// Records from which on a class's records are sorted by place: 100 primitives (78 253 records) gain 2 ms of
// 14.6 in the evaluation, 66 (36 236) 0.1 of 1.4 for 40 us of sorting; CH4 (29 129) and 41 primitives
// (7 917) gain nothing for 50 and 20 us.
constexpr int64_t kSortPlaces = 1 << 15;
// Polynomial table entries (doubles) held at a time: groups are taken in slabs of about this many
// (1 GB, and less than 1 MB for the largest group), so the table does not grow with the list.
constexpr int64_t kSlabTable = int64_t(1) << 27;

// One CUDA call or kernel launch after the other until one fails.
#define PREP_TRY(call)                  \
  do {                                  \
    if (e == cudaSuccess) e = (call);   \
  } while (0)
#define PREP_LAUNCH(...)                \
  do {                                  \
    if (e == cudaSuccess) {             \
      INCA_LAUNCH(c, __VA_ARGS__);      \
      e = cudaGetLastError();           \
    }                                   \
  } while (0)

int prepare_device(inca_ctx* c, double thresh, int normalize) {
  if (c->nprim <= 0) return set_error(c, INCA_E_STATE, "inca_prepare: primitives not set");
  if (c->nq <= 0) return set_error(c, INCA_E_STATE, "inca_prepare: no quartets loaded");
  if (!(thresh > 0.0)) return set_error(c, INCA_E_ARG, "inca_prepare: thresh must be > 0");
  int tmax = 0, lmax = 0;  // largest power, largest shell
  for (int p = 0; p < c->nprim; ++p) {
    int sum = 0;
    for (int d = 0; d < 3; ++d) {
      const int t = c->h_tmn[3 * p + d];
      if (t < 0 || t > 4)
        return set_error(c, INCA_E_LIMIT, "inca_prepare: Cartesian power above 4 (g) in primitive " +
                                              std::to_string(p + 1));
      tmax = std::max(tmax, t);
      sum += t;
    }
    lmax = std::max(lmax, sum);
  }
  c->lim = thresh * (1.0 / (double(c->nprim) * (double(c->nprim) + 1.0) * 0.5));
  const PrepConst pc = prep_constants(c, thresh, normalize);

  c->source_kept = false;  // the flags are written next
  const int64_t n = c->nq;
  const bool keep_values = n <= (int64_t(1) << 27);
  if (c->d_flags.reserve(n) != cudaSuccess) return set_error(c, INCA_E_NOMEM, "flags");
  if (keep_values) {
    if (c->d_s1.reserve(n) != cudaSuccess || c->d_s2.reserve(n) != cudaSuccess)
      return set_error(c, INCA_E_NOMEM, "screening values");
  }
  c->have_screen_values = keep_values;
  double* s1 = keep_values ? c->d_s1.p : nullptr;
  double* s2 = keep_values ? c->d_s2.p : nullptr;
  // sort and grouping scratch, owned by the context: kept between calls up to kPrepKeepBytes (a repeated
  // preparation then allocates and frees nothing, and no cudaFree stalls the stream), else given back
  DevBuf<uint64_t>& key = c->d_pkey;
  DevBuf<uint64_t>& key2 = c->d_pkey2;
  DevBuf<int64_t>& idx = c->d_pidx;
  DevBuf<int64_t>& idx2 = c->d_pidx2;
  DevBuf<int64_t>& sub_off = c->d_psub;
  DevBuf<unsigned char>& tmp = c->d_ptmp;
  DevBuf<unsigned char>& group = c->d_pgroup;
  DevBuf<unsigned char>& slab = c->d_pslab;
  DevBuf<unsigned char>& rbuf = c->d_prec;
  DevBuf<unsigned long long>& count = c->d_pcount;
  auto release_all = [&]() {
    key.release(); key2.release(); idx.release(); idx2.release(); sub_off.release(); tmp.release(); group.release();
    slab.release(); rbuf.release(); count.release();
  };
  auto cleanup = [&]() {
    const size_t held = 8 * (key.n + key2.n + idx.n + idx2.n + sub_off.n) + tmp.n + group.n + slab.n + rbuf.n;
    if (held > kPrepKeepBytes) release_all();
  };
  auto no_memory = [&](const char* what) {
    release_all();
    return set_error(c, INCA_E_NOMEM, std::string("inca_prepare: ") + what);
  };
  auto failed = [&](cudaError_t err, const char* what) {
    release_all();
    return cuda_error(c, err, what);
  };
  const int64_t keys = c->group_keys > 0 ? c->group_keys : n;
  const uint64_t fail_key = 4 * static_cast<uint64_t>(keys);
  int key_bits = 1;
  while ((fail_key >> key_bits) != 0) ++key_bits;
  // subgroups: at most one per quartet and one per key
  const int64_t scap = std::min<int64_t>(n, 4 * keys);
  const bool small = n <= kSmallList && key_bits <= 32;  // grouped, and sorted by class, by one block each
  if (key.reserve(n) || key2.reserve(n) || idx.reserve(n) || idx2.reserve(n) || sub_off.reserve(scap) ||
      count.reserve(kNCounts + (small ? 2 * n : 0)))
    return no_memory("sort buffers");
  auto storage = [&](size_t bytes) { return bytes > tmp.n ? tmp.reserve(bytes) : cudaSuccess; };
  // read back through pinned memory: the counters, and the first kPinClasses (kPinSmall) classes with them
  constexpr int64_t kPinClasses = 2048, kPinSmall = 256;
  constexpr size_t kPinBytes = 512 + 12 * kPinClasses;
  static_assert(8 * (kNCounts + 2 * kPinSmall) <= kPinBytes, "classes of a small list behind the counters");
  if (!c->h_pin && cudaMallocHost(reinterpret_cast<void**>(&c->h_pin), kPinBytes) != cudaSuccess)
    return no_memory("pinned memory");
  unsigned long long* hc = reinterpret_cast<unsigned long long*>(c->h_pin);
  static_assert(kNCounts * sizeof(unsigned long long) <= 512, "counters fit their part of the pinned buffer");
  int64_t* hcount = reinterpret_cast<int64_t*>(c->h_pin + 512);
  uint32_t* hkey = reinterpret_cast<uint32_t*>(hcount + kPinClasses);
  auto read_counts = [&](int64_t more = 0) {
    cudaError_t err = cudaMemcpyAsync(hc, count.p, (kNCounts + more) * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                      c->stream);
    return err != cudaSuccess ? err : cudaStreamSynchronize(c->stream);
  };
  auto device_count = [&](PrepCount k) { return reinterpret_cast<int64_t*>(count.p + k); };
  auto blocks = [](int64_t items, int per) { return static_cast<unsigned>((items + per - 1) / per); };
  cudaError_t e = cudaMemsetAsync(count.p, 0, kNCounts * sizeof(unsigned long long), c->stream);
  // JA8 of every primitive pair, once (up to kPairTableMax primitives: 128 MiB); beyond that each
  // quartet evaluates its two JA8 bounds itself
  const double* jtab = nullptr;
  if (e == cudaSuccess && c->nprim <= kPairTableMax) {
    const int64_t np2 = static_cast<int64_t>(c->nprim) * c->nprim;
    if (c->d_ja8.reserve(np2) == cudaSuccess) {
      PREP_LAUNCH(k_pair_ja8, blocks(np2, 128), 128, 0, pc, c->nprim, c->d_prims.p, c->d_ja8.p);
      jtab = c->d_ja8.p;
    }
  }
  PREP_LAUNCH(k_screen1, blocks(n, 256), 256, 0, pc, n, c->d_ijkl.p, c->d_v.p, c->d_prims.p, c->d_flags.p, s1, s2, key.p,
              idx.p, fail_key, count.p, jtab);
  // what the groups need, by subgroups (nsub of them at most)
  constexpr int64_t kMaxSlabs = 4096;
  size_t off = 0;
  auto carve = [&](size_t bytes) {
    const size_t at = off;
    off += (bytes + 255) & ~size_t(255);
    return at;
  };
  GroupRec* grp = nullptr;
  SubPowers* powers = nullptr;
  SubSize *size = nullptr, *sub_at = nullptr;
  int64_t *grp_sub = nullptr, *gcount = nullptr, *gstart = nullptr, *bound = nullptr;
  SmallScratch sx{};
  auto group_arrays = [&](int64_t nsub) {
    const size_t o_grp = carve(sizeof(GroupRec) * nsub), o_pow = carve(sizeof(SubPowers) * nsub);
    const size_t o_at = carve(sizeof(SubSize) * nsub), o_size = carve(sizeof(SubSize) * nsub);
    const size_t o_i64 = carve(8 * (nsub + kMaxSlabs));
    const size_t o_sums = carve(small ? 8 * nsub : 0), o_u32 = carve(small ? 4 * (4 * nsub + n) : 0);
    if (group.reserve(off)) return false;
    grp = reinterpret_cast<GroupRec*>(group.p + o_grp);
    powers = reinterpret_cast<SubPowers*>(group.p + o_pow);
    sub_at = reinterpret_cast<SubSize*>(group.p + o_at);
    size = reinterpret_cast<SubSize*>(group.p + o_size);
    static_assert(sizeof(SubSize) == 2 * sizeof(int64_t), "the groups' counts and places take the sizes' room");
    gcount = reinterpret_cast<int64_t*>(size);  // (the sizes are done with once they are added up)
    gstart = gcount + nsub;
    grp_sub = reinterpret_cast<int64_t*>(group.p + o_i64);
    bound = grp_sub + nsub;
    sx.sums = reinterpret_cast<unsigned long long*>(group.p + o_sums);
    sx.pows = reinterpret_cast<uint32_t*>(group.p + o_u32);
    sx.sub_key = sx.pows + nsub;
    sx.sub_grp = reinterpret_cast<int*>(sx.sub_key + nsub);
    sx.total = sx.sub_grp + nsub;
    sx.place_sub = sx.total + nsub;
    return true;
  };
  // the quartets that passed, by subgroup (stable: input order within it)
  size_t tb = 0;
  const thrust::counting_iterator<int64_t> places(0);
  if (small) {
    if (!group_arrays(scap)) return no_memory("groups");
    PREP_LAUNCH(k_small_groups, 1, kSmallThreads, 0, static_cast<int>(n), key_bits, key.p,
                static_cast<uint32_t>(fail_key), c->d_ijkl.p, c->d_prims.p, idx2.p, sub_off.p, powers, sub_at, grp_sub, sx,
                count.p);
  } else {
    PREP_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, key.p, key2.p, idx.p, idx2.p, n, 0, key_bits, c->stream));
    PREP_TRY(storage(tb));
    PREP_TRY(cub::DeviceRadixSort::SortPairs(tmp.p, tb, key.p, key2.p, idx.p, idx2.p, n, 0, key_bits, c->stream));
    const SubHead sub_head{key2.p, fail_key};
    PREP_TRY(cub::DeviceSelect::If(nullptr, tb, places, sub_off.p, device_count(kNSub), n, sub_head, c->stream));
    PREP_TRY(storage(tb));
    PREP_TRY(cub::DeviceSelect::If(tmp.p, tb, places, sub_off.p, device_count(kNSub), n, sub_head, c->stream));
  }
  PREP_TRY(read_counts());
  if (e != cudaSuccess) return failed(e, "inca_prepare (screening)");
  if (hc[kNBad]) {
    cleanup();
    return set_error(c, INCA_E_ARG, "inca_prepare: quartet index outside 1..nprim");
  }
  const int64_t npass = static_cast<int64_t>(hc[kNScreen1]), nsub = static_cast<int64_t>(hc[kNSub]);
  // the unsorted keys and indices are done with
  double* amp = reinterpret_cast<double*>(key.p);
  QuartetDesc* desc = reinterpret_cast<QuartetDesc*>(idx.p);

  // sizes of the subgroups, then the groups, slab by slab
  double* coef = nullptr;
  BuildTable built{};
  int64_t nrec = 0;
  const int w = [&]() {
    int bits = 1;
    while ((std::max(4 * tmax, std::min(4 * lmax, kMaxTotal)) >> bits) != 0) ++bits;
    return bits;
  }();
  int cls_bits = 4 * w + 1;
  for (int m = std::max(c->batch_molecules, 1) - 1; m > 0; m >>= 1) ++cls_bits;
  if (nsub > 0) {
    if (!small) {
      if (!group_arrays(nsub)) return no_memory("groups");
      const int team = npass <= 8 * nsub ? 8 : 32;
      const auto sub_sizes = team == 8 ? k_sub<8> : k_sub<32>;
      PREP_LAUNCH(sub_sizes, blocks(nsub, 256 / team), 256, 0, nsub, sub_off.p, npass, key2.p, idx2.p, c->d_ijkl.p,
                  c->d_prims.p, powers, size, count.p);
      const auto places_of = [&](size_t& bytes, void* t) {
        return cub::DeviceScan::ExclusiveScan(t, bytes, size, sub_at, cuda::std::plus<>(), SubSize{0, 0}, nsub, c->stream);
      };
      PREP_TRY(places_of(tb, nullptr));
      PREP_TRY(storage(tb));
      PREP_TRY(places_of(tb, tmp.p));
      const GroupHead group_head{key2.p, sub_off.p};
      PREP_TRY(cub::DeviceSelect::If(nullptr, tb, places, grp_sub, device_count(kNGroup), nsub, group_head, c->stream));
      PREP_TRY(storage(tb));
      PREP_TRY(cub::DeviceSelect::If(tmp.p, tb, places, grp_sub, device_count(kNGroup), nsub, group_head, c->stream));
      PREP_TRY(read_counts());
      if (e != cudaSuccess) return failed(e, "inca_prepare (groups)");
    }
    const int64_t ngroup = static_cast<int64_t>(hc[kNGroup]);
    const int64_t ntable = static_cast<int64_t>(hc[kNTable]), nentry = static_cast<int64_t>(hc[kNEntry]);
    const int64_t nslab = std::min(kMaxSlabs / 5 - 1, (ntable + kSlabTable - 1) / kSlabTable);
    // slab k: groups hb[5k] to hb[5k + 5], subgroups hb[5k + 1], quartets, entries and table from there on
    std::vector<int64_t> hb{0, 0, 0, 0, 0, ngroup, nsub, npass, nentry, ntable};
    if (nslab > 1) {
      hb.assign(5 * (nslab + 1), 0);
      PREP_LAUNCH(k_slabs, 1, 1024, 0, static_cast<int>(nslab), ngroup, nsub, npass, nentry, ntable, grp_sub, sub_off.p,
                  sub_at, bound);
      PREP_TRY(cudaMemcpyAsync(hb.data(), bound, sizeof(int64_t) * hb.size(), cudaMemcpyDeviceToHost, c->stream));
      PREP_TRY(cudaStreamSynchronize(c->stream));
      if (e != cudaSuccess) return failed(e, "inca_prepare (slabs)");
    }
    int64_t max_grp = 0, max_sub = 0, max_ent = 0, max_tab = 0;
    for (size_t k = 5; k < hb.size(); k += 5) {
      max_grp = std::max(max_grp, hb[k] - hb[k - 5]);
      max_sub = std::max(max_sub, hb[k + 1] - hb[k - 4]);
      max_ent = std::max(max_ent, hb[k + 3] - hb[k - 2]);
      max_tab = std::max(max_tab, hb[k + 4] - hb[k - 1]);
    }
    off = 0;
    const size_t o_coef = carve(sizeof(double) * hc[kNCoef]), o_tab = carve(sizeof(double) * max_tab);
    const size_t o_task = carve(sizeof(PolyTask) * max_ent), o_next = carve(sizeof(unsigned) * kMaxCoef);
    const size_t o_mark = carve(max_ent), o_sub = carve(sizeof(SubConst) * max_sub);
    const size_t o_list = carve(8 * max_grp), o_large = carve(8 * max_grp);
    if (slab.reserve(off)) return no_memory("polynomial table");
    coef = reinterpret_cast<double*>(slab.p + o_coef);
    double* table = reinterpret_cast<double*>(slab.p + o_tab);
    PolyTask* task = reinterpret_cast<PolyTask*>(slab.p + o_task);
    unsigned* next = reinterpret_cast<unsigned*>(slab.p + o_next);
    uint8_t* mark = slab.p + o_mark;
    int64_t *list = reinterpret_cast<int64_t*>(slab.p + o_list), *large = reinterpret_cast<int64_t*>(slab.p + o_large);
    const int total_max = std::min(4 * lmax, kMaxTotal);
    const int nc_max = merged_coefs(total_max), D = total_max + 1;
    constexpr int kTinySmem = static_cast<int>(sizeof(double)) * kGroupThreads * 3 * kTinyD;
    const int smem = std::max(kGroupThreads / 32 * group_smem(nc_max, D), kTinySmem);
    if (smem > 48 * 1024)  // f and g shells
      PREP_TRY(cudaFuncSetAttribute(k_groups, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    for (size_t k = 0; k + 5 < hb.size(); k += 5) {
      const int64_t g0 = hb[k], sb0 = hb[k + 1], p0 = hb[k + 2], e0 = hb[k + 3], t0 = hb[k + 4];
      const int64_t g1 = hb[k + 5], sb1 = hb[k + 6], p1 = hb[k + 7], ne = hb[k + 8] - e0;
      if (g1 == g0) continue;
      SubConst* sub = reinterpret_cast<SubConst*>(slab.p + o_sub) - sb0;  // of the slab's subgroups, by their numbers
      PREP_LAUNCH(k_sub_const, blocks(sb1 - sb0, 128), 128, 0, pc, sb0, sb1, nsub, npass, sub_off.p, idx2.p, c->d_ijkl.p,
                  c->d_prims.p, powers, sub);
      // the counters from kNSmall on are the slab's (and zero before the first)
      if (k > 0)
        PREP_TRY(cudaMemsetAsync(count.p + kNSmall, 0, sizeof(unsigned long long) * (kNCounts - kNSmall), c->stream));
      // next and mark: one after the other
      PREP_TRY(cudaMemsetAsync(next, 0, static_cast<size_t>(mark + ne - reinterpret_cast<uint8_t*>(next)), c->stream));
      PREP_LAUNCH(k_mark, blocks(p1 - p0, 256), 256, 0, pc, sb0, sb1, p0, p1, sub_off.p, idx2.p, c->d_ijkl.p, c->d_v.p,
                  c->d_prims.p, sub, sub_at, e0, t0, desc, amp, mark, table, count.p);
      const GroupArgs ga{grp_sub, sub_off.p, nsub, npass, ngroup, sub, sub_at, t0, table, idx2.p, desc, amp,
                         c->d_flags.p, s2, D, nc_max, group_smem(nc_max, D), coef, grp, gcount, list, large, g1 - g0, count.p};
      const int team = ne <= 4 * (sb1 - sb0) ? 4 : 16;
      const unsigned poly_blocks = tmax > 0 ? blocks(sb1 - sb0, kListThreads / team) : 0;
      PREP_LAUNCH(k_list, poly_blocks + blocks(g1 - g0, kListThreads), kListThreads, 0, poly_blocks, team, sb0, sb1, g0, g1,
                  e0, mark, next, task, ga);
      const auto poly = tmax <= 1 ? k_poly<1> : tmax == 2 ? k_poly<2> : k_poly<4>;
      if (tmax > 0) PREP_LAUNCH(poly, blocks(ne, 128), 128, 0, pc, task, count.p, sb0, sub, sub_at, t0, table);
      if (nslab == 1) built = BuildTable{table, sub_off.p, sub, sub_at, nsub};
      PREP_LAUNCH(k_groups, static_cast<unsigned>(std::min<int64_t>(g1 - g0, 8 * c->num_sms)), kGroupThreads, smem, pc, ga);
    }
    if (small) {
      if (rbuf.reserve(20 * static_cast<size_t>(npass))) return no_memory("record keys");
      PREP_LAUNCH(k_small_records, 1, kSmallThreads, 0, static_cast<int>(npass), cls_bits, grp, gcount,
                  c->d_flags.p, idx2.p, c->d_ijkl.p, c->d_prims.p, w, sx, key.p, reinterpret_cast<int64_t*>(rbuf.p),
                  count.p);
    } else {
      PREP_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, gcount, gstart, ngroup, c->stream));
      PREP_TRY(storage(tb));
      PREP_TRY(cub::DeviceScan::ExclusiveSum(tmp.p, tb, gcount, gstart, ngroup, c->stream));
    }
    PREP_TRY(read_counts(small ? 2 * std::min(npass, kPinSmall) : 0));
    if (e != cudaSuccess) return failed(e, "inca_prepare (groups)");
    nrec = static_cast<int64_t>(hc[kNRec]);
  }
  const int64_t nsurv = static_cast<int64_t>(hc[kNSurv]), ngroup = static_cast<int64_t>(hc[kNGroup]);
  const bool products = hc[kNProduct] > 0;

  // records by class: sources (two arrays), class keys (two) and the classes' keys and counts
  int64_t *rsrc = nullptr, *rsrc2 = nullptr;
  std::vector<uint32_t> hk;
  std::vector<int64_t> hcnt;
  if (nrec > 0 && small) {
    rsrc2 = reinterpret_cast<int64_t*>(rbuf.p);
    const int64_t nclass = static_cast<int64_t>(hc[kNClass]);
    std::vector<unsigned long long> cls(hc + kNCounts, hc + kNCounts + 2 * std::min(nclass, kPinSmall));
    if (nclass > kPinSmall) {
      cls.resize(2 * nclass);
      PREP_TRY(cudaMemcpyAsync(cls.data(), count.p + kNCounts, 16 * nclass, cudaMemcpyDeviceToHost, c->stream));
      PREP_TRY(cudaStreamSynchronize(c->stream));
      if (e != cudaSuccess) return failed(e, "inca_prepare (classes)");
    }
    for (int64_t r = 0; r < nclass; ++r) {
      hk.push_back(static_cast<uint32_t>(cls[2 * r]));
      hcnt.push_back(static_cast<int64_t>(cls[2 * r + 1]));
    }
  } else if (nrec > 0) {
    // (as many as quartets at most: the sorted list's keys, its descriptors and amplitudes are done with)
    if (rbuf.reserve(20 * static_cast<size_t>(nrec))) return no_memory("record keys");
    uint64_t *rkey = key.p, *rkey2 = key2.p;
    rsrc = idx.p;
    rsrc2 = reinterpret_cast<int64_t*>(rbuf.p);
    int64_t* ucount = rsrc2 + nrec;
    uint32_t* ukey = reinterpret_cast<uint32_t*>(ucount + nrec);
    // small lists keep their group order within a class: their few chunks are nearly all live everywhere
    const int place_bits = nrec >= kSortPlaces ? kPlaceBits : 0;
    cls_bits += place_bits;
    PREP_LAUNCH(k_record_keys, blocks(ngroup, 128), 128, 0, pc, ngroup, count.p, grp_sub, nsub, sub_off.p, npass, grp, gcount,
                gstart, c->d_flags.p, idx2.p, c->d_ijkl.p, c->d_prims.p, w, place_bits, rkey, rsrc);
    PREP_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, rkey, rkey2, rsrc, rsrc2, nrec, 0, cls_bits, c->stream));
    PREP_TRY(storage(tb));
    PREP_TRY(cub::DeviceRadixSort::SortPairs(tmp.p, tb, rkey, rkey2, rsrc, rsrc2, nrec, 0, cls_bits, c->stream));
    const auto classes = thrust::make_transform_iterator(rkey2, ClassOfKey{place_bits});
    PREP_TRY(cub::DeviceRunLengthEncode::Encode(nullptr, tb, classes, ukey, ucount, device_count(kNClass), nrec,
                                                c->stream));
    PREP_TRY(storage(tb));
    PREP_TRY(cub::DeviceRunLengthEncode::Encode(tmp.p, tb, classes, ukey, ucount, device_count(kNClass), nrec,
                                                c->stream));
    const int64_t pin = std::min(kPinClasses, nrec);
    PREP_TRY(cudaMemcpyAsync(hkey, ukey, sizeof(uint32_t) * pin, cudaMemcpyDeviceToHost, c->stream));
    PREP_TRY(cudaMemcpyAsync(hcount, ucount, sizeof(int64_t) * pin, cudaMemcpyDeviceToHost, c->stream));
    PREP_TRY(read_counts());
    if (e != cudaSuccess) return failed(e, "inca_prepare (classes)");
    const int64_t nclass = static_cast<int64_t>(hc[kNClass]);
    hk.assign(hkey, hkey + std::min(nclass, pin));
    hcnt.assign(hcount, hcount + std::min(nclass, pin));
    if (nclass > pin) {
      hk.resize(nclass);
      hcnt.resize(nclass);
      PREP_TRY(cudaMemcpyAsync(hk.data(), ukey, sizeof(uint32_t) * nclass, cudaMemcpyDeviceToHost, c->stream));
      PREP_TRY(cudaMemcpyAsync(hcnt.data(), ucount, sizeof(int64_t) * nclass, cudaMemcpyDeviceToHost, c->stream));
      PREP_TRY(cudaStreamSynchronize(c->stream));
    }
    if (e != cudaSuccess) return failed(e, "inca_prepare (classes)");
  }
  // class segments (the old records go here: until then a failed call leaves them to the evaluation)
  c->prepared = false;
  c->classes.clear();
  int64_t first = 0, off64 = 0, off32 = 0;
  for (size_t r = 0; r < hk.size(); ++r) {
    ClassSeg s;
    const uint32_t mask = (1u << w) - 1u;
    const bool merged = (hk[r] >> (4 * w)) & 1u;
    s.mol = static_cast<int>(hk[r] >> (4 * w + 1));
    s.shape = merged ? merged_shape(hk[r] & mask)
                     : product_shape((hk[r] >> (3 * w)) & mask, (hk[r] >> (2 * w)) & mask, (hk[r] >> w) & mask);
    s.nc = shape_coefs(s.shape);
    s.stride = (kRecHeader + s.nc + 1) & ~1;
    s.stride32 = (12 + 2 * s.nc + (merged ? ((s.shape >> 15) & 31) + 1 : 0) + 3) & ~3;
    s.per_chunk = std::max(1, std::min(32, kStageFloats / s.stride32));
    s.first = first;
    s.count = hcnt[r];
    s.off64 = off64;
    s.off32 = off32;
    off64 += s.count * s.stride;
    off32 += s.count * s.stride32;
    first += s.count;
    c->classes.push_back(s);
  }
  c->nsurv = nsurv;
  c->nrec = nrec;
  // work chunks within a class; each molecule's chunks are contiguous
  c->chunks.clear();
  const int nmol = std::max(c->batch_molecules, 1);
  c->mol_chunks.assign(nmol, ChunkRange{0, 0});
  c->mol_recs.assign(nmol, 0);
  std::vector<bool> seen(nmol, false);
  for (int s = 0; s < static_cast<int>(c->classes.size()); ++s) {
    const ClassSeg& sg = c->classes[s];
    if (sg.mol < 0 || sg.mol >= nmol) {
      cleanup();
      return set_error(c, INCA_E_STATE, "inca_prepare: molecule index outside the batch");
    }
    if (!seen[sg.mol]) {
      seen[sg.mol] = true;
      c->mol_chunks[sg.mol].begin = static_cast<int>(c->chunks.size());
    }
    c->mol_recs[sg.mol] += sg.count;
    for (int64_t f = 0; f < sg.count; f += sg.per_chunk) {
      WorkChunk wc;
      wc.cls = s;
      wc.count = static_cast<int>(std::min<int64_t>(sg.per_chunk, sg.count - f));
      wc.rec = sg.first + f;
      c->chunks.push_back(wc);
    }
    c->mol_chunks[sg.mol].end = static_cast<int>(c->chunks.size());
  }
  if (c->d_rec64.reserve(std::max<int64_t>(off64, 2)) || c->d_rec32.reserve(std::max<int64_t>(off32, 4)) ||
      c->d_classes.reserve(std::max<size_t>(c->classes.size(), 1)) ||
      c->d_chunks.reserve(std::max<size_t>(c->chunks.size(), 1)) ||
      c->d_bounds.reserve(std::max<size_t>(c->chunks.size(), 1)))
    return no_memory("survivor records");
  if (nrec > 0) {
    const int nseg = static_cast<int>(c->classes.size());
    // (from the pinned buffer where they fit: what it held has been read, and the call waits before it returns)
    const size_t cls_bytes = sizeof(ClassSeg) * c->classes.size(), chunk_bytes = sizeof(WorkChunk) * c->chunks.size();
    const void *cls_from = c->classes.data(), *chunks_from = c->chunks.data();
    if (cls_bytes + chunk_bytes <= kPinBytes) {
      cls_from = std::memcpy(c->h_pin, cls_from, cls_bytes);
      chunks_from = std::memcpy(c->h_pin + cls_bytes, chunks_from, chunk_bytes);
    }
    PREP_TRY(cudaMemcpyAsync(c->d_classes.p, cls_from, cls_bytes, cudaMemcpyHostToDevice, c->stream));
    PREP_TRY(cudaMemcpyAsync(c->d_chunks.p, chunks_from, chunk_bytes, cudaMemcpyHostToDevice, c->stream));
    PREP_LAUNCH(k_write, blocks(nrec, 32), 256, 0, pc, nrec, rsrc2, grp, coef, c->d_classes.p, nseg, c->d_rec64.p,
                c->d_rec32.p);
    if (products)
      PREP_LAUNCH(k_build, blocks(nrec, 128), 128, 0, pc, nrec, rsrc2, idx2.p, c->d_ijkl.p, c->d_v.p, c->d_prims.p,
                  c->d_classes.p, nseg, built, c->d_rec64.p, c->d_rec32.p);
    PREP_LAUNCH(k_chunk_bounds, blocks(static_cast<int64_t>(c->chunks.size()), 8), 256, 0,
                static_cast<int>(c->chunks.size()), c->d_chunks.p, c->d_classes.p, c->d_rec32.p, c->d_bounds.p);
  }
  PREP_TRY(cudaStreamSynchronize(c->stream));
  if (e != cudaSuccess) return failed(e, "inca_prepare (records)");
  cleanup();
  c->counts.read = n;
  c->counts.after_screen1 = npass;
  c->counts.after_screen2 = nsurv;
  c->prep_thresh = thresh;
  c->prep_normalize = normalize;
  c->prepared = c->source_kept = true;
  ++c->prepare_count;
  c->evaluated = false;
  return INCA_OK;
}
#undef PREP_TRY
#undef PREP_LAUNCH

// ---------------------------------------------------------------- survivor records, one per quartet
namespace {
// ncoef: coefficients a dimension of the list (the degrees of its basis), zeros above a record's own
__global__ void k_records(const __grid_constant__ PrepConst cP, int64_t n, int ncoef, const int64_t* __restrict__ idx, const int4* __restrict__ ijkl,
                          const double* __restrict__ v, const PrimD* __restrict__ prims, double* A, double* sqe,
                          double* d, int32_t* L, double* C) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  QRec rec;
  restate(cP, prims, ijkl[idx[i]], v[idx[i]], &rec);
  A[i] = rec.A;
  sqe[i] = rec.sqe;
  for (int x = 0; x < 3; ++x) {
    d[3 * i + x] = rec.d[x];
    L[3 * i + x] = rec.L[x];
    for (int m = 0; m < ncoef; ++m) C[(3 * i + x) * ncoef + m] = m <= rec.L[x] ? rec.C[x][m] : 0.0;
  }
}
}  // namespace

// The evaluation keeps merged records only, so the quartets' own records (inca_get_records) are
// restated from the input, with the arithmetic of the screening, in input order. A part at a time (kRecordPart
// survivors of kRecordBlock quartets, so the workspace does not grow with the list) goes to a buffer with only
// the coefficients that the basis can have; host threads write it out to the caller's rows of 17 (a copy of the
// full rows took twice as long: most of it the first touch of the caller's pages).
constexpr int64_t kRecordBlock = int64_t(1) << 20, kRecordPart = int64_t(1) << 15;
int get_records_device(inca_ctx* c, double* A, double* sqe, double* d, int32_t* L, double* C) {
  if (c->nsurv == 0) return INCA_OK;
  const int64_t block = std::min(c->nq, kRecordBlock), part = std::min(block, kRecordPart);
  int tmax = 0;
  for (int t : c->h_tmn) tmax = std::max(tmax, t);
  const int ncoef = std::min(4 * tmax + 1, kMaxCoef);
  const int64_t per = 5 + 3 * ncoef;  // doubles a record
  DevBuf<int64_t> idx, nsel;
  DevBuf<unsigned char> tmp;
  DevBuf<double> val;
  DevBuf<int32_t> deg;
  struct Guard {
    DevBuf<int64_t>&a, &b;
    DevBuf<unsigned char>& t;
    DevBuf<double>& v;
    DevBuf<int32_t>& l;
    ~Guard() { a.release(); b.release(); t.release(); v.release(); l.release(); }
  } guard{idx, nsel, tmp, val, deg};
  size_t tb = 0;
  const PrepConst pc = prep_constants(c, c->prep_thresh, c->prep_normalize);
  auto survivors_of = [&](int64_t first, int64_t n) {  // (tmp null: only the size of its storage)
    const thrust::counting_iterator<int64_t> places(first);
    return cub::DeviceSelect::If(tmp.p, tb, places, idx.p, nsel.p, n, Survivor{c->d_flags.p}, c->stream);
  };
  INCA_CUDA(c, survivors_of(0, block));
  if (idx.reserve(block) || nsel.reserve(1) || tmp.reserve(std::max<size_t>(tb, 1)) || val.reserve(part * per) ||
      deg.reserve(3 * part))
    return set_error(c, INCA_E_NOMEM, "inca_get_records");
  std::vector<double> host(part * per);
  int64_t o = 0;  // survivors written
  for (int64_t first = 0; first < c->nq; first += block) {
    int64_t found = 0;
    INCA_CUDA(c, survivors_of(first, std::min(block, c->nq - first)));
    INCA_CUDA(c, cudaMemcpyAsync(&found, nsel.p, sizeof(found), cudaMemcpyDeviceToHost, c->stream));
    INCA_CUDA(c, cudaStreamSynchronize(c->stream));
    if (found > c->nsurv - o) return set_error(c, INCA_E_STATE, "inca_get_records: more records than inca_prepare counted");
    for (int64_t from = 0; from < found; from += part) {
      const int64_t k = std::min(part, found - from);
      double *vA = val.p, *vs = vA + k, *vd = vs + k, *vC = vd + 3 * k;
      INCA_LAUNCH(c, k_records, static_cast<unsigned>((k + 127) / 128), 128, 0, pc, k, ncoef, idx.p + from, c->d_ijkl.p,
                  c->d_v.p, c->d_prims.p, vA, vs, vd, deg.p, vC);
      INCA_CUDA(c, cudaGetLastError());
      INCA_CUDA(c, cudaMemcpyAsync(host.data(), val.p, sizeof(double) * k * per, cudaMemcpyDeviceToHost, c->stream));
      if (L) INCA_CUDA(c, cudaMemcpyAsync(L + 3 * o, deg.p, sizeof(int32_t) * 3 * k, cudaMemcpyDeviceToHost, c->stream));
      INCA_CUDA(c, cudaStreamSynchronize(c->stream));
      const double *hs = host.data() + k, *hd = hs + k, *hC = hd + 3 * k;
      if (A) std::copy_n(host.data(), k, A + o);
      if (sqe) std::copy_n(hs, k, sqe + o);
      if (d) std::copy_n(hd, 3 * k, d + 3 * o);
      auto rows = [&](int64_t r0, int64_t r1) {
        for (int64_t r = r0; r < r1; ++r) {
          double* to = C + (3 * o + r) * kMaxCoef;
          std::copy_n(hC + r * ncoef, ncoef, to);
          std::fill(to + ncoef, to + kMaxCoef, 0.0);
        }
      };
      if (C) {
        constexpr int kThreads = 8;
        std::vector<std::thread> team;
        int64_t done = 0;  // rows given to a thread
        try {
          for (int t = 0; t + 1 < kThreads && k > 4096; ++t) {
            const int64_t to = 3 * k * (t + 1) / kThreads;
            team.emplace_back(rows, done, to);
            done = to;
          }
        } catch (const std::exception&) {  // no more threads: the rest here
        }
        rows(done, 3 * k);
        for (std::thread& t : team) t.join();
      }
      o += k;
    }
  }
  return INCA_OK;
}

// ---------------------------------------------------------------- closed-shell DM2 records
namespace {
// Record r of the folded list: pairs (i<=k) enumerated as p = index in the packed upper
// triangle; record = (pair_a, pair_b) for all pair_a, pair_b (unique: pair_a <= pair_b).
__device__ __forceinline__ void unpack_pair(int64_t p, int n, int* i, int* k) {
  // pairs ordered (0,0),(0,1)..(0,n-1),(1,1),...: row i has n-i entries
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    const int64_t start = static_cast<int64_t>(mid) * n - static_cast<int64_t>(mid) * (mid - 1) / 2;
    if (start <= p) lo = mid; else hi = mid - 1;
  }
  const int64_t start = static_cast<int64_t>(lo) * n - static_cast<int64_t>(lo) * (lo - 1) / 2;
  *i = lo;
  *k = lo + static_cast<int>(p - start);
}

__device__ __forceinline__ double gam(const double* D, int n, int i, int k, int j, int l) {
  return D[i + static_cast<int64_t>(n) * k] * D[j + static_cast<int64_t>(n) * l] -
         0.5 * D[i + static_cast<int64_t>(n) * l] * D[j + static_cast<int64_t>(n) * k];
}

__global__ void k_closed_shell(int64_t nrec, int n, int64_t npair, int unique, const double* D, int base,
                               int4* ijkl, double* v) {
  const int64_t r = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (r >= nrec) return;
  int64_t pa, pb;
  if (unique) {  // r enumerates pa <= pb in the packed triangle of the pair list
    int a, b;
    unpack_pair(r, static_cast<int>(npair), &a, &b);
    pa = a;
    pb = b;
  } else {
    pa = r / npair;
    pb = r % npair;
  }
  int i, k, j, l;
  unpack_pair(pa, n, &i, &k);
  unpack_pair(pb, n, &j, &l);
  // sum over the distinct orderings (i,k)/(k,i) x (j,l)/(l,j)
  double s = 0.0;
  const int ik[2][2] = {{i, k}, {k, i}}, jl[2][2] = {{j, l}, {l, j}};
  const int nik = (i == k) ? 1 : 2, njl = (j == l) ? 1 : 2;
  for (int a = 0; a < nik; ++a)
    for (int b = 0; b < njl; ++b) s += gam(D, n, ik[a][0], ik[a][1], jl[b][0], jl[b][1]);
  if (unique && pa != pb) s *= 2.0;  // Gamma_{ik,jl} + Gamma_{jl,ik}
  ijkl[r] = make_int4(base + i + 1, base + j + 1, base + k + 1, base + l + 1);
  v[r] = s;
}
}  // namespace

int64_t closed_shell_records(int n, int unique) {
  const int64_t npair = static_cast<int64_t>(n) * (n + 1) / 2;
  return unique ? npair * (npair + 1) / 2 : npair * npair;
}

// Records of one molecule's closed-shell DM2 (n primitives, 1-RDM D) into the context's quartet
// arrays at record offset `at`, with primitive indices offset by `base` (batches).
int gen_closed_shell_into(inca_ctx* c, int n, const double* D, int unique, int base, int64_t at) {
  const int64_t npair = static_cast<int64_t>(n) * (n + 1) / 2;
  const int64_t nrec = closed_shell_records(n, unique);
  DevBuf<double> dD;
  if (dD.reserve(static_cast<size_t>(n) * n)) return set_error(c, INCA_E_NOMEM, "D");
  cudaError_t e = cudaMemcpyAsync(dD.p, D, sizeof(double) * n * n, cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess && nrec > 0) {
    INCA_LAUNCH(c, k_closed_shell, static_cast<unsigned>((nrec + 255) / 256), 256, 0, nrec, n, npair, unique, dD.p,
                base, c->d_ijkl.p + at, c->d_v.p + at);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  dD.release();
  if (e != cudaSuccess) return cuda_error(c, e, "closed-shell DM2");
  return INCA_OK;
}

int gen_closed_shell_device(inca_ctx* c, const double* D, int unique, int64_t* nrec_out) {
  if (c->nprim <= 0) return set_error(c, INCA_E_STATE, "primitives not set");
  if (!D) return set_error(c, INCA_E_ARG, "D is null");
  const int n = c->nprim;
  const int64_t nrec = closed_shell_records(n, unique);
  c->source_kept = false;
  c->nq = 0;
  if (c->d_ijkl.reserve(nrec) || c->d_v.reserve(nrec)) return set_error(c, INCA_E_NOMEM, "quartet records");
  const int st = gen_closed_shell_into(c, n, D, unique, 0, 0);
  if (st) return st;
  c->nq = nrec;
  c->prepared = false;
  c->evaluated = false;
  if (nrec_out) *nrec_out = nrec;
  return INCA_OK;
}

}  // namespace inca
