// K1: per-quartet screening and set-up on the device (FP64).
//
// Restates the per-quartet part of calculate_intracule (src/mod_intracule.f90:282-343) and
// its helpers JA8 / polycoef / gauherm (src/mod_intrastuff.f90:32-341): normalisation,
// screen 1 |v| sqrt(J_ik J_jl) >= lim, Gaussian products, the three per-dimension
// polynomials (Gauss-Hermite right-hand side, Vandermonde system solved by LU with partial
// pivoting, zeroed on a singular matrix or |C| > 1e3) and screen 2 |A Ux Uy Uz| >= lim.
//
// One thread per quartet. The arithmetic is spelled out operation by operation (integer
// powers by repeated multiplication, half-integer powers through sqrt, a Cody-Waite/Taylor
// exponential) and this translation unit is compiled with -fmad=false, so every screening
// value is bit-identical to the CPU oracle's and the screening decisions are identical.
//
// The survivors are then merged. Quartets whose four primitives lie in the same shells (same
// exponent and centre) have the same Gaussian exp(-sqe^2 |r + d|^2), so their sum is that Gaussian
// times one trivariate polynomial: a group of the p components of four shells is one record with at
// most 35 coefficients instead of 81 products, each with an exponential of its own (CH4: 5.2
// quartets per record; molecules with d shells: 9 to 14). The survivors are sorted by group (stable
// radix sort), each group's polynomial is summed in FP64 in input order (k_merge, a warp per
// record), and the records are sorted by the shape of their polynomial and written as
// class-segmented FP64 records (the FP64 evaluation) and FP32 records (the mixed evaluation).
// A group keeps one product record per quartet where that is cheaper to evaluate (a few quartets of
// incomplete shells with high powers) or its total degree exceeds kMaxTotal.
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "hermite_table.h"
#include "inca_internal.h"

namespace inca {
namespace {


struct PrepConst {
  double wm[kMaxCoef];
  double gh_node[kMaxGH + 1][kMaxGH];
  double gh_w[kMaxGH + 1][kMaxGH];
  double pi15;
  double thresh;
  double c_u;  // sqrt(1/ln 2): u = c_u r' turns e^(-r'^2) into 2^(-u^2)
  int nprim;
  int normalize;
};
__constant__ PrepConst cP;

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

__device__ __forceinline__ double xmax(int n) { return cP.gh_node[n][n - 1]; }

// JA8 (src/mod_intrastuff.f90:32-123).
__device__ double ja8(const PrimD& a, const PrimD& b, double R2, double aik, double eik) {
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
__device__ void polycoef(const double R[4], double Pik, double Pjl, double Pijkl, const int t[4],
                         double sqe, double invz, double alf, double* C) {
  const int L = t[0] + t[1] + t[2] + t[3];
  const int np = L + 1;
  const int nn = L / 2 + 1;
  if (np == 1) {
    C[0] = cP.gh_w[1][0];
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
      const double zr = invz * cP.gh_node[nn][h];
      double W = ipow((zr + am) + (Pijkl - R[0]), t[0]) * ipow((zr + ap) + (Pijkl - R[1]), t[1]);
      W = W * ipow((zr + am) + (Pijkl - R[2]), t[2]);
      W = W * ipow((zr + ap) + (Pijkl - R[3]), t[3]);
      rhs = rhs + cP.gh_w[nn][h] * W;
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

struct QRec {
  double A, sqe, d[3];
  int L[3];
  double C[3][kMaxCoef];
};

// JA8 of every ordered primitive pair (i, k), with the arithmetic of prepare_one (Rik2, aik,
// eik), so a quartet's screen-1 value reads two table entries instead of evaluating JA8 twice
// and the values are the same bits.
__global__ void k_pair_ja8(int nprim, const PrimD* __restrict__ prims, double* __restrict__ J) {
  const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (t >= static_cast<int64_t>(nprim) * nprim) return;
  const PrimD Pi = prims[t / nprim], Pk = prims[t % nprim];
  const double aik = Pi.alpha + Pk.alpha;
  const double eik = (Pi.alpha * Pk.alpha) * (1.0 / aik);
  const double Xi[3] = {Pi.x, Pi.y, Pi.z}, Xk[3] = {Pk.x, Pk.y, Pk.z};
  double Rik2 = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) Rik2 = Rik2 + (Xi[d] - Xk[d]) * (Xi[d] - Xk[d]);
  J[t] = ja8(Pi, Pk, Rik2, aik, eik);
}

constexpr int kPairTableMax = 4096;
// inca_prepare keeps its sort scratch (about 32 B per quartet plus the radix sort's temporary
// storage) in the context for lists of up to 2^26 quartets (about 1.6 GB)
constexpr int64_t kPrepKeepQuartets = int64_t(1) << 26;
// Up to this many quartets the screening kernel keeps each survivor's quartet (QRec, 272 B: at
// most 272 MiB) for the record build, which then reads it instead of repeating the FP64
// normalisation, Gaussian products and Vandermonde solves (same values, so the same bits);
// larger lists rebuild each survivor from its indices.
constexpr int64_t kQRecCacheQuartets = int64_t(1) << 20;

// One quartet (src/mod_intracule.f90:282-343). Returns 0 / 1 (screen 1) / 3 (both).
// Jtab (optional): the JA8 table of k_pair_ja8.
__device__ int prepare_one(const PrimD* prims, int4 q, double v, QRec* out, double* s1o,
                           double* s2o, const double* __restrict__ Jtab = nullptr) {
  const PrimD Pi = prims[q.x - 1], Pj = prims[q.y - 1], Pk = prims[q.z - 1], Pl = prims[q.w - 1];
  double DMval = v;
  if (cP.normalize) DMval = v * (((Pi.norm * Pj.norm) * Pk.norm) * Pl.norm);
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
  const double Jik = Jtab ? Jtab[static_cast<int64_t>(q.x - 1) * cP.nprim + (q.z - 1)] : ja8(Pi, Pk, Rik2, aik, eik);
  const double Jjl = Jtab ? Jtab[static_cast<int64_t>(q.y - 1) * cP.nprim + (q.w - 1)] : ja8(Pj, Pl, Rjl2, ajl, ejl);
  const double lim = cP.thresh * Pi.lim_scale;
  const double screen1 = fabs(DMval) * sqrt(Jik * Jjl);
  *s1o = screen1;
  *s2o = 0.0;
  if (!(screen1 >= lim)) return 0;
  const double zeta = aik + ajl;
  const double eijkl = (aik * ajl) * (1.0 / zeta);
  const double sqe = sqrt(eijkl);
  double Pik[3], Pjl[3], Pijkl[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    Pik[d] = (Pi.alpha * Xi[d] + Pk.alpha * Xk[d]) * (1.0 / aik);
    Pjl[d] = (Pj.alpha * Xj[d] + Pl.alpha * Xl[d]) * (1.0 / ajl);
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) Pijkl[d] = (aik * Pik[d] + ajl * Pjl[d]) * (1.0 / zeta);
  const double invz = 1.0 / sqrt(zeta);
  const double alf = (0.5 * (aik - ajl)) * (1.0 / zeta);
  double A = DMval * (1.0 / (zeta * sqrt(zeta)));
  A = A * pexp((-eik) * Rik2 - ejl * Rjl2);
  double U[3];
  for (int d = 0; d < 3; ++d) {
    const double R[4] = {Xi[d], Xj[d], Xk[d], Xl[d]};
    const int t[4] = {Pi.t[d], Pj.t[d], Pk.t[d], Pl.t[d]};
    out->L[d] = t[0] + t[1] + t[2] + t[3];
    polycoef(R, Pik[d], Pjl[d], Pijkl[d], t, sqe, invz, alf, out->C[d]);
    U[d] = 0.0;
    for (int m = 0; m <= out->L[d]; ++m) U[d] = U[d] + out->C[d][m] * cP.wm[m];
  }
  const double screen2 = fabs(((A * U[0]) * U[1]) * U[2]);
  *s2o = screen2;
  if (!(screen2 >= lim)) return 1;
  out->A = A;
  out->sqe = sqe;
#pragma unroll
  for (int d = 0; d < 3; ++d) out->d[d] = Pik[d] - Pjl[d];
  return 3;
}

// Group of a quartet: its molecule's first key plus (pair of shells i, k; pair of shells j, l).
__device__ __forceinline__ uint64_t quartet_group_key(const PrimD& i, const PrimD& j, const PrimD& k, const PrimD& l) {
  const int64_t np = static_cast<int64_t>(i.nshell) * (i.nshell + 1) / 2;
  const int64_t hi = max(i.shell, k.shell), lo = min(i.shell, k.shell);
  const int64_t hj = max(j.shell, l.shell), lj = min(j.shell, l.shell);
  return static_cast<uint64_t>(i.gbase + (hi * (hi + 1) / 2 + lo) * np + hj * (hj + 1) / 2 + lj);
}

// Counters of a preparation, read back together.
enum PrepCount { kNScreen1 = 0, kNBad, kNSurv, kNGroup, kNRec, kNProduct, kNClass, kNCounts };

// Screening of every quartet; group key of the survivors (the others get fail_key and sort last).
__global__ void k_screen(int64_t n, const int4* __restrict__ ijkl, const double* __restrict__ v,
                         const PrimD* __restrict__ prims, uint8_t* flags, double* s1, double* s2, uint64_t* key,
                         int64_t* idx, uint64_t fail_key, unsigned long long* count,
                         const double* __restrict__ Jtab, QRec* qcache) {
  const int64_t q = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  int f = 0;
  if (q < n) {
    const int4 r = ijkl[q];
    idx[q] = q;
    uint64_t kq = fail_key;
    double a1 = 0.0, a2 = 0.0;
    if (r.x < 1 || r.y < 1 || r.z < 1 || r.w < 1 || r.x > cP.nprim || r.y > cP.nprim || r.z > cP.nprim ||
        r.w > cP.nprim) {
      count[kNBad] = 1;
    } else {
      QRec rec;
      f = prepare_one(prims, r, v[q], &rec, &a1, &a2, Jtab);
      if (f == 3) {
        kq = quartet_group_key(prims[r.x - 1], prims[r.y - 1], prims[r.z - 1], prims[r.w - 1]);
        if (qcache) qcache[q] = rec;
      }
    }
    flags[q] = static_cast<uint8_t>(f);
    if (s1) s1[q] = a1;
    if (s2) s2[q] = a2;
    key[q] = kq;
  }
  // warp-aggregated counts of the survivors
  const unsigned b1 = __ballot_sync(0xffffffffu, f & 1), b3 = __ballot_sync(0xffffffffu, f == 3);
  if ((threadIdx.x & 31) == 0) {
    if (b1) atomicAdd(&count[kNScreen1], static_cast<unsigned long long>(__popc(b1)));
    if (b3) atomicAdd(&count[kNSurv], static_cast<unsigned long long>(__popc(b3)));
  }
}

// First quartet of a group in the sorted keys.
struct GroupHead {
  const uint64_t* key;
  uint64_t fail_key;
  __device__ bool operator()(int64_t i) const {
    return key[i] != fail_key && (i == 0 || key[i] != key[i - 1]);
  }
};
struct Survivor {
  const uint8_t* flags;
  __device__ bool operator()(int64_t i) const { return flags[i] == 3; }
};

// Instructions a term costs at a point in the FP32 evaluation, counted in mixed_eval.cu's terms32:
// what decides between one merged record and a product record per quartet.
__device__ __forceinline__ int product_cost(int sum_l) { return 50 + 2 * sum_l; }
__device__ __forceinline__ int merged_cost(int shape) { return 44 + shape_coefs(shape) + 2 * ((shape >> 15) & 31); }

// Shape and record count of every group: one warp per group. gkey: (molecule, shape) of a merged
// group; gcount: its records (1, or one per quartet when the products stay).
__global__ void k_classify(const int64_t* __restrict__ goff, const int64_t* __restrict__ idx,
                           const int4* __restrict__ ijkl, const PrimD* __restrict__ prims, uint32_t* gkey,
                           int64_t* gcount, unsigned long long* count) {
  const int lane = threadIdx.x & 31;
  const int64_t ngroup = static_cast<int64_t>(count[kNGroup]), nsurv = static_cast<int64_t>(count[kNSurv]);
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x / 32);
  unsigned long long nrec = 0, nprod = 0;
  for (int64_t g = blockIdx.x * static_cast<int64_t>(blockDim.x / 32) + (threadIdx.x >> 5); g < ngroup; g += warps) {
    const int64_t m0 = goff[g], m1 = g + 1 < ngroup ? goff[g + 1] : nsurv;
    int L[3] = {0, 0, 0}, total = 0, mol = 0;
    unsigned long long cost = 0;
    for (int64_t m = m0 + lane; m < m1; m += 32) {
      const int4 q = ijkl[idx[m]];
      const PrimD &Pi = prims[q.x - 1], &Pj = prims[q.y - 1], &Pk = prims[q.z - 1], &Pl = prims[q.w - 1];
      int sum = 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int l = Pi.t[d] + Pj.t[d] + Pk.t[d] + Pl.t[d];
        L[d] = max(L[d], l);
        sum += l;
      }
      total = max(total, sum);
      cost += product_cost(sum);
      mol = Pi.mol;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) L[d] = __reduce_max_sync(0xffffffffu, L[d]);
    total = __reduce_max_sync(0xffffffffu, total);
    mol = __reduce_max_sync(0xffffffffu, mol);
    for (int o = 16; o > 0; o >>= 1) cost += __shfl_xor_sync(0xffffffffu, cost, o);
    // up to total degree 2 the full polynomial (1, 4 or 10 coefficients, unrolled in the kernels)
    if (total <= 2) L[0] = L[1] = L[2] = total;
    bool merged = total <= kMaxTotal;
    const int shape = pack_shape(L[0], L[1], L[2], merged ? total : 0, true);
    merged = merged && merged_cost(shape) <= cost;
    if (lane == 0) {
      gkey[g] = (static_cast<uint32_t>(mol) << 21) | static_cast<uint32_t>(shape);
      gcount[g] = merged ? 1 : m1 - m0;
      nrec += merged ? 1 : m1 - m0;
      nprod += merged ? 0 : m1 - m0;
    }
  }
  if (lane == 0 && nrec) atomicAdd(&count[kNRec], nrec);
  if (lane == 0 && nprod) atomicAdd(&count[kNProduct], nprod);
}

// Class key and source of every record: merged records point at their group (>= 0), product records
// at their quartet's place in the sorted list (-1 - place). gstart: first record of each group.
__global__ void k_record_keys(int64_t ngroup, int64_t nsurv, const int64_t* __restrict__ goff,
                              const uint32_t* __restrict__ gkey, const int64_t* __restrict__ gcount,
                              const int64_t* __restrict__ gstart, const int64_t* __restrict__ idx,
                              const int4* __restrict__ ijkl, const PrimD* __restrict__ prims, uint32_t* rkey,
                              int64_t* rsrc) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x / 32);
  for (int64_t g = blockIdx.x * static_cast<int64_t>(blockDim.x / 32) + (threadIdx.x >> 5); g < ngroup; g += warps) {
    const int64_t m0 = goff[g], m1 = g + 1 < ngroup ? goff[g + 1] : nsurv, at = gstart[g];
    // a group of one quartet may be either kind: the cost decided, and the key tells them apart
    int shape = static_cast<int>(gkey[g] & 0x1FFFFFu);
    if (gcount[g] == 1 && m1 - m0 > 1) {
      if (lane == 0) {
        rkey[at] = gkey[g];
        rsrc[at] = g;
      }
      continue;
    }
    for (int64_t m = m0 + lane; m < m1; m += 32) {
      const int4 q = ijkl[idx[m]];
      const PrimD &Pi = prims[q.x - 1], &Pj = prims[q.y - 1], &Pk = prims[q.z - 1], &Pl = prims[q.w - 1];
      int L[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) L[d] = Pi.t[d] + Pj.t[d] + Pk.t[d] + Pl.t[d];
      const int sum = L[0] + L[1] + L[2];
      const bool merged = m1 - m0 == 1 && sum <= kMaxTotal && merged_cost(shape) <= product_cost(sum);
      rkey[at + (m - m0)] = merged ? gkey[g]
                                   : (static_cast<uint32_t>(Pi.mol) << 21) |
                                         static_cast<uint32_t>(pack_shape(L[0], L[1], L[2], 0, false));
      rsrc[at + (m - m0)] = merged ? g : -1 - m;
    }
  }
}

__global__ void k_iota(int64_t n, int64_t* x) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i < n) x[i] = i;
}

__device__ __forceinline__ int segment_of(const ClassSeg* __restrict__ segs, int nseg, int64_t r) {
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (segs[mid].first <= r) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ void hi_lo(double x, float* hi, float* lo) {
  *hi = static_cast<float>(x);
  *lo = static_cast<float>(x - static_cast<double>(*hi));
}

// Shared memory of k_merge: the polynomials (D coefficients a dimension, ascending powers) and
// amplitudes of 32 quartets, the record's coefficients and their exponents.
inline size_t merge_smem(int D, int nc) {
  return sizeof(double) * (32 * (3 * D + 1) + static_cast<size_t>(nc) + 8) + sizeof(uint16_t) * static_cast<size_t>(nc);
}

// Merged records, one warp each: the group's quartets 32 at a time (a lane restates one quartet, or
// reads it where k_screen kept it), then every lane sums its coefficients over them in input order.
//   FP64 record [1, sqe, d0, d1, d2, 0, c_abc...] (powers of r' = sqe (r + d));
//   FP32 record [s_hi, s_lo, b_hi[3], b_lo[3], 0, quartets, ks, ks, c_hi..., c_lo..., S_total..., S_0]
// with s = sqe c_u, b_d = s d_d, u = s (r + d) = c_u r', the polynomial rewritten in u and divided by
// the power of two 2^ks above its largest coefficient (applied exactly by the evaluation's exp2), and
// S_k = sqrt(sum over a + b + c = k of c_abc^2 a! b! c! / k!): by Cauchy-Schwarz
// sum |c_abc u_x^a u_y^b u_z^c| <= sum_k S_k |u|^k, which the error bounds use (one Horner loop over
// the total degree instead of a second one over all coefficients). hi/lo pairs carry the FP64 value
// to about 2^-48.
__global__ void __launch_bounds__(32)
k_merge(const int64_t* __restrict__ rsrc, const int64_t* __restrict__ goff, int64_t ngroup, int64_t nsurv,
        const int64_t* __restrict__ idx, const int4* __restrict__ ijkl, const double* __restrict__ v,
        const PrimD* __restrict__ prims, const ClassSeg* __restrict__ segs, int nseg, int D, int nc_max,
        double* rec64, float* rec32, const double* __restrict__ Jtab, const QRec* __restrict__ qcache) {
  extern __shared__ double sm[];
  const int64_t r = blockIdx.x;
  const ClassSeg sg = segs[segment_of(segs, nseg, r)];
  if (!(sg.shape & kMergedBit)) return;
  const int lane = threadIdx.x, nc = sg.nc;
  const int Lx = sg.shape & 31, Ly = (sg.shape >> 5) & 31, Lz = (sg.shape >> 10) & 31, total = (sg.shape >> 15) & 31;
  double* pol = sm;
  double* amp = pol + 32 * 3 * D;
  double* head = amp + 32;  // sqe, d0, d1, d2
  double* coef = head + 8;
  uint16_t* abc = reinterpret_cast<uint16_t*>(coef + nc_max);
  {
    int i = 0;
    for (int a = min(Lx, total); a >= 0; --a)
      for (int b = min(Ly, total - a); b >= 0; --b)
        for (int c = min(Lz, total - a - b); c >= 0; --c, ++i)
          if ((i & 31) == lane) {
            abc[i] = static_cast<uint16_t>(a | (b << 5) | (c << 10));
            coef[i] = 0.0;
          }
  }
  const int64_t g = rsrc[r];
  const int64_t m0 = goff[g], m1 = g + 1 < ngroup ? goff[g + 1] : nsurv;
  for (int64_t at = m0; at < m1; at += 32) {
    const int k = static_cast<int>(min(static_cast<int64_t>(32), m1 - at));
    __syncwarp();
    if (lane < k) {
      const int64_t q = idx[at + lane];
      QRec own;
      const QRec* rec = &own;
      if (qcache) {
        rec = qcache + q;
      } else {
        double a1, a2;
        prepare_one(prims, ijkl[q], v[q], &own, &a1, &a2, Jtab);
      }
      amp[lane] = rec->A;
      for (int d = 0; d < 3; ++d) {
        const int L = rec->L[d];
        for (int p = 0; p < D; ++p) pol[(lane * 3 + d) * D + p] = p <= L ? rec->C[d][L - p] : 0.0;
      }
      if (at == m0 && lane == 0) {
        head[0] = rec->sqe;
        for (int d = 0; d < 3; ++d) head[1 + d] = rec->d[d];
      }
    }
    __syncwarp();
    for (int i = lane; i < nc; i += 32) {
      const int a = abc[i] & 31, b = (abc[i] >> 5) & 31, c = abc[i] >> 10;
      double s = coef[i];
      for (int m = 0; m < k; ++m) {
        const double* P = pol + m * 3 * D;
        s = s + (amp[m] * P[a]) * (P[D + b] * P[2 * D + c]);
      }
      coef[i] = s;
    }
  }
  __syncwarp();
  const int64_t local = r - sg.first;
  double* r64 = rec64 + sg.off64 + local * sg.stride;
  float* r32 = rec32 + sg.off32 + local * sg.stride32;
  double big = 0.0;
  for (int i = lane; i < sg.stride - kRecHeader; i += 32) r64[kRecHeader + i] = i < nc ? coef[i] : 0.0;
  __syncwarp();
  for (int i = lane; i < nc; i += 32) {
    const int k = (abc[i] & 31) + ((abc[i] >> 5) & 31) + (abc[i] >> 10);
    coef[i] = coef[i] * ipow(1.0 / cP.c_u, k);
    big = fmax(big, fabs(coef[i]));
  }
  for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
  int ks = 0;
  if (big > 0.0) frexp(big, &ks);
  for (int i = lane; i < nc; i += 32) {
    coef[i] = ldexp(coef[i], -ks);
    hi_lo(coef[i], &r32[12 + i], &r32[12 + nc + i]);
  }
  __syncwarp();
  if (lane <= total) {
    double s2 = 0.0;
    for (int i = 0; i < nc; ++i) {
      const int a = abc[i] & 31, b = (abc[i] >> 5) & 31, c = abc[i] >> 10;
      if (a + b + c != lane) continue;
      double w = 1.0;  // a! b! c! / k! = 1 / (binom(a + b, b) binom(k, c))
      for (int p = 1; p <= b; ++p) w = w * static_cast<double>(p) / static_cast<double>(a + p);
      for (int p = 1; p <= c; ++p) w = w * static_cast<double>(p) / static_cast<double>(a + b + p);
      s2 = s2 + coef[i] * coef[i] * w;
    }
    // raised by a margin for its FP32 rounding and that of the evaluation's |u|
    r32[12 + 2 * nc + total - lane] = static_cast<float>(sqrt(s2) * (1.0 + 1e-6 * (4 + lane)));
  }
  for (int i = 12 + 2 * nc + total + 1 + lane; i < sg.stride32; i += 32) r32[i] = 0.0f;
  if (lane == 0) {
    const double sqe = head[0], s = sqe * cP.c_u;
    r64[0] = 1.0;
    r64[1] = sqe;
    hi_lo(s, &r32[0], &r32[1]);
    for (int d = 0; d < 3; ++d) {
      r64[2 + d] = head[1 + d];
      hi_lo(s * head[1 + d], &r32[2 + d], &r32[5 + d]);
    }
    r64[5] = 0.0;
    r32[8] = 0.0f;
    r32[9] = static_cast<float>(m1 - m0);
    r32[10] = r32[11] = static_cast<float>(ks);
  }
}

// Product records, one thread each: restate the quartet (identical arithmetic) and write
// its records into the class segments:
//   FP64 record [A, sqe, d0, d1, d2, A', Cx.., Cy.., Cz..] (C highest degree first);
//   FP32 record [s_hi, s_lo, b_hi[3], b_lo[3], A'_hi, A'_lo, la, 0, Cn_hi (x,y,z), Cn_lo (x,y,z)]
// with s = sqe c_u, b_d = s d_d, u = s (r + d) = c_u r', the polynomials rewritten in u and
// scaled by kappa_d (largest |coefficient|) so that Cn has max |coefficient| 1, A' = A prod
// kappa_d, and la = log2(|A'| prod_d sum_k |Cn_dk|). hi/lo pairs carry the FP64 value to
// ~2^-48 relative (see mixed_eval.cu).
__global__ void k_build(int64_t nrec, const int64_t* __restrict__ rsrc, const int64_t* __restrict__ idx,
                        const int4* __restrict__ ijkl, const double* __restrict__ v,
                        const PrimD* __restrict__ prims, const ClassSeg* __restrict__ segs, int nseg, double* rec64,
                        float* rec32, const double* __restrict__ Jtab, const QRec* __restrict__ qcache) {
  const int64_t p = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (p >= nrec) return;
  const ClassSeg sg = segs[segment_of(segs, nseg, p)];
  if (sg.shape & kMergedBit) return;
  const int64_t src = idx[-1 - rsrc[p]];
  QRec rec;
  if (qcache) {
    rec = qcache[src];
  } else {
    double a1, a2;
    prepare_one(prims, ijkl[src], v[src], &rec, &a1, &a2, Jtab);
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
static cudaError_t upload_constants(inca_ctx* c, double thresh, int normalize) {
  PrepConst hc;
  std::memset(&hc, 0, sizeof(hc));
  const double pi = 4.0 * std::atan(1.0);
  for (int m = 1; m <= kMaxCoef; ++m)
    hc.wm[m - 1] = (m == 1) ? 1.0 : std::pow(double(m) * 0.5, double(m) * 0.5) * std::exp(-double(m) * 0.5);
  for (int n = 0; n <= kMaxGH; ++n)
    for (int h = 0; h < kMaxGH; ++h) {
      hc.gh_node[n][h] = inca_gh::kNode[n][h];
      hc.gh_w[n][h] = inca_gh::kWeight[n][h];
    }
  hc.pi15 = pi * std::sqrt(pi);
  hc.thresh = thresh;
  hc.c_u = std::sqrt(1.0 / std::log(2.0));
  hc.nprim = c->nprim;
  hc.normalize = normalize ? 1 : 0;
  return cudaMemcpyToSymbolAsync(cP, &hc, sizeof(hc), 0, cudaMemcpyHostToDevice, c->stream);
}

// Bytes of each of the two staging buffers that a work chunk may fill: with 16 one-warp CTAs per SM
// the mixed evaluation has 14 KB of shared memory per CTA, 3 KB of it for its tables. (A class whose
// record alone is larger gets chunks of one record.)
constexpr int kStageFloats = 1344;

int prepare_device(inca_ctx* c, double thresh, int normalize) {
  if (c->nprim <= 0) return set_error(c, INCA_E_STATE, "inca_prepare: primitives not set");
  if (c->nq <= 0) return set_error(c, INCA_E_STATE, "inca_prepare: no quartets loaded");
  if (!(thresh > 0.0)) return set_error(c, INCA_E_ARG, "inca_prepare: thresh must be > 0");
  for (int p = 0; p < c->nprim; ++p)
    for (int d = 0; d < 3; ++d)
      if (c->h_tmn[3 * p + d] < 0 || c->h_tmn[3 * p + d] > 4)
        return set_error(c, INCA_E_LIMIT, "inca_prepare: Cartesian power above 4 (g) in primitive " +
                                              std::to_string(p + 1));
  c->lim = thresh * (1.0 / (double(c->nprim) * (double(c->nprim) + 1.0) * 0.5));
  INCA_CUDA(c, upload_constants(c, thresh, normalize));

  const int64_t n = c->nq;
  const bool keep_values = n <= (int64_t(1) << 27);
  if (c->d_flags.reserve(n) != cudaSuccess) return set_error(c, INCA_E_NOMEM, "flags");
  if (keep_values) {
    if (c->d_s1.reserve(n) != cudaSuccess || c->d_s2.reserve(n) != cudaSuccess)
      return set_error(c, INCA_E_NOMEM, "screening values");
  }
  c->have_screen_values = keep_values;
  // sort and grouping scratch, owned by the context: kept between calls for lists of up to
  // kPrepKeepQuartets quartets (a repeated preparation then allocates and frees nothing, and no
  // cudaFree stalls the stream), given back after the call for larger lists
  DevBuf<uint64_t>& key = c->d_pkey;
  DevBuf<uint64_t>& key2 = c->d_pkey2;
  DevBuf<int64_t>& idx = c->d_pidx;
  DevBuf<int64_t>& idx2 = c->d_pidx2;
  DevBuf<int64_t>& goff = c->d_pgoff;
  DevBuf<unsigned char>& tmp = c->d_ptmp;
  DevBuf<unsigned char>& group = c->d_pgroup;
  DevBuf<unsigned char>& rbuf = c->d_prec;
  DevBuf<unsigned long long>& count = c->d_pcount;
  DevBuf<unsigned char>& qrec = c->d_pqrec;
  auto release_all = [&]() {
    key.release(); key2.release(); idx.release(); idx2.release(); goff.release(); tmp.release(); group.release();
    rbuf.release(); count.release(); qrec.release();
  };
  const bool keep_scratch = n <= kPrepKeepQuartets;
  auto cleanup = [&]() {
    if (!keep_scratch) release_all();
  };
  // groups: at most one per quartet and one per key
  const int64_t gcap = std::min<int64_t>(n, c->group_keys);
  const uint64_t fail_key = static_cast<uint64_t>(c->group_keys);
  int key_bits = 1;
  while ((fail_key >> key_bits) != 0) ++key_bits;
  // gcount and gstart (8 bytes each) and gkey (4) of every group
  if (key.reserve(n) || key2.reserve(n) || idx.reserve(n) || idx2.reserve(n) || goff.reserve(gcap) ||
      group.reserve(20 * static_cast<size_t>(gcap)) || count.reserve(kNCounts)) {
    release_all();
    return set_error(c, INCA_E_NOMEM, "inca_prepare: sort buffers");
  }
  int64_t* gcount = reinterpret_cast<int64_t*>(group.p);
  int64_t* gstart = gcount + gcap;
  uint32_t* gkey = reinterpret_cast<uint32_t*>(gstart + gcap);
  QRec* qcache = nullptr;
  if (n <= kQRecCacheQuartets) {
    if (qrec.reserve(sizeof(QRec) * std::max<int64_t>(n, 1)) == cudaSuccess)
      qcache = reinterpret_cast<QRec*>(qrec.p);
    else
      (void)cudaGetLastError();  // no room: build the records from the indices instead
  }
  auto storage = [&](size_t bytes) { return bytes > tmp.n ? tmp.reserve(bytes) : cudaSuccess; };
  cudaError_t e = cudaMemsetAsync(count.p, 0, kNCounts * sizeof(unsigned long long), c->stream);
  const int bs = 128;
  const int64_t grid = (n + bs - 1) / bs;
  // JA8 of every primitive pair, once (up to kPairTableMax primitives: 128 MiB); beyond that each
  // quartet evaluates its two JA8 bounds itself
  const double* jtab = nullptr;
  if (e == cudaSuccess && c->nprim <= kPairTableMax) {
    const int64_t np2 = static_cast<int64_t>(c->nprim) * c->nprim;
    if (c->d_ja8.reserve(np2) == cudaSuccess) {
      INCA_LAUNCH(c, k_pair_ja8, static_cast<unsigned>((np2 + 127) / 128), 128, 0, c->nprim, c->d_prims.p,
                  c->d_ja8.p);
      e = cudaGetLastError();
      jtab = c->d_ja8.p;
    }
  }
  if (e == cudaSuccess) {
    INCA_LAUNCH(c, k_screen, static_cast<unsigned>(grid), bs, 0, n, c->d_ijkl.p, c->d_v.p, c->d_prims.p, c->d_flags.p,
                keep_values ? c->d_s1.p : nullptr, keep_values ? c->d_s2.p : nullptr, key.p, idx.p, fail_key, count.p,
                jtab, qcache);
    e = cudaGetLastError();
  }
  // survivors by group (stable: a group's quartets stay in input order)
  size_t tb = 0;
  if (e == cudaSuccess)
    e = cub::DeviceRadixSort::SortPairs(nullptr, tb, key.p, key2.p, idx.p, idx2.p, n, 0, key_bits, c->stream);
  if (e == cudaSuccess) e = storage(tb);
  if (e == cudaSuccess)
    e = cub::DeviceRadixSort::SortPairs(tmp.p, tb, key.p, key2.p, idx.p, idx2.p, n, 0, key_bits, c->stream);
  const thrust::counting_iterator<int64_t> places(0);
  int64_t* ngroup_dev = reinterpret_cast<int64_t*>(count.p + kNGroup);
  if (e == cudaSuccess)
    e = cub::DeviceSelect::If(nullptr, tb, places, goff.p, ngroup_dev, n, GroupHead{key2.p, fail_key}, c->stream);
  if (e == cudaSuccess) e = storage(tb);
  if (e == cudaSuccess)
    e = cub::DeviceSelect::If(tmp.p, tb, places, goff.p, ngroup_dev, n, GroupHead{key2.p, fail_key}, c->stream);
  const unsigned gblocks = static_cast<unsigned>(std::min<int64_t>((gcap + 7) / 8, 16LL * c->num_sms));
  if (e == cudaSuccess) {
    INCA_LAUNCH(c, k_classify, gblocks, 256, 0, goff.p, idx2.p, c->d_ijkl.p, c->d_prims.p, gkey, gcount, count.p);
    e = cudaGetLastError();
  }
  unsigned long long hc[kNCounts] = {};
  if (e == cudaSuccess) e = cudaMemcpyAsync(hc, count.p, sizeof(hc), cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) {
    release_all();
    return cuda_error(c, e, "inca_prepare (screening)");
  }
  if (hc[kNBad]) {
    cleanup();
    return set_error(c, INCA_E_ARG, "inca_prepare: quartet index outside 1..nprim");
  }
  const int64_t nsurv = static_cast<int64_t>(hc[kNSurv]), ngroup = static_cast<int64_t>(hc[kNGroup]);
  const int64_t nrec = static_cast<int64_t>(hc[kNRec]);
  // records by class: sources (two arrays), class keys (two) and the classes' keys and counts
  int64_t *rsrc = nullptr, *rsrc2 = nullptr, *ucount = nullptr;
  uint32_t *rkey = nullptr, *rkey2 = nullptr, *ukey = nullptr;
  std::vector<uint32_t> hk;
  std::vector<int64_t> hcnt;
  if (nrec > 0) {
    if (rbuf.reserve(36 * static_cast<size_t>(nrec))) {
      release_all();
      return set_error(c, INCA_E_NOMEM, "inca_prepare: record keys");
    }
    rsrc = reinterpret_cast<int64_t*>(rbuf.p);
    rsrc2 = rsrc + nrec;
    ucount = rsrc2 + nrec;
    rkey = reinterpret_cast<uint32_t*>(ucount + nrec);
    rkey2 = rkey + nrec;
    ukey = rkey2 + nrec;
    if (hc[kNProduct] == 0) {  // every group is one merged record
      INCA_LAUNCH(c, k_iota, static_cast<unsigned>((nrec + 255) / 256), 256, 0, nrec, rsrc);
      rkey = gkey;
    } else {
      e = cub::DeviceScan::ExclusiveSum(nullptr, tb, gcount, gstart, ngroup, c->stream);
      if (e == cudaSuccess) e = storage(tb);
      if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(tmp.p, tb, gcount, gstart, ngroup, c->stream);
      if (e == cudaSuccess)
        INCA_LAUNCH(c, k_record_keys, gblocks, 256, 0, ngroup, nsurv, goff.p, gkey, gcount, gstart, idx2.p,
                    c->d_ijkl.p, c->d_prims.p, rkey, rsrc);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess)
      e = cub::DeviceRadixSort::SortPairs(nullptr, tb, rkey, rkey2, rsrc, rsrc2, nrec, 0, 28, c->stream);
    if (e == cudaSuccess) e = storage(tb);
    if (e == cudaSuccess)
      e = cub::DeviceRadixSort::SortPairs(tmp.p, tb, rkey, rkey2, rsrc, rsrc2, nrec, 0, 28, c->stream);
    int64_t* nclass_dev = reinterpret_cast<int64_t*>(count.p + kNClass);
    if (e == cudaSuccess)
      e = cub::DeviceRunLengthEncode::Encode(nullptr, tb, rkey2, ukey, ucount, nclass_dev, nrec, c->stream);
    if (e == cudaSuccess) e = storage(tb);
    if (e == cudaSuccess)
      e = cub::DeviceRunLengthEncode::Encode(tmp.p, tb, rkey2, ukey, ucount, nclass_dev, nrec, c->stream);
    int64_t nclass = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&nclass, nclass_dev, sizeof(nclass), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    hk.resize(nclass);
    hcnt.resize(nclass);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(hk.data(), ukey, sizeof(uint32_t) * nclass, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(hcnt.data(), ucount, sizeof(int64_t) * nclass, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) {
      release_all();
      return cuda_error(c, e, "inca_prepare (classes)");
    }
  }
  // class segments
  c->classes.clear();
  int64_t first = 0, off64 = 0, off32 = 0;
  int max_l = 0, max_nc = 1;  // of the merged records
  for (size_t r = 0; r < hk.size(); ++r) {
    ClassSeg s;
    s.mol = static_cast<int>(hk[r] >> 21);
    s.shape = static_cast<int>(hk[r] & 0x1FFFFFu);
    s.nc = shape_coefs(s.shape);
    const bool merged = (s.shape & kMergedBit) != 0;
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
    if (merged) {
      max_l = std::max({max_l, s.shape & 31, (s.shape >> 5) & 31, (s.shape >> 10) & 31});
      max_nc = std::max(max_nc, s.nc);
    }
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
      WorkChunk w;
      w.cls = s;
      w.count = static_cast<int>(std::min<int64_t>(sg.per_chunk, sg.count - f));
      w.rec = sg.first + f;
      c->chunks.push_back(w);
    }
    c->mol_chunks[sg.mol].end = static_cast<int>(c->chunks.size());
  }
  e = cudaSuccess;
  if (c->d_rec64.reserve(std::max<int64_t>(off64, 2)) || c->d_rec32.reserve(std::max<int64_t>(off32, 4)) ||
      c->d_classes.reserve(std::max<size_t>(c->classes.size(), 1)) ||
      c->d_chunks.reserve(std::max<size_t>(c->chunks.size(), 1))) {
    release_all();
    return set_error(c, INCA_E_NOMEM, "inca_prepare: survivor records");
  }
  if (!c->classes.empty())
    e = cudaMemcpyAsync(c->d_classes.p, c->classes.data(), sizeof(ClassSeg) * c->classes.size(),
                        cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess && !c->chunks.empty())
    e = cudaMemcpyAsync(c->d_chunks.p, c->chunks.data(), sizeof(WorkChunk) * c->chunks.size(),
                        cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess && nrec > 0) {
    const int nseg = static_cast<int>(c->classes.size());
    const int D = max_l + 1;
    INCA_LAUNCH(c, k_merge, static_cast<unsigned>(nrec), 32, merge_smem(D, max_nc), rsrc2, goff.p, ngroup, nsurv,
                idx2.p, c->d_ijkl.p, c->d_v.p, c->d_prims.p, c->d_classes.p, nseg, D, max_nc, c->d_rec64.p,
                c->d_rec32.p, jtab, qcache);
    e = cudaGetLastError();
    if (e == cudaSuccess && hc[kNProduct] > 0) {
      INCA_LAUNCH(c, k_build, static_cast<unsigned>((nrec + bs - 1) / bs), bs, 0, nrec, rsrc2, idx2.p, c->d_ijkl.p,
                  c->d_v.p, c->d_prims.p, c->d_classes.p, nseg, c->d_rec64.p, c->d_rec32.p, jtab, qcache);
      e = cudaGetLastError();
    }
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) {
    release_all();
    return cuda_error(c, e, "inca_prepare (records)");
  }
  cleanup();
  c->counts.read = n;
  c->counts.after_screen1 = static_cast<int64_t>(hc[kNScreen1]);
  c->counts.after_screen2 = nsurv;
  c->prep_thresh = thresh;
  c->prep_normalize = normalize;
  c->prepared = true;
  ++c->prepare_count;
  c->evaluated = false;
  return INCA_OK;
}

// ---------------------------------------------------------------- survivor records, one per quartet
namespace {
__global__ void k_records(int64_t n, const int64_t* __restrict__ idx, const int4* __restrict__ ijkl,
                          const double* __restrict__ v, const PrimD* __restrict__ prims, double* A, double* sqe,
                          double* d, int32_t* L, double* C) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  QRec rec;
  double a1, a2;
  prepare_one(prims, ijkl[idx[i]], v[idx[i]], &rec, &a1, &a2);
  A[i] = rec.A;
  sqe[i] = rec.sqe;
  for (int x = 0; x < 3; ++x) {
    d[3 * i + x] = rec.d[x];
    L[3 * i + x] = rec.L[x];
    for (int m = 0; m < kMaxCoef; ++m) C[(3 * i + x) * kMaxCoef + m] = m <= rec.L[x] ? rec.C[x][m] : 0.0;
  }
}
}  // namespace

// The evaluation keeps merged records only, so the quartets' own records (inca_get_records) are
// restated from the input, with the arithmetic of the screening, in input order.
int get_records_device(inca_ctx* c, double* A, double* sqe, double* d, int32_t* L, double* C) {
  const int64_t ns = c->nsurv;
  if (ns == 0) return INCA_OK;
  constexpr int64_t kPart = int64_t(1) << 18;  // survivors at a time (120 MB)
  const int64_t part = std::min(ns, kPart);
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
  const thrust::counting_iterator<int64_t> places(0);
  size_t tb = 0;
  INCA_CUDA(c, upload_constants(c, c->prep_thresh, c->prep_normalize));
  INCA_CUDA(c, cub::DeviceSelect::If(nullptr, tb, places, idx.p, nsel.p, c->nq, Survivor{c->d_flags.p}, c->stream));
  if (idx.reserve(ns) || nsel.reserve(1) || tmp.reserve(std::max<size_t>(tb, 1)) ||
      val.reserve(part * (5 + 3 * kMaxCoef)) || deg.reserve(3 * part))
    return set_error(c, INCA_E_NOMEM, "inca_get_records");
  INCA_CUDA(c, cub::DeviceSelect::If(tmp.p, tb, places, idx.p, nsel.p, c->nq, Survivor{c->d_flags.p}, c->stream));
  double *vA = val.p, *vs = vA + part, *vd = vs + part, *vC = vd + 3 * part;
  for (int64_t o = 0; o < ns; o += part) {
    const int64_t k = std::min(part, ns - o);
    INCA_LAUNCH(c, k_records, static_cast<unsigned>((k + 127) / 128), 128, 0, k, idx.p + o, c->d_ijkl.p, c->d_v.p,
                c->d_prims.p, vA, vs, vd, deg.p, vC);
    INCA_CUDA(c, cudaGetLastError());
    auto copy = [&](auto* to, const auto* from, int64_t per) {
      return to ? cudaMemcpyAsync(to + o * per, from, sizeof(*to) * k * per, cudaMemcpyDeviceToHost, c->stream)
                : cudaSuccess;
    };
    INCA_CUDA(c, copy(A, vA, 1));
    INCA_CUDA(c, copy(sqe, vs, 1));
    INCA_CUDA(c, copy(d, vd, 3));
    INCA_CUDA(c, copy(L, deg.p, 3));
    INCA_CUDA(c, copy(C, vC, 3 * kMaxCoef));
    INCA_CUDA(c, cudaStreamSynchronize(c->stream));
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
