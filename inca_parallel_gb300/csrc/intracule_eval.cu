// K2: evaluation of the intracule at every grid point (src/mod_intracule.f90:345-358):
//   I(r_g) = sum over surviving quartets q of A_q exp(-|r'|^2) Vx(r'_x) Vy(r'_y) Vz(r'_z),
//   r' = sqe_q (r_g + P_ik - P_jl), V_d a Horner polynomial of degree L_d.
// Quartets of the same four shells share A's Gaussian and come merged into one record, with one
// trivariate polynomial in the place of their products (quartet_prep.cu).
//
// Work decomposition (both precisions): a CTA owns a tile of grid points (registers) and a
// strided subset of the class-uniform work chunks (<= 32 records of one class, staged in shared
// memory). Each (tile, split) writes its FP64 partial sums; a second
// kernel adds the splits in a fixed order, so results are bit-reproducible run to run.
//
// INCA_FP64: every term in FP64 (the "plain FP64 GPU form").
// INCA_MIXED: see mixed_eval.cu.
#include <algorithm>
#include <cmath>

#include "exp64.cuh"
#include "inca_internal.h"

namespace inca {

int eval_mixed(inca_ctx* c, double tol);        // mixed_eval.cu
int eval_mixed_graph(inca_ctx* c, double tol);  // mixed_eval.cu

namespace {

constexpr int kThreads64 = 128, kCtas64 = 10;  // CTAs per SM
constexpr int kPPT64 = 2;  // points per thread
constexpr int kTile64 = kThreads64 * kPPT64;

// The trivariate polynomial of a merged record (FP64 records: powers of r + d) by nested Horner, at
// N points. Full polynomials of total degree 0, 1 and 2 are unrolled.
template <int N>
__device__ __forceinline__ void merged_value64(int total, const double* __restrict__ C, const double (&u)[3][N],
                                               double (&v)[N]) {
  if (total == 0) {
#pragma unroll
    for (int p = 0; p < N; ++p) v[p] = C[0];
    return;
  }
  if (total == 1) {  // x, y, z, 1
#pragma unroll
    for (int p = 0; p < N; ++p) v[p] = fma(C[0], u[0][p], fma(C[1], u[1][p], fma(C[2], u[2][p], C[3])));
    return;
  }
  if (total == 2) {  // xx, xy, xz, x, yy, yz, y, zz, z, 1
#pragma unroll
    for (int p = 0; p < N; ++p) {
      const double x = u[0][p], y = u[1][p], z = u[2][p];
      const double fx = fma(C[0], x, fma(C[1], y, fma(C[2], z, C[3])));
      const double fy = fma(C[4], y, fma(C[5], z, C[6]));
      v[p] = fma(fx, x, fma(fy, y, fma(fma(C[7], z, C[8]), z, C[9])));
    }
    return;
  }
#pragma unroll
  for (int p = 0; p < N; ++p) v[p] = 0.0;
#pragma unroll 1
  for (int nb = 0; nb <= total; ++nb) {
    double w[N];
#pragma unroll
    for (int p = 0; p < N; ++p) w[p] = 0.0;
#pragma unroll 1
    for (int nz = 0; nz <= nb; ++nz) {
      double t[N];
      const double c0 = *C++;
#pragma unroll
      for (int p = 0; p < N; ++p) t[p] = c0;
#pragma unroll 1
      for (int k = 0; k < nz; ++k) {
        const double c = *C++;
#pragma unroll
        for (int p = 0; p < N; ++p) t[p] = fma(t[p], u[2][p], c);
      }
#pragma unroll
      for (int p = 0; p < N; ++p) w[p] = nz == 0 ? t[p] : fma(w[p], u[1][p], t[p]);
    }
#pragma unroll
    for (int p = 0; p < N; ++p) v[p] = nb == 0 ? w[p] : fma(v[p], u[0][p], w[p]);
  }
}

// Terms of record R (FP64 record of the given shape) at N points, added to acc. Merged records: 14
// FP64 instructions and one a coefficient (CH4: 16.6 on average where a quartet of its own took about
// 40); product records keep the reference's form.
template <int kTab, int N>
__device__ __forceinline__ void terms64(const double* __restrict__ R, int shape, const double (&x)[3][N],
                                        const double* __restrict__ tab, double (&acc)[N]) {
  const int Lx = shape & 31, Ly = (shape >> 5) & 31, Lz = (shape >> 10) & 31;
  double u[3][N], v[N];
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int p = 0; p < N; ++p) u[d][p] = x[d][p] + R[2 + d];
  if (shape & kMergedBit) {
    merged_value64<N>((shape >> 15) & 31, R + kRecHeader, u, v);
#pragma unroll
    for (int p = 0; p < N; ++p)
      acc[p] = add_term64(
          exp2_neg64<kTab>(R[0], fma(u[2][p], u[2][p], fma(u[1][p], u[1][p], u[0][p] * u[0][p])), tab), v[p], acc[p]);
    return;
  }
  const double A = R[0], s = R[1];
  const double* Cx = R + kRecHeader;
  const double* Cy = Cx + Lx + 1;
  const double* Cz = Cy + Ly + 1;
#pragma unroll
  for (int p = 0; p < N; ++p) {
    const double rx = s * u[0][p], ry = s * u[1][p], rz = s * u[2][p];
    double vx = Cx[0], vy = Cy[0], vz = Cz[0];
    for (int m = 1; m <= Lx; ++m) vx = fma(vx, rx, Cx[m]);
    for (int m = 1; m <= Ly; ++m) vy = fma(vy, ry, Cy[m]);
    for (int m = 1; m <= Lz; ++m) vz = fma(vz, rz, Cz[m]);
    const double e = exp(-(rx * rx + ry * ry + rz * rz));
    acc[p] += A * e * vx * vy * vz;
  }
}

__global__ void __launch_bounds__(kThreads64, kCtas64)
k_eval_fp64(const WorkChunk* __restrict__ chunks, int nchunks, const ClassSeg* __restrict__ segs,
            const double* __restrict__ rec64, const double* __restrict__ px,
            const double* __restrict__ py, const double* __restrict__ pz, int64_t ngrid, int nsplit,
            const double* __restrict__ exp_tab, double* __restrict__ partial) {
  extern __shared__ double sh[];
  __shared__ double tab[kExp64TabLarge];
  const int tid = threadIdx.x;
  for (int i = tid; i < kExp64TabLarge; i += kThreads64) tab[i] = exp_tab[i];
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kTile64;
  double x[3][kPPT64], acc[kPPT64];
#pragma unroll
  for (int p = 0; p < kPPT64; ++p) {
    const int64_t g = base + tid + p * kThreads64;
    const bool ok = g < ngrid;
    x[0][p] = ok ? px[g] : 0.0;
    x[1][p] = ok ? py[g] : 0.0;
    x[2][p] = ok ? pz[g] : 0.0;
    acc[p] = 0.0;
  }
  for (int ch = blockIdx.y; ch < nchunks; ch += nsplit) {
    const WorkChunk w = chunks[ch];
    const ClassSeg& sg = segs[w.cls];
    const int stride = sg.stride, shape = sg.shape;
    const double* src = rec64 + sg.off64 + (w.rec - sg.first) * stride;
    const int nd = w.count * stride;
    __syncthreads();
    for (int i = tid; i < nd; i += kThreads64) sh[i] = src[i];
    __syncthreads();
    for (int q = 0; q < w.count; ++q) terms64<kExp64TabLarge, kPPT64>(sh + q * stride, shape, x, tab, acc);
  }
#pragma unroll
  for (int p = 0; p < kPPT64; ++p) {
    const int64_t g = base + tid + p * kThreads64;
    if (g < ngrid) partial[static_cast<int64_t>(blockIdx.y) * ngrid + g] = acc[p];
  }
}

// A few points: a lane per record, a warp per chunk (every nsplit-th from its own on), all points one after
// the other (kFewStep at a time), each point's terms added over the lanes in a fixed tree. With a thread per
// point most threads would have none: two points took 515 us, the latency of one thread's 32 records a chunk.
// At most kFewSplits warps: the partial sums (4 MB), and the sum over them, do not grow with the list.
constexpr int kFewPoints = 128;
constexpr int kFewStep = 2;
constexpr int kFewSplits = 4096;
__global__ void __launch_bounds__(kThreads64)
k_eval_fp64_few(const WorkChunk* __restrict__ chunks, int nchunks, const ClassSeg* __restrict__ segs,
                const double* __restrict__ rec64, const double* __restrict__ px, const double* __restrict__ py,
                const double* __restrict__ pz, int npts, int nsplit, const double* __restrict__ exp_tab,
                double* __restrict__ partial) {
  __shared__ double tab[kExp64Tab];
  __shared__ double xs[3][kFewPoints + kFewStep];
  __shared__ double sums[kThreads64 / 32][kFewPoints];
  for (int i = threadIdx.x; i < kExp64Tab; i += kThreads64) tab[i] = exp_tab[i * (kExp64TabLarge / kExp64Tab)];
  for (int i = threadIdx.x; i < npts + kFewStep; i += kThreads64) {
    xs[0][i] = i < npts ? px[i] : 0.0;
    xs[1][i] = i < npts ? py[i] : 0.0;
    xs[2][i] = i < npts ? pz[i] : 0.0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, split = blockIdx.x * (kThreads64 / 32) + warp;
  if (split >= nsplit) return;
  for (int ch = split; ch < nchunks; ch += nsplit) {
    const WorkChunk w = chunks[ch];
    const ClassSeg& sg = segs[w.cls];
    const int shape = __reduce_max_sync(0xffffffffu, sg.shape);
    const double* R = rec64 + sg.off64 + (w.rec - sg.first + min(lane, w.count - 1)) * sg.stride;
    for (int p = 0; p < npts; p += kFewStep) {
      double x[3][kFewStep], acc[kFewStep];
#pragma unroll
      for (int k = 0; k < kFewStep; ++k) {
        acc[k] = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) x[d][k] = xs[d][p + k];
      }
      terms64<kExp64Tab, kFewStep>(R, shape, x, tab, acc);
#pragma unroll
      for (int k = 0; k < kFewStep; ++k) {
        double t = lane < w.count ? acc[k] : 0.0;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0 && p + k < npts) {  // (sums: lane 0's alone)
          if (ch > split) t += sums[warp][p + k];
          if (ch + nsplit < nchunks)
            sums[warp][p + k] = t;
          else
            partial[static_cast<int64_t>(split) * npts + p + k] = t;
        }
      }
    }
  }
}

}  // namespace

// Sums over the split partials of each point in a fixed order, a block of 16 x 16 threads per 16
// points: thread (y, x) adds every 16th split of point x from y on, then the 16 sums in thread order.
// (One thread a point added up to 4 096 splits one after the other: 84 us for two points.)
__global__ void __launch_bounds__(256)
k_reduce_splits(const double* __restrict__ partial, int nsplit, int64_t ngrid, double* __restrict__ out) {
  __shared__ double sh[16][17];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t g = blockIdx.x * 16LL + tx;
  double s = 0.0;
  if (g < ngrid)
    for (int k = ty; k < nsplit; k += 16) s += partial[static_cast<int64_t>(k) * ngrid + g];
  sh[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && g < ngrid) {
    double t = sh[0][tx];
#pragma unroll
    for (int r = 1; r < 16; ++r) t += sh[r][tx];
    out[g] = t;
  }
}

// Number of quartet splits so that tiles x splits fill the GPU a few times over.
int choose_splits(int64_t tiles, int64_t nchunks, int num_sms, int ctas_per_sm) {
  // the FP64 pipe of an SM is shared by its CTAs, so an SM takes as long as its number of CTAs: from four
  // CTAs an SM to six rounds of resident ones, the count that leaves the SMs and the chunks of a split most
  // even (16.1 CTAs an SM and 9.7 chunks a split ran 6.47 ms on CH4's radial plot, 32 and 3 run 6.29)
  const double sms = num_sms;
  const int64_t most = std::min<int64_t>(std::min<int64_t>(nchunks, 4096),
                                         static_cast<int64_t>(6 * sms * ctas_per_sm) / std::max<int64_t>(tiles, 1));
  const int64_t least = std::min<int64_t>(most, static_cast<int64_t>(4 * sms) / std::max<int64_t>(tiles, 1));
  int64_t best = std::max<int64_t>(least, 1);
  double best_share = 0.0;
  for (int64_t s = best; s <= most; ++s) {
    const double ctas = static_cast<double>(tiles * s) / sms, chunks = static_cast<double>(nchunks) / s;
    const double share = ctas / std::ceil(ctas) * (chunks / std::ceil(chunks));
    if (share > 1.005 * best_share) {
      best = s;
      best_share = share;
    }
  }
  return static_cast<int>(best);
}

// The large table of exp2_neg64 (2^(j/2048); every fourth entry is the small one), uploaded once per context.
int ensure_exp64_table(inca_ctx* c) {
  if (c->d_exp64tab.n != 0) return INCA_OK;
  std::vector<double> t(kExp64TabLarge);
  for (int j = 0; j < kExp64TabLarge; ++j) t[j] = std::exp2(double(j) / kExp64TabLarge);
  if (c->d_exp64tab.reserve(kExp64TabLarge)) return set_error(c, INCA_E_NOMEM, "exp table");
  INCA_CUDA(c, cudaMemcpy(c->d_exp64tab.p, t.data(), sizeof(double) * t.size(), cudaMemcpyHostToDevice));
  return INCA_OK;
}

int ensure_events(inca_ctx* c) {
  for (auto& e : c->ev)
    if (!e) INCA_CUDA(c, cudaEventCreate(&e));
  return INCA_OK;
}

int eval_device(inca_ctx* c, int mode, double tol, bool graph) {
  if (!c->prepared) return set_error(c, INCA_E_STATE, "inca_eval: call inca_prepare first");
  if (c->grid_kind == GRID_NONE || c->ngrid <= 0) return set_error(c, INCA_E_STATE, "inca_eval: no grid");
  if (c->batch_molecules > 0 && c->batch_grid_version != c->grid_version)
    return set_error(c, INCA_E_STATE, "inca_eval: the batch's grid was replaced; prepare the batch again");
  if (c->d_ivec.reserve(c->ngrid)) return set_error(c, INCA_E_NOMEM, "ivec");
  c->t_total_ms = c->t_kernel_ms = c->t_pass2_ms = 0;
  c->t_kernel_launches = c->t_launches = 0;
  c->pairs_fp32 = c->pairs_fp64 = c->pairs_skip = c->corrected_points = c->pairs_cheap = 0;
  if (mode == INCA_MIXED) {
    const int st = graph ? eval_mixed_graph(c, tol > 0 ? tol : 1e-10) : eval_mixed(c, tol > 0 ? tol : 1e-10);
    if (st == INCA_OK) c->evaluated = true;
    return st;
  }
  if (mode == INCA_FP64_SCREENED && !cube_separable(c)) {
    bool plain = false;
    const int st = eval_fp64_screened(c, tol > 0 ? tol : 1e-10, &plain);
    if (st != INCA_OK) return st;
    if (!plain) {
      c->evaluated = true;
      return INCA_OK;
    }
  } else if (mode != INCA_FP64 && mode != INCA_FP64_SCREENED) {
    return set_error(c, INCA_E_ARG, "inca_eval: unknown mode");
  }
  const int64_t ngrid = c->ngrid;
  const int nchunks = static_cast<int>(c->chunks.size());
  int st64 = ensure_exp64_table(c);
  if (st64) return st64;
  if ((st64 = ensure_events(c))) return st64;
  const cudaEvent_t e0 = c->ev[0], e1 = c->ev[1], e2 = c->ev[2];
  if (nchunks == 0) {
    INCA_CUDA(c, cudaMemsetAsync(c->d_ivec.p, 0, sizeof(double) * ngrid, c->stream));
    INCA_CUDA(c, cudaStreamSynchronize(c->stream));
    c->evaluated = true;
    return INCA_OK;
  }
  size_t smem = 0;
  for (const ClassSeg& sg : c->classes) smem = std::max(smem, sizeof(double) * sg.per_chunk * sg.stride);
  // one launch pair per molecule of a batch (each molecule's points against its own chunks)
  const int nmol = c->batch_molecules > 0 ? c->batch_molecules : 1;
  INCA_CUDA(c, cudaEventRecord(e0, c->stream));
  int launches = 0;
  for (int m = 0; m < nmol; ++m) {
    const int64_t p0 = c->batch_molecules > 0 ? c->h_mol_off[m] : 0;
    const int64_t np = c->batch_molecules > 0 ? c->h_mol_off[m + 1] - p0 : ngrid;
    const int cb = c->mol_chunks[m].begin, nch = c->mol_chunks[m].end - c->mol_chunks[m].begin;
    if (np == 0) continue;
    if (nch <= 0) {
      INCA_CUDA(c, cudaMemsetAsync(c->d_ivec.p + p0, 0, sizeof(double) * np, c->stream));
      continue;
    }
    const int64_t tiles = (np + kTile64 - 1) / kTile64;
    const bool few = np <= kFewPoints;
    const int nsplit = few ? std::min(nch, kFewSplits) : choose_splits(tiles, nch, c->num_sms, kCtas64);
    if (c->d_partial.reserve(static_cast<size_t>(nsplit) * np)) return set_error(c, INCA_E_NOMEM, "partials");
    if (few) {
      constexpr int per = kThreads64 / 32;
      INCA_LAUNCH(c, k_eval_fp64_few, static_cast<unsigned>((nsplit + per - 1) / per), kThreads64, 0, c->d_chunks.p + cb,
                  nch, c->d_classes.p, c->d_rec64.p, c->d_px.p + p0, c->d_py.p + p0, c->d_pz.p + p0,
                  static_cast<int>(np), nsplit, c->d_exp64tab.p, c->d_partial.p);
    } else {
      dim3 grid(static_cast<unsigned>(tiles), static_cast<unsigned>(nsplit));
      INCA_LAUNCH(c, k_eval_fp64, grid, kThreads64, smem, c->d_chunks.p + cb, nch, c->d_classes.p, c->d_rec64.p,
                  c->d_px.p + p0, c->d_py.p + p0, c->d_pz.p + p0, np, nsplit, c->d_exp64tab.p, c->d_partial.p);
    }
    INCA_CUDA(c, cudaGetLastError());
    INCA_LAUNCH(c, k_reduce_splits, static_cast<unsigned>((np + 15) / 16), 256, 0, c->d_partial.p, nsplit, np,
                c->d_ivec.p + p0);
    INCA_CUDA(c, cudaGetLastError());
    launches += 2;
  }
  INCA_CUDA(c, cudaEventRecord(e1, c->stream));
  INCA_CUDA(c, cudaEventRecord(e2, c->stream));
  INCA_CUDA(c, cudaEventSynchronize(e2));
  float a = 0, b = 0;
  cudaEventElapsedTime(&a, e0, e1);
  cudaEventElapsedTime(&b, e0, e2);
  c->t_kernel_ms = a;
  c->t_total_ms = b;
  c->t_kernel_launches = launches / 2;
  c->t_launches = launches;
  c->evaluated = true;
  return INCA_OK;
}

}  // namespace inca
