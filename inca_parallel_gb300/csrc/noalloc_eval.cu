// FP64 evaluation of the intracule (the point loop of src/mod_intracule.f90:345-358) from
// caller-owned device records into a caller-owned device output, allocating nothing.
//
// The context API (inca_eval) grows its own device buffers with cudaMalloc. Some callers
// cannot allow that: code running inside a caller-managed memory pool or arena, or a service
// that must not allocate after start-up so that it cannot run out of memory later. This entry
// point takes every input and output from the caller and keeps its only intermediate (the
// per-split partial sums) in a fixed file-scope device array.
//
// Work decomposition: a CTA owns 256 points (2 per thread; 128, 1 per thread, for up to 128 points) and
// one contiguous range of records (its split); it writes one partial per point into the fixed scratch
// array, and a second kernel adds the splits of each point in split order, so a call is deterministic.
//
// FP64 issue bounds it, and two thirds of a record's FP64 instructions are its Gaussian, which the
// quartets of the same four shells share (3.8 of them on CH4, side by side in no order that a caller is
// likely to have). So calls with enough work sort an index of the records by a hash of exponent and
// centre first (in blocks of kSortMax records, in fixed device arrays like the scratch; the sort is
// stable and the sum's order fixed), and a thread evaluates a Gaussian once per run of equal ones. CH4,
// 111 080 records at 1 777 points: 12.3 ms in the caller's order, 4.6 ms sorted, of it 0.06 for the sort.
//
// Every scratch element a call reads was written earlier in the same call: nothing has to
// be cleared beforehand. Calls that overlap in time on one device (two streams, two host
// threads) share the scratch arrays and race.
#include <algorithm>
#include <mutex>

#include <cub/device/device_radix_sort.cuh>
#include <cuda.h>  // driver API types only: the two functions used are resolved at run time

#include "exp2_table.h"
#include "exp64.cuh"
#include "inca_internal.h"

// Scratch capacity: splits x points <= INCA_NOALLOC_MAX_POINTS doubles (16 MiB).
static __device__ __align__(256) double g_noalloc_scratch[INCA_NOALLOC_MAX_POINTS];
// The sort of one block of records: two buffers of keys, two of indices, and the sort's own storage.
constexpr int kSortMax = 1 << 19;
constexpr int kSortBits = 24;  // of the hash: 30 000 Gaussians meet in 2^24 values 27 times
constexpr size_t kSortStorage = 1 << 20;
static __device__ __align__(256) uint32_t g_noalloc_keys[2 * kSortMax];
static __device__ __align__(256) uint32_t g_noalloc_index[2 * kSortMax];
static __device__ __align__(256) unsigned char g_noalloc_sort[kSortStorage];

namespace {

constexpr int kThreads = 128, kCtasPerSm = 8;
// Records x points from which on the records are sorted: 60 us of sorting against 1.9 ms of evaluation
// in the caller's order, and against half of that where the records share their Gaussians as CH4's do.
constexpr double kSortWork = 3.4e7;
constexpr int kMaxDevices = 256;
constexpr int kCoef = INCA_MAX_DEGREE + 1;

// Per-device set-up, done with that device current, once per CUDA context: the scratch
// array's address belongs to the context that loaded the module, so a context created anew
// on the device (after cudaDeviceReset, or a caller's own context) is set up again.
struct DeviceSlot {
  bool ready = false;
  unsigned long long ctx_id = 0;
  double* scratch = nullptr;
  uint32_t *keys = nullptr, *index = nullptr;
  unsigned char* sort = nullptr;
  int num_sms = 0;
  bool sorted_once = false;  // the sort's kernels are loaded
};
std::mutex g_setup_mutex;
DeviceSlot g_slots[kMaxDevices];

using PfnCtxGetCurrent = CUresult (*)(CUcontext*);
using PfnCtxGetId = CUresult (*)(CUcontext, unsigned long long*);
PfnCtxGetCurrent g_ctx_get_current = nullptr;
PfnCtxGetId g_ctx_get_id = nullptr;

// Sort key (a hash of exponent and centre) and index of each record.
__global__ void k_record_hash(int n, const double* __restrict__ sqe, const double* __restrict__ d, uint32_t* key,
                              uint32_t* index) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  unsigned long long h = 0;
  const double v[4] = {sqe[q], d[3LL * q], d[3LL * q + 1], d[3LL * q + 2]};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    h = (h ^ static_cast<unsigned long long>(__double_as_longlong(v[k]))) * 0x9E3779B97F4A7C15ull;
    h ^= h >> 29;
  }
  key[q] = static_cast<uint32_t>(h >> (64 - kSortBits));
  index[q] = static_cast<uint32_t>(q);
}

// order (may be null: the caller's): the records' places
template <int kPPT>
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
k_eval_records(int64_t nrec, int64_t per_split, const uint32_t* __restrict__ order, const double* __restrict__ A,
               const double* __restrict__ sqe, const double* __restrict__ d,
               const int32_t* __restrict__ L, const double* __restrict__ C, int64_t npts,
               const double* __restrict__ r, double* __restrict__ partial) {
  __shared__ double tab[inca::kExp64Tab];
  const int tid = threadIdx.x;
  for (int i = tid; i < inca::kExp64Tab; i += kThreads) tab[i] = inca::kExp2Table[i];
  __syncthreads();
  const int64_t base = static_cast<int64_t>(blockIdx.x) * (kThreads * kPPT);
  if (base + (tid & ~31) >= npts) return;  // none of the warp's points
  double x[3][kPPT], acc[kPPT], u[3][kPPT], e[kPPT], t[kPPT];
#pragma unroll
  for (int p = 0; p < kPPT; ++p) {
    const int64_t g = base + tid + p * kThreads;
    const bool ok = g < npts;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      x[k][p] = ok ? r[3 * g + k] : 0.0;
      u[k][p] = 0.0;
    }
    e[p] = acc[p] = t[p] = 0.0;
  }
  const int64_t q0 = static_cast<int64_t>(blockIdx.y) * per_split;
  const int64_t q1 = min(nrec, q0 + per_split);
  // Runs of records with the same exponent and centre: their Gaussian once, the sum of their
  // polynomials t, and acc += e t at the end. A factor of degree zero is a number of the record, which
  // goes into its amplitude; u_k = s (x_k + d_k) is formed when a record of the run needs it.
  // (Equal as bits: comparisons in FP64 would be four more instructions of the pipe that is short.)
  long long last[4] = {0, 0, 0, 0};
  int scaled = 0;
  for (int64_t at = q0; at < q1; ++at) {
    // (cut at the list's end: calls that race for the arrays get wrong sums, not reads out of range)
    const int64_t q = order ? min(static_cast<int64_t>(order[at]), nrec - 1) : at;
    const double s = sqe[q], dq[3] = {d[3 * q + 0], d[3 * q + 1], d[3 * q + 2]};
    const long long now[4] = {__double_as_longlong(s), __double_as_longlong(dq[0]), __double_as_longlong(dq[1]),
                              __double_as_longlong(dq[2])};
    double a = A[q];
    if (at == q0 || ((now[0] ^ last[0]) | (now[1] ^ last[1]) | (now[2] ^ last[2]) | (now[3] ^ last[3])) != 0) {
      const double s2 = (s * 1.4426950408889634) * s;  // e^-y = 2^-(y / ln 2)
      scaled = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) last[k] = now[k];
#pragma unroll
      for (int p = 0; p < kPPT; ++p) {
        acc[p] = inca::add_term64(e[p], t[p], acc[p]);
        t[p] = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) u[k][p] = x[k][p] + dq[k];
        e[p] = inca::exp2_neg64(s2, fma(u[2][p], u[2][p], fma(u[1][p], u[1][p], u[0][p] * u[0][p])), tab);
      }
    }
    const double* Cq = C + 3 * q * kCoef;  // highest degree first
    // degrees outside 0..INCA_MAX_DEGREE are clamped so that reads stay inside the record
    int Lq[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      Lq[k] = min(max(L[3 * q + k], 0), INCA_MAX_DEGREE);
      if (Lq[k] == 0) a *= Cq[k * kCoef];
    }
    double v[kPPT];
#pragma unroll
    for (int p = 0; p < kPPT; ++p) v[p] = a;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (Lq[k] > 0) {
        if (!(scaled >> k & 1)) {
          scaled |= 1 << k;
#pragma unroll
          for (int p = 0; p < kPPT; ++p) u[k][p] *= s;
        }
        double w[kPPT];
        const double c0 = Cq[k * kCoef], c1 = Cq[k * kCoef + 1];
#pragma unroll
        for (int p = 0; p < kPPT; ++p) w[p] = fma(c0, u[k][p], c1);
        for (int m = 2; m <= Lq[k]; ++m) {
          const double c = Cq[k * kCoef + m];
#pragma unroll
          for (int p = 0; p < kPPT; ++p) w[p] = fma(w[p], u[k][p], c);
        }
#pragma unroll
        for (int p = 0; p < kPPT; ++p) v[p] *= w[p];
      }
#pragma unroll
    for (int p = 0; p < kPPT; ++p) t[p] += v[p];
  }
#pragma unroll
  for (int p = 0; p < kPPT; ++p) acc[p] = inca::add_term64(e[p], t[p], acc[p]);
#pragma unroll
  for (int p = 0; p < kPPT; ++p) {
    const int64_t g = base + tid + p * kThreads;
    if (g < npts) partial[static_cast<int64_t>(blockIdx.y) * npts + g] = acc[p];
  }
}

// Sums over the splits of each point in a fixed order (add: onto what out holds), a block of 16 x 16 threads per 16 points.
__global__ void __launch_bounds__(256)
k_sum_record_splits(const double* __restrict__ partial, int nsplit, int64_t npts, int add, double* __restrict__ out) {
  __shared__ double sh[16][17];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t g = blockIdx.x * 16LL + tx;
  double s = 0.0;
  if (g < npts)
    for (int k = ty; k < nsplit; k += 16) s += partial[static_cast<int64_t>(k) * npts + g];
  sh[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && g < npts) {
    double t = sh[0][tx];
#pragma unroll
    for (int r = 1; r < 16; ++r) t += sh[r][tx];
    out[g] = add ? out[g] + t : t;
  }
}

// Id of the calling thread's current CUDA context (0: none is current yet). Ids are unique
// for the life of the process, so a context created after a reset has a new one.
int current_ctx_id(unsigned long long* id) {
  if (!g_ctx_get_current || !g_ctx_get_id) {
    void* f1 = nullptr;
    void* f2 = nullptr;
    cudaDriverEntryPointQueryResult q1, q2;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1) != cudaSuccess ||
        cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2) != cudaSuccess ||
        q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess || !f1 || !f2)
      return INCA_E_CUDA;
    g_ctx_get_current = reinterpret_cast<PfnCtxGetCurrent>(f1);
    g_ctx_get_id = reinterpret_cast<PfnCtxGetId>(f2);
  }
  CUcontext c = nullptr;
  if (g_ctx_get_current(&c) != CUDA_SUCCESS) return INCA_E_CUDA;
  *id = 0;
  if (c && g_ctx_get_id(c, id) != CUDA_SUCCESS) return INCA_E_CUDA;
  return INCA_OK;
}

cudaError_t sort_index(const DeviceSlot& slot, int n, cudaStream_t s, const uint32_t** order) {
  cub::DoubleBuffer<uint32_t> keys(slot.keys, slot.keys + kSortMax), index(slot.index, slot.index + kSortMax);
  size_t bytes = 0;
  cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, bytes, keys, index, n, 0, kSortBits, s);
  if (e != cudaSuccess || bytes > kSortStorage) return e;  // (0.2 MB for a full block; else the caller's order)
  e = cub::DeviceRadixSort::SortPairs(slot.sort, bytes, keys, index, n, 0, kSortBits, s);
  if (e == cudaSuccess) *order = index.Current();
  return e;
}

// Loads every kernel that a later call may launch. Code is loaded at its first use, which can take device
// memory: a large call after a small one would allocate. The sort's kernels have no names to ask for: one
// item and more than a block of them, in the fixed arrays, are sorted on the first call that is not captured.
cudaError_t load_kernels() {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, k_eval_records<1>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_eval_records<2>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_record_hash);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_sum_record_splits);
  return e;
}
cudaError_t load_sort(const DeviceSlot& slot, cudaStream_t s) {
  const uint32_t* order = nullptr;
  const cudaError_t e = sort_index(slot, 1, s, &order);
  return e == cudaSuccess ? sort_index(slot, 1 << 16, s, &order) : e;
}

// Set-up of a device for the current context: resolve the scratch array's address and the
// SM count, load the kernels (first call on the device, and again whenever the current context has changed).
int device_setup(int dev, cudaStream_t stream, DeviceSlot* out) {
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  unsigned long long id = 0;
  int st = current_ctx_id(&id);
  if (st != INCA_OK) return st;
  DeviceSlot& s = g_slots[dev];
  if (!s.ready || id == 0 || s.ctx_id != id) {
    void* p = nullptr;
    // with no context current yet, this call also initialises the device's primary context
    void *keys = nullptr, *index = nullptr, *sort = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess ||
        cudaGetSymbolAddress(&keys, g_noalloc_keys) != cudaSuccess ||
        cudaGetSymbolAddress(&index, g_noalloc_index) != cudaSuccess ||
        cudaGetSymbolAddress(&sort, g_noalloc_sort) != cudaSuccess)
      return INCA_E_CUDA;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      return INCA_E_CUDA;
    if (id == 0 && ((st = current_ctx_id(&id)) != INCA_OK || id == 0)) return st != INCA_OK ? st : INCA_E_CUDA;
    s.scratch = static_cast<double*>(p);
    s.keys = static_cast<uint32_t*>(keys);
    s.index = static_cast<uint32_t*>(index);
    s.sort = static_cast<unsigned char*>(sort);
    s.num_sms = sms;
    if (load_kernels() != cudaSuccess) return INCA_E_CUDA;
    s.ctx_id = id;
    s.ready = true;
    s.sorted_once = false;
  }
  if (!s.sorted_once) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess) return INCA_E_CUDA;
    if (capture == cudaStreamCaptureStatusNone) {
      if (load_sort(s, stream) != cudaSuccess) return INCA_E_CUDA;
      s.sorted_once = true;
    }
  }
  *out = s;
  return INCA_OK;
}

}  // namespace

extern "C" int inca_eval_records_noalloc(int64_t nrec, const double* A, const double* sqe,
                                         const double* d, const int32_t* L, const double* C,
                                         int64_t npts, const double* r, double* ivec,
                                         void* stream) {
  if (nrec < 0 || npts < 0) return INCA_E_ARG;
  if (npts > INCA_NOALLOC_MAX_POINTS) return INCA_E_LIMIT;
  if (npts == 0) return INCA_OK;
  if (!r || !ivec || (nrec > 0 && (!A || !sqe || !d || !L || !C))) return INCA_E_ARG;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return INCA_E_CUDA;
  if (dev < 0 || dev >= kMaxDevices) return INCA_E_LIMIT;
  // an error left pending by the caller's own work is reported, not cleared, and nothing is
  // queued (otherwise the launch checks below would take it for a failure of this call)
  if (cudaPeekAtLastError() != cudaSuccess) return INCA_E_CUDA;
  DeviceSlot slot;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int st = device_setup(dev, s, &slot);
  if (st != INCA_OK) return st;
  if (nrec == 0) {
    return cudaMemsetAsync(ivec, 0, sizeof(double) * npts, s) == cudaSuccess ? INCA_OK : INCA_E_CUDA;
  }
  const bool sorted = static_cast<double>(nrec) * static_cast<double>(npts) >= kSortWork;
  const int ppt = npts <= kThreads ? 1 : 2;
  const int64_t tiles = (npts + kThreads * ppt - 1) / (kThreads * ppt);
  for (int64_t first = 0; first < nrec;) {
    // sorted: a block of records at a time
    const int64_t n = sorted ? std::min<int64_t>(nrec - first, kSortMax) : nrec;
    const double *bA = A + first, *bs = sqe + first, *bd = d + 3 * first, *bC = C + 3 * first * kCoef;
    const int32_t* bL = L + 3 * first;
    const uint32_t* order = nullptr;
    if (sorted) {
      const int m = static_cast<int>(n);
      k_record_hash<<<(m + 255) / 256, 256, 0, s>>>(m, bs, bd, slot.keys, slot.index);
      if (cudaGetLastError() != cudaSuccess) return INCA_E_CUDA;
      if (sort_index(slot, m, s, &order) != cudaSuccess) return INCA_E_CUDA;
    }
    // Splits: (tiles x splits) CTAs that fill the GPU at most four times over (rounded down: four
    // CTAs more than two rounds took a third one), bounded by the number of record groups of 32 and
    // by the scratch capacity.
    const int64_t target = static_cast<int64_t>(slot.num_sms) * kCtasPerSm * 4;
    int64_t nsplit = target / tiles;
    nsplit = std::min<int64_t>(nsplit, (n + 31) / 32);
    nsplit = std::min<int64_t>(nsplit, INCA_NOALLOC_MAX_POINTS / npts);
    nsplit = std::max<int64_t>(std::min<int64_t>(nsplit, 4096), 1);
    const int64_t per_split = (n + nsplit - 1) / nsplit;
    dim3 grid(static_cast<unsigned>(tiles), static_cast<unsigned>(nsplit));
    if (ppt == 1)
      k_eval_records<1><<<grid, kThreads, 0, s>>>(n, per_split, order, bA, bs, bd, bL, bC, npts, r, slot.scratch);
    else
      k_eval_records<2><<<grid, kThreads, 0, s>>>(n, per_split, order, bA, bs, bd, bL, bC, npts, r, slot.scratch);
    if (cudaGetLastError() != cudaSuccess) return INCA_E_CUDA;
    k_sum_record_splits<<<static_cast<unsigned>((npts + 15) / 16), 256, 0, s>>>(
        slot.scratch, static_cast<int>(nsplit), npts, first > 0 ? 1 : 0, ivec);
    if (cudaGetLastError() != cudaSuccess) return INCA_E_CUDA;
    first += n;
  }
  return INCA_OK;
}
