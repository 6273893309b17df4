// Device helpers shared by the FP32-pipe evaluation kernels (mixed_eval.cu, cube_eval.cu):
// double-buffered staging of quartet-record chunks into shared memory by 1-D TMA bulk copies
// (cp.async.bulk + mbarrier, every wait bounded), the persistent work counter, and
// double-float (hi + lo FP32 pair, ~2^-44 relative) arithmetic with its exp2.
// Explicit round-to-nearest intrinsics only: results do not depend on FMA contraction.
#pragma once
#include <cstdint>

#include "inca_internal.h"

namespace inca {
namespace {

constexpr int kExpTab = 256;         // 2^(j/256), j = 0..255 (double-float exp2 table)
constexpr int kWaitLimit = 1 << 22;  // bounded mbarrier waits
// |u_d| limit for the polynomial factors: 2^(-u^2 + ks) is zero beyond sqrt(126 + ks) < 64
// for every representable A' scale ks used here, and 64^16 stays finite in FP32
constexpr float kUClamp = 64.0f;

// ---------------------------------------------------------------- TMA bulk staging
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// One thread: expect `bytes` on the barrier and start the bulk copy global -> shared.
// Requires 16-byte aligned addresses and a size that is a multiple of 16.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// Bounded wait for the barrier phase with the given parity; false if the limit ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int limit = kWaitLimit) {
  for (int it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

struct ChunkRef {
  const float* src;
  uint32_t bytes;
};
__device__ __forceinline__ ChunkRef chunk_ref(const WorkChunk* chunks, const ClassSeg* segs, const float* rec32,
                                              int ch) {
  const WorkChunk w = chunks[ch];
  const ClassSeg sg = segs[w.cls];
  return {rec32 + sg.off32 + (w.rec - sg.first) * sg.stride32,
          static_cast<uint32_t>(w.count * sg.stride32 * sizeof(float))};
}

// Shared-memory stage of a warp-CTA (dynamic shared memory): two barriers, then two chunk
// buffers of `floats` floats each (the largest chunk present).
// Buffer k & 1 is addressed by arithmetic on the shared-memory base (not by indexing an array of
// pointers, which the compiler keeps in local memory): the record reads stay shared-memory loads.
struct Stage {
  uint64_t* bar;
  float* buf0;
  int floats;
  __device__ __forceinline__ float* buf(int k) const { return buf0 + (k & 1) * floats; }
};
__device__ __forceinline__ Stage stage_view(unsigned char* dsm, int floats) {
  Stage S;
  S.bar = reinterpret_cast<uint64_t*>(dsm);
  S.buf0 = reinterpret_cast<float*>(dsm + 128);
  S.floats = floats;
  return S;
}

// Set up the two barriers (once per CTA; they then serve every work item of the CTA).
__device__ __forceinline__ void stage_init(const Stage& S) {
  if (threadIdx.x == 0) {
    mbar_init(&S.bar[0]);
    mbar_init(&S.bar[1]);
    fence_mbar_init();
  }
  __syncwarp();
}

// Start the copy of an item's first chunk (global chunk counter k) into buffer k & 1.
// issue = false (test of the bounded waits only): no copy is started, so the wait on that
// buffer runs out.
__device__ __forceinline__ void stage_first(const Stage& S, const WorkChunk* chunks, const ClassSeg* segs,
                                            const float* rec32, int k, int ch, bool issue = true) {
  if (threadIdx.x == 0 && issue) {
    fence_proxy_async();  // earlier generic-proxy reads of that buffer are done (warp-synchronous)
    const ChunkRef r = chunk_ref(chunks, segs, rec32, ch);
    bulk_load(S.buf(k), r.src, r.bytes, &S.bar[k & 1]);
  }
}

// The molecule owning a work item / sorted point / tile: the last entry whose start is <= x
// (molecules without work share their start with the next one and are never returned).
__device__ __forceinline__ int mol_of_item(const MolWork* __restrict__ mw, int nmol, int64_t x) {
  int lo = 0, hi = nmol - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (mw[mid].item0 <= x) lo = mid; else hi = mid - 1;
  }
  return lo;
}
__device__ __forceinline__ int mol_of_point(const MolWork* __restrict__ mw, int nmol, int64_t x) {
  int lo = 0, hi = nmol - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (mw[mid].p0 <= x) lo = mid; else hi = mid - 1;
  }
  return lo;
}
__device__ __forceinline__ int mol_of_tile(const MolWork* __restrict__ mw, int nmol, int64_t x) {
  int lo = 0, hi = nmol - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (mw[mid].tile0 <= x) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Next work item of a persistent CTA: (tile, split) pairs, taken from a device counter.
__device__ __forceinline__ int64_t next_item(unsigned long long* work) {
  unsigned long long it = 0;
  if (threadIdx.x == 0) it = atomicAdd(work, 1ull);
  return static_cast<int64_t>(__shfl_sync(0xffffffffu, it, 0));
}

// Before working on chunk k: start the copy of the next chunk into the other buffer, then wait
// for this one. Returns false if the wait gave up; the other buffer's copy (if started) is then
// drained, again with a bounded wait, so no copy is left in flight when the CTA exits.
// limit / issue: the wait limit, and whether copies are started (see stage_first).
__device__ __forceinline__ bool stage_next(const Stage& S, const WorkChunk* chunks, const ClassSeg* segs,
                                           const float* rec32, int k, int next, int nchunks,
                                           int limit = kWaitLimit, bool issue = true) {
  if (threadIdx.x == 0 && next < nchunks && issue) {
    fence_proxy_async();  // the generic-proxy reads of that buffer (chunk k-1) are done
    const ChunkRef r = chunk_ref(chunks, segs, rec32, next);
    bulk_load(S.buf(k + 1), r.src, r.bytes, &S.bar[(k + 1) & 1]);
  }
  if (mbar_wait(&S.bar[k & 1], static_cast<uint32_t>((k >> 1) & 1), limit)) return true;
  if (next < nchunks) mbar_wait(&S.bar[(k + 1) & 1], static_cast<uint32_t>(((k + 1) >> 1) & 1), limit);
  return false;
}

// ---------------------------------------------------------------- double-float arithmetic
struct f2 {
  float hi, lo;
};
__device__ __forceinline__ f2 two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return {s, e};
}
__device__ __forceinline__ f2 fast_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ f2 df_add(f2 x, f2 y) {
  const f2 s = two_sum(x.hi, y.hi);
  return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(x.lo, y.lo)));
}
__device__ __forceinline__ f2 df_mul(f2 x, f2 y) {
  const float p = __fmul_rn(x.hi, y.hi);
  float e = __fmaf_rn(x.hi, y.hi, -p);
  e = __fmaf_rn(x.hi, y.lo, e);
  e = __fmaf_rn(x.lo, y.hi, e);
  return fast_two_sum(p, e);
}
// The forms below leave their result as a sum hi + lo that is not renormalised: |lo| stays near
// 2^-22 of the operands, which is all that the next product or sum needs (the products of two low
// parts that are dropped are 2^-44 of it, and 2^-46 with an exponential). A renormalisation is three
// instructions each time.

// x y + z
__device__ __forceinline__ f2 df_fma_raw(f2 x, f2 y, f2 z) {
  const float p = __fmul_rn(x.hi, y.hi);
  float e = __fmaf_rn(x.hi, y.hi, -p);
  e = __fmaf_rn(x.hi, y.lo, e);
  e = __fmaf_rn(x.lo, y.hi, e);
  const f2 s = two_sum(p, z.hi);
  return {s.hi, __fadd_rn(s.lo, __fadd_rn(e, z.lo))};
}
__device__ __forceinline__ f2 df_mul_raw(f2 x, f2 y) {
  const float p = __fmul_rn(x.hi, y.hi);
  float e = __fmaf_rn(x.hi, y.hi, -p);
  e = __fmaf_rn(x.hi, y.lo, e);
  return {p, __fmaf_rn(x.lo, y.hi, e)};
}
// s x + b for a coordinate x = xh + xl, a scale and a shift. Renormalised: the split of a coordinate
// is up to 32 ulps off the nearest float, and a low part of 2^-19 would lose 2^-38 in each product.
__device__ __forceinline__ f2 df_coord(float s_hi, float s_lo, float b_hi, float b_lo, float xh, float xl) {
  const float p = __fmul_rn(s_hi, xh);
  float e = __fmaf_rn(s_hi, xh, -p);
  const f2 t = two_sum(p, b_hi);
  e = __fadd_rn(e, t.lo);
  e = __fmaf_rn(s_hi, xl, e);
  e = __fmaf_rn(s_lo, xh, e);
  return fast_two_sum(t.hi, __fadd_rn(e, b_lo));  // |e| << |t.hi| except near 0, where it is harmless
}
// x^2, the square of the low part included (near x = 0 the low part may rival the high one)
__device__ __forceinline__ f2 df_sqr_raw(f2 x) {
  const float p = __fmul_rn(x.hi, x.hi);
  const float e = __fmaf_rn(x.hi, x.hi, -p);
  return {p, __fmaf_rn(__fmaf_rn(2.0f, x.hi, x.lo), x.lo, e)};
}

// 2^(-y + ks) in double-float for y >= 0: -y = n + j/256 + g, |g| <= 1/512 (256 y rounded to an
// integer in the low mantissa bits, so n and j are its bits); 2^g = 1 + x + x^2/2 + x^3/6 + x^4/24 with
// x = g ln2 - y.lo ln2 in double-float; times 2^(j/256) from a table and 2^(n + ks) in the exponent (zero
// below 2^-126, and from y = 8000 on, where it is for every ks).
// Relative error 2.2e-14 rms up to y = 5 and 3.1e-14 up to 30 (400 000 random arguments, emulated), at
// most 2.8e-13. x^2/2, up to 2^-20, is kept with its rounding error and joins x before the table's
// product, so the result's low part is below 2^-24 of it. Added to the low parts in FP32 it left 3.4e-14 and
// 5.2e-14, and a product of two such factors lost their low parts' product, which has one sign (-9e-14 on
// lattices of positive terms; CH4 48^3 1.2e-13 from the FP64 form as a root mean square against 3.3e-14). 9
// instructions of a term's 120: 2 % on few points, 0.8 % on CH4's radial plot.
__device__ __forceinline__ f2 df_exp2_neg(f2 y, int ks, const float2* __restrict__ tab) {
  const float yc = fminf(y.hi, 8000.0f);
  const float t = __fmaf_rn(yc, -256.0f, 12582912.0f);  // 1.5 * 2^23
  const int m = __float_as_int(t) - 0x4B400000;
  const float g = -__fmaf_rn(__fsub_rn(t, 12582912.0f), 0.00390625f, yc);  // exact
  const float kLn2Hi = 0.693147182464599609375f, kLn2Lo = -1.904654323148236e-09f;
  const float xh = __fmul_rn(g, kLn2Hi);
  float zl = __fmaf_rn(g, kLn2Hi, -xh);
  zl = __fmaf_rn(g, kLn2Lo, zl);
  zl = __fmaf_rn(y.lo, -kLn2Hi, zl);
  const f2 x = fast_two_sum(xh, zl);  // zl holds y.lo too: its square counts
  const float hx = __fmul_rn(0.5f, x.hi), w = __fmul_rn(hx, x.hi);
  float we = __fmaf_rn(hx, x.hi, -w);
  we = __fmaf_rn(__fmul_rn(x.hi, w), __fmaf_rn(x.hi, 0.083333333333333333f, 0.33333333333333333f), we);
  const f2 z = fast_two_sum(x.hi, w);
  zl = __fadd_rn(z.lo, __fadd_rn(x.lo, we));
  const float2 T = tab[m & (kExpTab - 1)];
  const float p = __fmul_rn(T.x, z.hi);
  const float pe = __fmaf_rn(T.x, z.hi, -p);
  const f2 s = fast_two_sum(T.x, p);
  float lo = __fadd_rn(s.lo, __fmaf_rn(T.y, z.hi, __fadd_rn(T.y, pe)));
  lo = __fmaf_rn(T.x, zl, lo);
  const int e = min(max((m >> 8) + ks + 127, 0), 254);
  const float sc = __int_as_float(e << 23);  // 2^(n + ks)
  const bool on = y.hi < 8000.0f;  // beyond it the low part may not be finite
  return {on ? __fmul_rn(s.hi, sc) : 0.0f, on ? __fmul_rn(lo, sc) : 0.0f};
}

// The unpacked shape of a record's polynomial (ClassSeg::shape). total: the total degree (of a product
// record the sum of its three degrees, which L holds).
struct Shape {
  int L[3];
  int total, nc;
  bool merged;
};
__device__ __forceinline__ Shape unpack(int shape, int nc) {
  Shape g;
  g.L[0] = shape & 31;
  g.L[1] = (shape >> 5) & 31;
  g.L[2] = (shape >> 10) & 31;
  g.merged = (shape & kMergedBit) != 0;
  g.total = g.merged ? (shape >> 15) & 31 : g.L[0] + g.L[1] + g.L[2];
  g.nc = nc;
  return g;
}
// The class's shape in uniform registers: it passes through a warp reduction, whose result is
// warp-uniform by construction, so the degree tests and Horner loops of every term are uniform
// branches (no reconvergence bookkeeping) and their counters leave the vector pipes.
__device__ __forceinline__ Shape uniform_shape(const ClassSeg& sg) {
  return unpack(__reduce_max_sync(0xffffffffu, sg.shape), __reduce_max_sync(0xffffffffu, sg.nc));
}

// sum_k S_k rho^k of a merged record (S highest degree first, after both coefficient sets).
__device__ __forceinline__ float merged_majorant(const float* __restrict__ R, const Shape& g, float rho) {
  const float* S = R + 12 + 2 * g.nc;
  float s = S[0];
#pragma unroll 1
  for (int k = 1; k <= g.total; ++k) s = __fmaf_rn(s, rho, S[k]);
  return s;
}

// log2 upper bound of a record's term over a box lo[3], hi[3] of points, from its FP32 record
// (u = s (r + d), E = 2^(-|u|^2 + ks)), with m_d / M_d the smallest / largest |u_d| over the box,
// widened by a relative and absolute 1e-5:
//  * merged: 2^ks sum_k S_k max(1, |M|)^k 2^-|m|^2, |M| cut at kUClamp (E is zero beyond it);
//  * product: la + sum_d [L_d log2 max(1, M_d) - m_d^2], la = log2(|A'| prod_d sum_k |Cn_dk|).
// *lerr gets the log2 bound of the FP32 error bound e over the box and *umax the largest M_d.
// Explicit round-to-nearest intrinsics: kernels that take the same decision see the same bits.
__device__ __forceinline__ float log2_bound(const float* __restrict__ R, const Shape& g, const float* box,
                                           float* lerr = nullptr, float* umax = nullptr) {
  float lb = __fadd_rn(R[10], 0.02f);
  float y2 = 0.0f, mm = 0.0f, m2 = 0.0f;
  const float s = R[0];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float b = R[2 + d];
    const float a0 = __fmaf_rn(s, box[d], b), a1 = __fmaf_rn(s, box[3 + d], b);
    float m = (a0 <= 0.0f && a1 >= 0.0f) ? 0.0f : fminf(fabsf(a0), fabsf(a1));
    float M = fmaxf(fabsf(a0), fabsf(a1));
    m = fmaxf(0.0f, __fsub_rn(__fmul_rn(m, 1.0f - 1e-5f), 1e-5f));
    M = __fadd_rn(__fmul_rn(M, 1.0f + 1e-5f), 1e-5f);
    if (!g.merged) lb = __fmaf_rn(static_cast<float>(g.L[d]), __log2f(fmaxf(M, 1.0f)), lb);
    m2 = __fmaf_rn(m, m, m2);
    y2 = __fmaf_rn(M, M, y2);
    mm = fmaxf(mm, M);
  }
  if (g.merged) {
    const float rho = fminf(fmaxf(__fsqrt_rn(y2), 1.0f), kUClamp);
    lb = __fadd_rn(lb, __log2f(merged_majorant(R, g, rho)));
  }
  lb = __fsub_rn(lb, __fmul_rn(m2, 1.0f - 1e-6f));
  if (umax) *umax = mm;
  if (lerr)
    *lerr = __fadd_rn(__fadd_rn(lb, __log2f(__fmaf_rn(3.0f, y2, static_cast<float>(10 + 2 * g.total)))), 0.02f - 24.0f);
  return lb;
}

// The chunks of a work item (every nsplit-th from `first`) that may hold a record with a term above
// 2^thr over the tile box, in order. Each lane bounds one of the next 32 chunks with the form of
// log2_bound over the chunk's own ranges (a record's bound is never above its chunk's), so chunks that
// are left out whole cost neither their staging nor a bound per record. With the records of a class
// sorted by centre and reach this takes 8 % off a 66-primitive molecule's evaluation (1.67 to 1.54 ms), 13 %
// off 100 primitives (14.6 to 12.7 ms); where every chunk is live it costs 1 %. What is left out is
// counted: quartets in `skipped`, the sum of the bounds in `mass`.
constexpr int kNoChunk = 0x7FFFFFFF;
struct ChunkWalk {
  const ChunkBound* bounds;
  int base, end, nsplit;
  uint32_t mask;
  int block;  // chunk of mask bit 0
  __device__ __forceinline__ ChunkWalk(const ChunkBound* b, int first, int last, int step)
      : bounds(b), base(first), end(last), nsplit(step), mask(0u), block(first) {}
  // errthr: also stop at chunks that may hold a record whose error bound is above 2^errthr
  __device__ __forceinline__ int next(const float* box, float thr, float& mass, unsigned long long& skipped,
                                      float errthr = HUGE_VALF) {
    while (mask == 0u) {
      if (base >= end) return kNoChunk;
      const int64_t ch = base + static_cast<int64_t>(threadIdx.x & 31) * nsplit;
      bool live = false;
      if (ch < end) {
        const ChunkBound B = bounds[ch];
        float m2 = 0.0f, M2 = 0.0f;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const float lo = __fadd_rn(box[d], B.dlo[d]), hi = __fadd_rn(box[3 + d], B.dhi[d]);
          const float m = (lo <= 0.0f && hi >= 0.0f) ? 0.0f : fminf(fabsf(lo), fabsf(hi));
          const float M = fmaxf(fabsf(lo), fabsf(hi));
          m2 = __fmaf_rn(m, m, m2);
          M2 = __fmaf_rn(M, M, M2);
        }
        const float m = fmaxf(0.0f, __fsub_rn(__fmul_rn(__fmul_rn(B.smin, __fsqrt_rn(m2)), 1.0f - 5e-5f), 5e-5f));
        const float M = __fadd_rn(__fmul_rn(__fmul_rn(B.smax, __fsqrt_rn(M2)), 1.0f + 5e-5f), 5e-5f);
        const float lb = __fsub_rn(__fmaf_rn(B.total, __log2f(fmaxf(M, 1.0f)), B.la), __fmul_rn(m, m));
        live = !(lb <= thr);
        if (errthr < HUGE_VALF)
          live |= !(lb + __log2f(__fmaf_rn(3.0f * M, M, 10.0f + 2.0f * B.total)) - 23.9f <= errthr);
        if (!live) {
          mass += static_cast<float>(B.records) * exp2f(lb);
          skipped += B.quartets;
        }
      }
      mask = __ballot_sync(0xffffffffu, live);
      block = base;
      base = static_cast<int>(min(static_cast<long long>(base) + 32LL * nsplit, static_cast<long long>(kNoChunk)));
    }
    const int b = __ffs(mask) - 1;
    mask &= mask - 1;
    return block + b * nsplit;
  }
};

}  // namespace
}  // namespace inca
