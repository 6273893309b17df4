// 2^-x for the FP64 evaluation kernels.
//
// FP64 instructions are what those kernels run out of (a GB300 SM issues two lanes a clock), so the
// exponential is spelled out: the argument is a product s w that the caller has not formed, rounded to
// a multiple of 1/kTab by one FMA into the low mantissa bits (m / kTab, |f| <= 1/(2 kTab) what is left,
// one more FMA and exact), 2^-f - 1 by a polynomial, 2^(-m/kTab) from a table and the exponent bits: where
// exp() takes about 16 FP64 instructions and the argument another 2, 8 with a table of 512 and the Taylor
// polynomial of degree 4 (remainder 1.2e-18), 7 with one of 2048 (16 KB, for kernels that load it once for
// many records) and degree 3, its f^4 replaced by f^2 / 4096^2 (remainder 8.5e-18). Results below 2^-1022
// are zero. Error below 1.2 units in the last place: 0.5 of the last product, 0.5 of the table's entry (correctly
// rounded in exp2_table.h; 0.51 of one uploaded by a context, the host's exp2).
#pragma once
#include <cstdint>

namespace inca {
namespace {

constexpr int kExp64Tab = 512, kExp64TabLarge = 2048;

template <int kTab = kExp64Tab>
__device__ __forceinline__ double exp2_neg64(double s, double w, const double* __restrict__ tab) {
  static_assert(kTab == kExp64Tab || kTab == kExp64TabLarge, "shift and polynomial of these tables");
  constexpr bool kLarge = kTab == kExp64TabLarge;
  constexpr int kBits = kLarge ? 11 : 9;
  const double kShift = kLarge ? 3298534883328.0 : 13194139533312.0;  // 1.5 * 2^(52 - kBits): last place 1/kTab
  const double t = fma(s, w, kShift);
  const double f = fma(s, w, kShift - t);
  double q;
  if (kLarge) {
    q = fma(f, -0.055504108664821580, 0.24022650753238586);             // -ln2^3/6, ln2^2/2 + ln2^4/24/4096^2
  } else {
    q = fma(f, 0.0096181291076284772, -0.055504108664821580);           // ln2^4/24, -ln2^3/6
    q = fma(f, q, 0.24022650695910072);                                 // ln2^2/2
  }
  q = fma(f, q, -0.69314718055994531);
  const int m = -__double2loint(t);
  const double T = tab[m & (kTab - 1)];
  const double r = fma(T, f * q, T);
  const double scaled = __hiloint2double(__double2hiint(r) + ((m >> kBits) << 20), __double2loint(r));
  // t >= kShift + 1021 and not NaN, compared as bits (t is positive): a comparison in FP64 is one more
  // instruction of the pipe that these kernels wait for (5 % of CH4's radial plot)
  const unsigned long long kZero = kLarge ? 0x42880000001FE800ull : 0x42A800000007FA00ull;
  const unsigned long long kInf = 0x7FF0000000000000ull;
  const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(t));
  return bits - kZero <= kInf - kZero ? 0.0 : scaled;
}

// acc + e v, and acc where the Gaussian e is zero: a merged polynomial far out may be infinite where the product
// form multiplied e into each factor first. (e compared as bits: outside the FP64 pipe.)
__device__ __forceinline__ double add_term64(double e, double v, double acc) {
  const double t = fma(e, v, acc);
  return __double_as_longlong(e) == 0 ? acc : t;
}

}  // namespace
}  // namespace inca
