// Fixed-point stencil sums: sum_j w_j x_j of float64 weights and values with
// integer multiply-adds, rounded once.
//
// GB300 issues 2 FP64 instructions per SM and clock, and 32 widening 32-bit
// integer multiply-adds and 64 integer logic or shift instructions beside
// them (measured together: 16 multiply-adds per DFMA cost the DFMA nothing).
// A weighted sum of seven or eight neighbour values costs about 14 integer
// instructions per term on those otherwise idle pipes and one FP64
// instruction in all, instead of one FP64 instruction per term.
//
// Values.  The producing pass stores, beside the double x, a 64-bit word:
// the mantissa as a two's complement integer X in bits 8..63 (low byte of X
// zero, 2^60 <= |X| < 2^63) and in the low byte an exponent q in steps of 3,
//     x = X 2^(3 q - 377),   1 <= q <= 127,
// exact for 2^-314 <= |x| < 2^67; zero is the word 0.  Anything else (NaN,
// infinities, magnitudes outside that range) sets the low byte's top bit.
//
// Weights.  w = (hi 2^28 + lo) 2^e with -2^27 <= lo < 2^27 and 2^55 <=
// |hi 2^28 + lo| < 2^56, exact for 2^-400 <= |w| <= 2^400 and for 0.
//
// Sum.  Every X_j is shifted right by the distance of its product's exponent
// e_j + 3 q_j below the largest one, so the products share one binary point,
// and the three significant partial products of (hi, lo) x (X's halves) are
// accumulated in 64 bits.  With M the largest |w_j x_j|: the shifts drop at
// most 2^-59 M per term, the product lo x (low half) at most 2^-56 M per
// term (rms below 2^-57.5, of either sign as lo is), and the final rounding
// 2^-56 M.  A chain of FP64 multiply-adds rounds by up to 2^-53 of each
// partial sum; a sum of zero products is exactly zero.
//
// A zero has no exponent: its word gives the product the exponent e_j of its
// weight alone, which could shift smaller products out (2^-314 of that weight
// and less).  Three ways around it (FxZeros): where the largest exponent is no
// more than a bound `top` of the e_j and some word is not zero, the sum leaves
// the zeros' exponents out, or it is left to FP64 with those below; or it
// cannot happen, with weights that lie within FX_PV_SPREAD binades of each
// other and words of values not so small (fx_word<FX_PV_MINQ>).  The tracer
// passes take weights below 2^36 and the constant FX_TOP: only sums with M
// below 2^-278 are left to FP64.
//
// A term that cannot be represented (a flagged word, or a weight out of
// range) makes the caller evaluate that one sum in FP64 instead: infinities
// and NaN propagate as they would there.
#pragma once

#include <cstring>

#ifdef __CUDACC__
#define SWG_HD __host__ __device__ __forceinline__
#else
#define SWG_HD inline
#endif

namespace swg {

using fx_t = unsigned long long;

constexpr unsigned FX_FLAG = 0x80; // low-byte bit of an unrepresentable value
constexpr int FX_ZERO_EXP = -100000; // exponent of a zero weight
constexpr int FX_BAD_EXP = 100000;   // and of a table's out-of-range weight
constexpr int FX_TOP = -20;          // largest exponent of a tracer weight
constexpr int FX_PV_MINQ = 8;        // smallest q of a word of the PV sums, and
constexpr int FX_PV_SPREAD = 3 * FX_PV_MINQ - 1; // what their weights differ by
constexpr int FX_SCALE = -317;       // 60 - 377: result exponent offset

struct Wt {
  int hi, lo, e;
};

SWG_HD fx_t fx_bits(double x) {
#ifdef __CUDA_ARCH__
  return fx_t(__double_as_longlong(x));
#else
  fx_t b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}

// whether the bits are those of +0 or -0, in 32-bit pieces (a 64-bit test
// becomes an FP64 comparison)
SWG_HD bool fx_is_zero(fx_t b) {
  const unsigned hi = unsigned(b >> 32), lo = unsigned(b);
  return ((hi & 0x7fffffffu) | lo) == 0;
}

// arithmetic right shift by any s >= 0 (64 and more: the sign)
SWG_HD long long fx_sar(long long x, unsigned s) {
#ifdef __CUDA_ARCH__
  long long r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
  return r;
#else
  return x >> (s > 63 ? 63 : s);
#endif
}

// The weight w; sets FX_FLAG in `flag` when it is out of range, or its exponent
// above TOP.
template <int TOP = 345> SWG_HD Wt fx_weight(double w, unsigned &flag) {
  static_assert(TOP <= 345, "2^400");
  const fx_t b = fx_bits(w);
  const int eb = int(unsigned(b >> 52) & 0x7ff);
  const long long s = (long long)b >> 63;
  long long W = (long long)(((b & 0xfffffffffffffULL) | 0x10000000000000ULL) << 3);
  W = (W ^ s) - s;
  Wt r;
  r.hi = int((W + (1LL << 27)) >> 28);
  r.lo = int(unsigned(W) << 4) >> 4;
  r.e = eb - 1078;
  if (unsigned(eb - 623) > unsigned(TOP + 455)) { // |w| below 2^-400, or above
    if (!fx_is_zero(b))
      flag |= FX_FLAG;
    r.hi = r.lo = 0;
    r.e = FX_ZERO_EXP;
  }
  return r;
}

// The word of the value x; MINQ: values with a smaller q are flagged.
template <int MINQ = 1> SWG_HD fx_t fx_word(double x) {
  const fx_t b = fx_bits(x);
  const unsigned eo = (unsigned(b >> 52) & 0x7ff) - 709u;
  const unsigned q = (eo * 21846u) >> 16; // eo / 3 for eo <= 380
  const unsigned r = eo - 3 * q;
  const long long s = (long long)b >> 63;
  long long X = (long long)(((b & 0xfffffffffffffULL) | 0x10000000000000ULL)
                            << ((8 + r) & 63));
  X = (X ^ s) - s;
  fx_t w = fx_t(X) | (q + 1);
  constexpr unsigned LEAST = 3 * (MINQ - 1);
  if (eo - LEAST > 380u - LEAST)
    w = fx_is_zero(b) ? 0 : 0xff;
  return w;
}

// The weight w for a table: exponent FX_BAD_EXP when it is out of range.
SWG_HD Wt fx_table_weight(double w) {
  unsigned bad = 0;
  Wt r = fx_weight<FX_TOP>(w, bad);
  if (bad)
    r.e = FX_BAD_EXP;
  return r;
}

// What a sum starts from, given the sum of the terms' hi: the low half x_l of
// an X enters the multiply-add as the signed number x_l - 2^31, so 2^31 hi is
// owed per term; and the rounding of the last shift.
SWG_HD long long fx_start(long long sum_hi) {
  return (sum_hi << 27) + (1LL << 27);
}

// R 2^(P + FX_SCALE) as a double (|P + FX_SCALE| below 900)
SWG_HD double fx_value(long long R, int P) {
#ifdef __CUDA_ARCH__
  const double d = __ll2double_rn(R);
  const int hi = __double2hiint(d);
  return __hiloint2double(hi == 0 ? 0 : hi + int(unsigned(P + FX_SCALE) << 20),
                          __double2loint(d));
#else
  const double d = double(R);
  fx_t b = fx_bits(d);
  if (b)
    b += fx_t((long long)(P + FX_SCALE)) << 52;
  double r;
  std::memcpy(&r, &b, 8);
  return r;
#endif
}

// c + 64-bit a b: written as the instruction, because the compiler otherwise
// sees through the halves of a 64-bit word and multiplies in 64 bits
SWG_HD void fx_mad(long long &c, int a, int b) {
#ifdef __CUDA_ARCH__
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(c) : "r"(a), "r"(b));
#else
  c += (long long)a * b;
#endif
}

// the product exponent e + 3 q of a word's low byte and a weight
SWG_HD int fx_exp(fx_t x, int e) {
#ifdef __CUDA_ARCH__
  unsigned r;
  asm("dp4a.u32.u32 %0, %1, %2, %3;"
      : "=r"(r)
      : "r"(unsigned(x)), "r"(3u), "r"(unsigned(e)));
  return int(r);
#else
  return int(unsigned(x) & 0xff) * 3 + e;
#endif
}

// Running state of one sum.
struct FxAcc {
  long long hh, m1, m2;
};
SWG_HD void fx_mac(FxAcc &a, const Wt &w, fx_t x, int P, int p) {
  const long long X =
      fx_sar((long long)(x & ~fx_t(0xff)), unsigned(P - p));
  const int xh = int(X >> 32);
  const int xl = int(unsigned(X) ^ 0x80000000u); // low half - 2^31
  fx_mad(a.hh, w.hi, xh);
  fx_mad(a.m1, w.hi, xl);
  fx_mad(a.m2, w.lo, xh);
}
SWG_HD double fx_finish(const FxAcc &a, int P) {
  const long long t = a.m2 + (a.m1 >> 4);
  return fx_value(a.hh + (t >> 28), P);
}

// The exponents p of N products and their largest; f: the words or-ed.
template <int N>
SWG_HD int fx_exps(const Wt (&w)[N], const fx_t (&x)[N], int (&p)[N],
                   unsigned &f) {
  f = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    f |= unsigned(x[j]);
    p[j] = fx_exp(x[j], w[j].e);
  }
  int P = p[0];
#pragma unroll
  for (int j = 1; j < N; ++j)
    P = P > p[j] ? P : p[j];
  return P;
}

// the largest exponent of the weights
template <int N> SWG_HD int fx_top(const Wt (&w)[N]) {
  int t = w[0].e;
#pragma unroll
  for (int j = 1; j < N; ++j)
    t = t > w[j].e ? t : w[j].e;
  return t;
}

// FX_FLAG where a sum with FX_LEAVE is left to FP64: a flagged word, or a largest
// exponent that may be a zero's beside a word that is not zero (without a weight
// that is not zero the sum is, and the exponent below half FX_ZERO_EXP).
SWG_HD unsigned fx_left(int P, int top, unsigned f) {
  constexpr int NONE = FX_ZERO_EXP / 2;
  if (unsigned(P - NONE) <= unsigned(top - NONE) && f != 0)
    f = FX_FLAG;
  return f & FX_FLAG;
}

// What a sum does about zeros under large weights (see above).
enum FxZeros { FX_RESOLVE, FX_LEAVE, FX_NONE };

// sum_j w_j x_j over N <= 14 terms; start = fx_start(sum of hi_j), top: no
// weight's exponent is above it.  The result is meaningless when a word's
// FX_FLAG is set, or with FX_LEAVE where fx_left says so, which is reported in
// `flag` (or-ed in).  FX_RESOLVE is for any weights and values, and what the
// others are tested beside; no pass takes it, as its branch keeps the compiler
// from mixing what stands before and after it: k_aux2 takes 3 %
// longer with it, k_cell_tracers with 8 tracers 8 % (630 -> 681 us at
// 256x256x64) and the batched edge pass 6 %.  FX_LEAVE takes 0.8, 0 and 4 %.
template <int N, FxZeros Z>
SWG_HD double fx_sum(const Wt (&w)[N], const fx_t (&x)[N], long long start,
                     int top, unsigned &flag) {
  static_assert(N <= 14, "the 64-bit accumulators hold 14 products");
  int p[N];
  unsigned f;
  int P = fx_exps(w, x, p, f);
  if (Z == FX_RESOLVE && P <= top && f != 0) {
    P = FX_ZERO_EXP;
#pragma unroll
    for (int j = 0; j < N; ++j)
      P = unsigned(x[j]) != 0 && p[j] > P ? p[j] : P;
  }
  // (each flag where the sums of its passes are the faster: 634 -> 630 us for
  // k_cell_tracers, 318 -> 304 us for the edge pass of 12 members)
  if (Z == FX_LEAVE)
    flag |= fx_left(P, top, f);
  FxAcc a{0, 0, start};
#pragma unroll
  for (int j = 0; j < N; ++j)
    fx_mac(a, w[j], x[j], P, p[j]);
  if (Z != FX_LEAVE)
    flag |= f & FX_FLAG;
  return fx_finish(a, P);
}
template <int N>
SWG_HD double fx_sum(const Wt (&w)[N], const fx_t (&x)[N], long long start,
                     unsigned &flag) {
  return fx_sum<N, FX_RESOLVE>(w, x, start, fx_top(w), flag);
}

// ---- sums of float64 values as they are
//
// The same sums from the bits of the doubles, for values gathered too few
// times to be worth a word: about 20 integer instructions per term.
// X = mantissa 2^8 (2^60 <= |X| < 2^61), a negative one's complement instead
// of its negation (2^-60 of it).  Weights carry their exponent as
// (e - 65) 2^20, so that adding the double's exponent field gives the
// product's; magnitudes 2^-120 .. 2^120.  A largest product outside
// 2^-760 .. 2^770 or so (all terms zero, infinities, NaN, subnormals among
// them) makes the caller evaluate the sum in FP64.
constexpr int FXR_ZERO = -0x7fffffff - 1;
SWG_HD Wt fx_raw_weight(double w, unsigned &flag) {
  Wt r = fx_weight(w, flag);
  if (r.e == FX_ZERO_EXP) {
    r.e = FXR_ZERO;
  } else {
    if (r.e < -175 || r.e > 65)
      flag |= FX_FLAG;
    r.e = (r.e - 65) * (1 << 20);
  }
  return r;
}

// sum_j w_j x_j; sets `slow` when it has to be evaluated in FP64 (a value that is
// not finite under a zero weight does not: the tables have none but padding)
template <int N>
SWG_HD double fx_raw_sum(const Wt (&w)[N], const double (&x)[N], bool &slow) {
  static_assert(N <= 7, "the sum of hi in 32 bits");
  int p[N], P = FXR_ZERO, sum = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    p[j] = int(unsigned(fx_bits(x[j]) >> 32) & 0x7ff00000u) + w[j].e;
    P = P > p[j] ? P : p[j];
    sum += w[j].hi;
  }
  FxAcc a{0, 0, fx_start(sum)};
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const fx_t b = fx_bits(x[j]);
    const unsigned s = (unsigned(P) - unsigned(p[j])) >> 20;
    fx_t X = ((b & 0xfffffffffffffULL) | 0x10000000000000ULL) << 8;
#ifdef __CUDA_ARCH__
    asm("shr.u64 %0, %0, %1;" : "+l"(X) : "r"(s));
#else
    X = s > 63 ? 0 : X >> s;
#endif
    const unsigned sgn = unsigned(int(unsigned(b >> 32)) >> 31);
    const int xh = int(unsigned(X >> 32) ^ sgn);
    const int xl = int(unsigned(X) ^ sgn ^ 0x80000000u);
    fx_mad(a.hh, w[j].hi, xh);
    fx_mad(a.m1, w[j].hi, xl);
    fx_mad(a.m2, w[j].lo, xh);
  }
  slow = slow || unsigned(P) - (200u << 20) >= (1535u << 20);
  const long long t = a.m2 + (a.m1 >> 4);
  const long long R = a.hh + (t >> 28);
#ifdef __CUDA_ARCH__
  const double d = __ll2double_rn(R);
  const int hi = __double2hiint(d);
  return __hiloint2double(hi == 0 ? 0 : hi + (P - (958 << 20)),
                          __double2loint(d));
#else
  const double d = double(R);
  fx_t b = fx_bits(d);
  if (b)
    b += fx_t((long long)(P - (958 << 20))) << 32;
  double r;
  std::memcpy(&r, &b, 8);
  return r;
#endif
}

} // namespace swg
