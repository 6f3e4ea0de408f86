// fftoc — the batched forward-FFT kernel template (one launch = `batch`
// transforms of size N, TPB transforms per CTA).
#pragma once
#include <cstring>
#include <utility>
#include "fft_core.cuh"

namespace fftoc {

// Fixed-point scale: input magnitudes are mapped below 2^FxBits<N>, leaving
// log2(N) + 2 bits of headroom under 2^63 (worst-case growth N, plus the
// sqrt(2)-scaled sums inside the radix-8/16 kernels and the 2^61 limit of the
// limb products).
template <int N> struct FxBits {
  static constexpr int B = (61 - ilog2c(N)) < 53 ? (61 - ilog2c(N)) : 53;
};

// Natural-word engine (EngFxN): the input has 53 bits, and passes 1..quarter
// scale their products by a quarter, so that the last pass has 53 - 2 quarter
// bits, at least FxBits<N>::B.  With input components below 2^53 the modulus
// is below 2^53.5, times the radix of each pass and a quarter in those passes:
// below 2^62.5 at the end for every N, and for every compiled plan at most
// 2^61.5 at the input of a pass with twiddles and 2^59.5 at a radix-16 pass's
// constant products.
template <int N> struct FxPasses {
  static constexpr int quarter = (53 - FxBits<N>::B) / 2;  // 0 up to N = 512, 1 at 1024 and 2048, 2 at 4096
};

// Rounding of the binary64 -> fixed-point input conversion of a size N.
// Small transforms (N <= 32) stream at the HBM limit with every resident CTA
// slot in use; there the truncating sequence (round toward zero, a negation
// after the shift) fits 64 registers and measured fastest (+9% at N = 8 on
// GB300).  From N = 64 up the kernels are bound by the integer pipes, and the
// floor sequence (the sign complemented before the shift, fewer instructions)
// measured 1-5% faster.  Every path of one size (batched, uneven, on-chip,
// device executors) uses its size's rounding, so their results agree bit for
// bit.
template <int N> struct FxTrunc {
  static constexpr bool value = N <= 32;
};

// Sizes whose kernels convert threads with widely spread values by fx_in_far
// instead of the general conversion (values over twelve decades leave the fast
// path in most threads).  Same values, one more block of code: measured 5 %
// faster on such data at N = 64, 128 and 1024 (1 GiB, log-uniform in [1e-6, 1e6]:
// 365 -> 347, 385 -> 366, 517 -> 490 us) with ordinary data unchanged; at 256,
// 512 and 2048 3-5 % faster there but up to 1 % slower on ordinary data, at 4096
// no faster.
template <int N> struct FxFar {
  static constexpr bool value = N == 64 || N == 128 || N == 1024;
};

// --- binary64 <-> block fixed point -------------------------------------------
FFTOC_HD unsigned hi_word(double v) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2hiint(v);
#else
  unsigned long long b;
  memcpy(&b, &v, 8);
  return (unsigned)(b >> 32);
#endif
}
FFTOC_HD unsigned lo_word(double v) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2loint(v);
#else
  unsigned long long b;
  memcpy(&b, &v, 8);
  return (unsigned)b;
#endif
}
FFTOC_HD double from_words(unsigned hi, unsigned lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const unsigned long long b = ((unsigned long long)hi << 32) | lo;
  double v;
  memcpy(&v, &b, 8);
  return v;
#endif
}

FFTOC_HD int expo_of(unsigned hw) { return (int)((hw >> 20) & 0x7FFu); }

// value * 2^(1022 + B - Emax), eref = Emax + 53 - B, with M the 53-bit
// significand and d = eref - e: M >> d for a positive value.  A negative one
// gives -(M >> d) (TRUNC: toward zero) or ~(M >> d) = floor(-M / 2^d) -
// [2^d divides M] (floor: the complement of the shifted magnitude, which the
// fast path below forms by complementing before the shift).  Zeros of either
// sign give 0.
template <bool TRUNC = false>
FFTOC_HD long long fx_in(unsigned hw, unsigned lw, int eref) {
  const int e = expo_of(hw);
  const unsigned mh = (hw & 0xFFFFFu) | (e ? 0x100000u : 0u);
  if ((mh | lw) == 0u) return 0;
  const int ee = e > 1 ? e : 1;
  const int d0 = eref - ee;
  const int d = d0 < 63 ? d0 : 63;
  const unsigned long long m = ((((unsigned long long)mh) << 32) | lw) >> d;
  const long long r = (long long)m;
  return ((int)hw < 0) ? (TRUNC ? -r : ~r) : r;
}

// x * 2^K, K = Emax - 1022 - B: the correctly rounded conversion with K added
// to its exponent field (exact).  Valid while every result exponent stays in
// the normal range (fx_scale's `slow` is false); one FP64-pipe instruction.
// HI_ZERO: test the converted high word for zero (a nonzero integer converts
// to a normal number, so the two tests agree).
template <bool HI_ZERO = false>
FFTOC_HD double fx_out(long long x, int kshift) {
  const double d = (double)x;
  const unsigned hi = hi_word(d);
  const bool nonzero = HI_ZERO ? hi != 0u : x != 0;
  return from_words(nonzero ? hi + (unsigned)kshift : hi, lo_word(d));
}

// Transforms whose outputs may be subnormal or overflow: ldexp.  Kept out of
// line so the compiler cannot if-convert it into the fast path (predicated-off
// FP64 instructions would still occupy the FP64 pipe).
#ifdef __CUDA_ARCH__
__device__ __noinline__ double fx_out_slow(long long x, int K) { return ldexp((double)x, K); }
#else
inline double fx_out_slow(long long x, int K) { return ldexp((double)x, K); }
#endif

// fx_in out of line, for the rare transforms that leave the fast input path.
#ifdef __CUDA_ARCH__
template <bool TRUNC>
__device__ __noinline__ long long fx_in_slow(unsigned hw, unsigned lw, int eref) { return fx_in<TRUNC>(hw, lw, eref); }
#else
template <bool TRUNC>
inline long long fx_in_slow(unsigned hw, unsigned lw, int eref) { return fx_in<TRUNC>(hw, lw, eref); }
#endif

// Scale parameters of a transform from its largest biased exponent.
struct FxScale {
  int eref, K, kshift;
  bool slow, special;
};
// H: bits of scale that the passes take off (EngFxN's quarter-scale products).
template <int B, int H = 0>
FFTOC_HD FxScale fx_scale(int em) {
  FxScale s;
  s.special = (em == 0x7FF);
  // subnormals (exponent field 0) are scaled like exponent field 1
  if (em < 1) em = 1;
  s.K = em - 1022 - (B - H);
  s.kshift = (int)((unsigned)s.K << 20);
  s.slow = (em < B - H) || (em > 1983 + (B - H));
  s.eref = em + 53 - B;
  return s;
}
// Scale of a size under engine E: input bits and the bits its passes take off.
template <class E, int N>
FFTOC_HD FxScale fx_size_scale(int em) {
  if constexpr (E::kNatural) return fx_scale<53, 2 * FxPasses<N>::quarter>(em);
  else return fx_scale<FxBits<N>::B>(em);
}

// Fast conversion for values within 2^31 of the transform's largest exponent
// (all normal), bit-identical to fx_in there.  With S the sign mask
// (0 or ~0), the 96-bit word S:(M ^ S) is shifted right by d with two
// wrap-mode funnel shifts, which use d mod 32: d is taken as
// eref - (hw >> 20), whose sign bit at position 11 is a multiple of 32.
FFTOC_HD long long fx_in_near(unsigned hw, unsigned lw, int eref) {
  const unsigned S = (unsigned)((int)hw >> 31);
  const unsigned mh = (hw & 0xFFFFFu) ^ (S ^ 0x100000u);  // ((hw & 0xFFFFF) | 0x100000) ^ S
  const unsigned l = lw ^ S;
  const unsigned d = (unsigned)eref - (hw >> 20);
#ifdef __CUDA_ARCH__
  unsigned lo, hi;
  asm("shf.r.wrap.b32 %0, %1, %2, %3;" : "=r"(lo) : "r"(l), "r"(mh), "r"(d));
  asm("shf.r.wrap.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(mh), "r"(S), "r"(d));
#else
  const unsigned sh = d & 31u;
  const unsigned lo = (unsigned)((((unsigned long long)mh << 32) | l) >> sh);
  const unsigned hi = (unsigned)((((unsigned long long)S << 32) | mh) >> sh);
#endif
  return (long long)(((unsigned long long)hi << 32) | lo);
}

// Conversion of a normal value at any distance below the transform's largest
// exponent, bit-identical to fx_in (floor): from 32 bits down the 96-bit word
// is taken one word further up, and past 63 it is the sign.  5 instructions
// more than fx_in_near, about 8 fewer than fx_in.
FFTOC_HD long long fx_in_far(unsigned hw, unsigned lw, int eref) {
  const unsigned S = (unsigned)((int)hw >> 31);
  unsigned mh = (hw & 0xFFFFFu) ^ (S ^ 0x100000u);
  unsigned l = lw ^ S;
  const int d0 = eref - expo_of(hw), d = d0 < 63 ? d0 : 63;
  if (d & 32) {
    l = mh;
    mh = S;
  }
#ifdef __CUDA_ARCH__
  unsigned lo, hi;
  asm("shf.r.wrap.b32 %0, %1, %2, %3;" : "=r"(lo) : "r"(l), "r"(mh), "r"(d));
  asm("shf.r.wrap.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(mh), "r"(S), "r"(d));
#else
  const unsigned sh = (unsigned)d & 31u;
  const unsigned lo = (unsigned)((((unsigned long long)mh << 32) | l) >> sh);
  const unsigned hi = (unsigned)((((unsigned long long)S << 32) | mh) >> sh);
#endif
  return (long long)(((unsigned long long)hi << 32) | lo);
}

// The truncating fast conversion (bit-identical to fx_in<true> on the same
// domain): the shifted magnitude, negated for a negative value.
FFTOC_HD long long fx_in_near_trunc(unsigned hw, unsigned lw, int eref) {
  const int d = eref - expo_of(hw);
  const unsigned mh = (hw & 0xFFFFFu) | 0x100000u;
#ifdef __CUDA_ARCH__
  const unsigned lo = __funnelshift_r(lw, mh, d);
#else
  const unsigned lo = (unsigned)((((unsigned long long)mh << 32) | lw) >> d);
#endif
  const unsigned hi = mh >> d;
  const long long m = (long long)(((unsigned long long)hi << 32) | lo);
  return ((int)hw < 0) ? -m : m;
}

// Largest and smallest biased exponents of a thread's raw points: from the
// sign-cleared high words (floor sizes), or the exponent fields in two loops
// (the sequence that fits the small sizes' register budget).
template <int P, bool TRUNC = false>
FFTOC_HD void fx_exponent_range(const double2 (&raw)[P], int& emax, int& emin) {
  if constexpr (TRUNC) {
    int em = 0, en = 0x7FF;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const int a = expo_of(hi_word(raw[i].x)), b = expo_of(hi_word(raw[i].y));
      const int hi = a > b ? a : b;
      em = em > hi ? em : hi;
    }
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const int a = expo_of(hi_word(raw[i].x)), b = expo_of(hi_word(raw[i].y));
      en = en < a ? en : a;
      en = en < b ? en : b;
    }
    emax = em;
    emin = en;
  } else {
#ifdef __CUDA_ARCH__
    // The sign-cleared words ordered as binary32 values (three-operand
    // minimum and maximum with the sign cleared in the operand: 2.2
    // instructions a point against 4.5 for the integer form).  Exponent
    // fields from 0x7F8 up look like infinities and NaNs there: the maximum
    // then is NaN or infinity, and the integer form below decides.
    float fmax = 0.0f, fmin = __uint_as_float(0x7F800000u);
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const float a = fabsf(__uint_as_float(hi_word(raw[i].x))), b = fabsf(__uint_as_float(hi_word(raw[i].y)));
      asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(fmax) : "f"(a), "f"(b));
      asm("min.f32 %0, %0, %1, %2;" : "+f"(fmin) : "f"(a), "f"(b));
    }
    emax = (int)(__float_as_uint(fmax) >> 20);
    emin = (int)(__float_as_uint(fmin) >> 20);
    if (emax < 0x7F8) return;
#endif
    unsigned amax = 0u, amin = 0x7FFFFFFFu;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const unsigned a = hi_word(raw[i].x) & 0x7FFFFFFFu, b = hi_word(raw[i].y) & 0x7FFFFFFFu;
      const unsigned hi = a > b ? a : b, lo = a < b ? a : b;
      amax = amax > hi ? amax : hi;
      amin = amin < lo ? amin : lo;
    }
    emax = (int)(amax >> 20);
    emin = (int)(amin >> 20);
  }
}

// Convert a thread's P raw points; the fast path is taken when every value is
// normal and within 2^31 of the transform maximum (the usual case), the next
// (FAR, fx_in_far) when every value is normal.  emin is the thread's smallest
// biased exponent (fx_exponent_range).
// OUTLINE: the other path calls the out-of-line fx_in_slow.  TRUNC: the
// size's rounding (FxTrunc).
template <int P, bool OUTLINE = false, bool TRUNC = false, bool FAR = false>
FFTOC_HD void fx_convert_in(const double2 (&raw)[P], long long (&re)[P], long long (&im)[P], int eref, int emin) {
  if (emin >= 1 && eref - emin < 32) {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      if constexpr (TRUNC) {
        re[i] = fx_in_near_trunc(hi_word(raw[i].x), lo_word(raw[i].x), eref);
        im[i] = fx_in_near_trunc(hi_word(raw[i].y), lo_word(raw[i].y), eref);
      } else {
        re[i] = fx_in_near(hi_word(raw[i].x), lo_word(raw[i].x), eref);
        im[i] = fx_in_near(hi_word(raw[i].y), lo_word(raw[i].y), eref);
      }
    }
  } else if (FAR && emin >= 1) {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      re[i] = fx_in_far(hi_word(raw[i].x), lo_word(raw[i].x), eref);
      im[i] = fx_in_far(hi_word(raw[i].y), lo_word(raw[i].y), eref);
    }
  } else if constexpr (OUTLINE) {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      re[i] = fx_in_slow<TRUNC>(hi_word(raw[i].x), lo_word(raw[i].x), eref);
      im[i] = fx_in_slow<TRUNC>(hi_word(raw[i].y), lo_word(raw[i].y), eref);
    }
  } else {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      re[i] = fx_in<TRUNC>(hi_word(raw[i].x), lo_word(raw[i].x), eref);
      im[i] = fx_in<TRUNC>(hi_word(raw[i].y), lo_word(raw[i].y), eref);
    }
  }
}
template <int P, bool OUTLINE = false, bool TRUNC = false>
FFTOC_HD void fx_convert_in(const double2 (&raw)[P], long long (&re)[P], long long (&im)[P], int eref) {
  int emax, emin;
  fx_exponent_range<P, TRUNC>(raw, emax, emin);
  fx_convert_in<P, OUTLINE, TRUNC>(raw, re, im, eref, emin);
}

// Largest value of em over the T consecutive threads of each transform (TPB
// transforms per CTA, thread tid, transform j = tid / T).  T <= 32: within the
// warp (a warp reduction for T = 32, shuffles over the T lanes otherwise).
// T > 32 (whole warps per transform): a warp reduction, one word per warp in
// `red` (TPB * T / 32 ints of shared memory) and one __syncthreads().
template <int T, int TPB>
__device__ __forceinline__ int fx_transform_max(int em, int tid, int j, int* red) {
  if constexpr (T == 32) {
    em = __reduce_max_sync(0xffffffffu, em);
  } else if constexpr (T > 1 && T < 32) {
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) em = max(em, __shfl_xor_sync(0xffffffffu, em, o, T));
  } else if constexpr (T > 32) {
    constexpr int W = T / 32;
    em = __reduce_max_sync(0xffffffffu, em);
    if ((tid & 31) == 0) red[tid >> 5] = em;
    __syncthreads();
    em = red[j * W];
#pragma unroll
    for (int w = 1; w < W; ++w) em = max(em, red[j * W + w]);
  }
  return em;
}

// Binary64 transforms with a component of 2^1021 / N or more: the outputs are
// below 2 N times the largest component, and inside EngF64's butterflies values
// reach sqrt(2) times the moduli of the plain products, which may overflow where
// no output does.  Such transforms (non-finite ones with them) run on inputs
// scaled by 2^-down, and their outputs are scaled back: both exact but for
// outputs that are not representable, and for parts 2^-1000 times the largest.
template <int N> struct F64Range {
  static constexpr int down = ilog2c(N) + 4;
  // the largest exponent field that is transformed as it is: all below 2^1021 / N,
  // and below the fields that f64_exponent cannot tell apart
  static constexpr int top = 2044 - ilog2c(N) < 2039 ? 2044 - ilog2c(N) : 2039;
};
// The largest exponent field of a thread's points, ordered as binary32 values
// (fx_exponent_range); 0x7F8 or 0x7FF for fields from 0x7F8 up.
template <int P>
__device__ __forceinline__ int f64_exponent(const double (&re)[P], const double (&im)[P]) {
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const float a = fabsf(__int_as_float(__double2hiint(re[i]))), b = fabsf(__int_as_float(__double2hiint(im[i])));
    asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(a), "f"(b));
  }
  return (int)(__float_as_uint(m) >> 20);
}
// Values times 2^-D and back, on the words: predicated multiplications would
// occupy the FP64 pipe in every transform (38 % more time at N = 16).  Infinities
// and NaNs stay, values below 2^(D - 1022) become zero, and on the way back what
// is not representable becomes an infinity.
template <int D>
__device__ __forceinline__ double f64_down(double v) {
  const int hi = __double2hiint(v), a = hi & 0x7FFFFFFF;
  const bool none = a < ((D + 1) << 20);
  return __hiloint2double(none ? 0 : a >= 0x7FF00000 ? hi : hi - (D << 20), none ? 0 : __double2loint(v));
}
template <int D>
__device__ __forceinline__ double f64_up(double v) {
  const int hi = __double2hiint(v), a = hi & 0x7FFFFFFF;
  if (a < (1 << 20) || a >= 0x7FF00000) return v;
  const bool over = a >= ((0x7FF - D) << 20);
  return __hiloint2double(over ? (hi & (int)0x80000000) | 0x7FF00000 : hi + (D << 20), over ? 0 : __double2loint(v));
}
template <int D, int P>
__device__ __forceinline__ void f64_scale_down(double (&re)[P], double (&im)[P]) {
#pragma unroll
  for (int i = 0; i < P; ++i) {
    re[i] = f64_down<D>(re[i]);
    im[i] = f64_down<D>(im[i]);
  }
}
template <int D, int P>
__device__ __forceinline__ void f64_scale_up(double (&re)[P], double (&im)[P]) {
#pragma unroll
  for (int i = 0; i < P; ++i) {
    re[i] = f64_up<D>(re[i]);
    im[i] = f64_up<D>(im[i]);
  }
}

// Programmatic dependent launch (launch_overlapped): a kernel may start while the one
// before it in its stream drains.  after_previous() waits for that kernel's
// completion and must come before any access to the caller's buffers;
// allow_next(), after it, lets the next kernel's CTAs take the places that this
// grid does not need (they wait at their own after_previous(); called before
// the wait, it would let a chain of small grids pile up on the device, on
// whichever SMs have room: 9.2 instead of 5.4 us for 1/3 of a wave of N = 512).
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// A tile loop's first tile, as a value that exists only after
// after_previous(): read-only loads whose addresses follow from it cannot move
// above.  32 bits, as blockIdx is: a 64-bit value here cost the exact-slice
// kernels 4 to 7 % at N = 128 and 512.
__device__ __forceinline__ unsigned first_tile() {
  unsigned t = blockIdx.x;
  asm volatile("" : "+r"(t)::"memory");
  return t;
}
// A point of the caller's input.  Not __ldg: a kernel launched with the overlap
// is there while the one before it still writes this memory, and a read-only
// load is defined only where nothing writes during the kernel's lifetime (the
// compiler may move it above after_previous(), and a line that it left in L1
// need not be dropped by the wait).
__device__ __forceinline__ double2 load_point(const double2* p) {
  double2 v;
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

// A store without a branch, which would keep the stores behind the last pass.
__device__ __forceinline__ void store_point_if(double2* p, double2 v, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\t@q st.global.v2.f64 [%0], {%1, %2};\n\t}" ::"l"(p), "d"(v.x),
               "d"(v.y), "r"((int)on)
               : "memory");
}

// --- the kernel ---------------------------------------------------------------
template <class E, class PL>
struct Fft {
  using S = typename E::S;
  using TW = typename E::TW;
  static constexpr int N = PL::N;
  static constexpr int TPB = PL::TPB;
  static constexpr int P = PL::P;
  static constexpr int T = PL::T;
  static constexpr int NS = PL::S;
  // padded shared layout: one 16-byte pad slot after every 2^SH points, so
  // the first pass's stride-R writes and every stride-1 read hit distinct
  // bank groups, and all addresses are a per-thread base plus a constant
  static constexpr int SH = PL::R[0] >= 16 ? 4 : 3;
  static constexpr int NP = N + (N >> SH);
  static constexpr int THREADS = T * TPB;
  static constexpr bool STAGED = T < 8 && !PL::NO_STAGE;  // small N: stage HBM tiles through smem
  static constexpr int SMEM = TPB * NP * 16 + 64;  // + 16 words of exponent scratch
  static_assert(T <= 32 || TPB * (T / 32) <= 16, "exponent scratch holds one word per warp, 16 words");

  // 16-byte slot of element e of block-local transform j
  __device__ __forceinline__ static int slot(int j, int e) { return j * NP + e + (e >> SH); }

  template <int s, int b>
  __device__ __forceinline__ static void butterfly(S (&re)[P], S (&im)[P], int t, const TW* __restrict__ tw) {
    constexpr int R = PL::R[s];
    constexpr int B = P / R;
    constexpr int p = PL::span(s);
    if constexpr (s > 0) {
      const int tp = t + T * b;
      const int k = tp & (p - 1);
      const TW* base = tw + PL::tw_offset(s) + k;
      if constexpr (E::kNatural) {
        const int2* sums = reinterpret_cast<const int2*>(tw + PL::TW_COUNT) + PL::tw_offset(s) + k;
        constexpr bool QUARTER = s <= FxPasses<N>::quarter;
        if constexpr (QUARTER) {  // the untwiddled input too
          re[b] >>= 2;
          im[b] >>= 2;
        }
#pragma unroll
        for (int m = 1; m < R; ++m)
          E::template cmul<QUARTER>(re[b + B * m], im[b + B * m], __ldg(base + (m - 1) * p), __ldg(sums + (m - 1) * p));
      } else if constexpr (E::kId == EngF64::kId) {
        constexpr int H = R / 2;
#pragma unroll
        for (int m = 1; m < H; ++m) E::cmul(re[b + B * m], im[b + B * m], __ldg(base + (m - 1) * p));
#pragma unroll
        for (int m = 0; m < H; ++m)
          E::twiddled_sum(re[b + B * m], im[b + B * m], re[b + B * (m + H)], im[b + B * (m + H)],
                          __ldg(base + (m + H - 1) * p), E::tangent_turned((m + H) * k, R * p));
        f64_finish<R, b, B, P>(re, im);
        return;
      } else {
#pragma unroll
        for (int m = 1; m < R; ++m) {
          const TW w = __ldg(base + (m - 1) * p);
          E::cmul(re[b + B * m], im[b + B * m], w);
        }
      }
    }
    dft<E, R, b, B, P>(re, im);
  }

  template <int s, int... bs>
  __device__ __forceinline__ static void pass(S (&re)[P], S (&im)[P], int t, const TW* __restrict__ tw,
                                              std::integer_sequence<int, bs...>) {
    (butterfly<s, bs>(re, im, t, tw), ...);
  }

  // destination index of output m of butterfly b in pass s
  template <int s>
  __device__ __forceinline__ static int dest(int t, int b, int m) {
    constexpr int R = PL::R[s];
    constexpr int p = PL::span(s);
    const int tp = t + T * b;
    const int k = tp & (p - 1);
    return (tp - k) * R + k + m * p;
  }

  // Slots and elements below are a base per thread and butterfly plus a
  // constant per point.  The base's pad is computed once, since every constant
  // is a multiple of 2^SH (left to the compiler, the pad of each slot cost
  // 3 instructions a point and exchange at N = 512).
  //
  // slot of output 0 of butterfly b in pass s; output m is m * slot_step<s>() further
  template <int s>
  __device__ __forceinline__ static int slot0(int j, int t, int b) {
    const int e = dest<s>(t, b, 0);
    return j * NP + e + (e >> SH);
  }
  template <int s>
  __host__ __device__ static constexpr int slot_step() {
    constexpr int p = PL::span(s);
    static_assert((s == 0 && PL::R[0] <= (1 << SH)) || p % (1 << SH) == 0, "an output's pad is a constant");
    return p + (p >> SH);
  }
  static constexpr bool FIXED_PADS = PL::R[0] == (1 << SH);

  template <int s>
  __device__ __forceinline__ static void write_smem(S (&re)[P], S (&im)[P], int j, int t, longlong2* sm) {
    constexpr int R = PL::R[s];
    constexpr int B = P / R;
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const int q = FIXED_PADS ? slot0<s>(j, t, b) : 0;
#pragma unroll
      for (int m = 0; m < R; ++m) {
        longlong2 v;
        v.x = to_bits(re[b + B * m]);
        v.y = to_bits(im[b + B * m]);
        if constexpr (FIXED_PADS) sm[q + m * slot_step<s>()] = v;
        else sm[slot(j, dest<s>(t, b, m))] = v;
      }
    }
  }

  __device__ __forceinline__ static void read_smem(S (&re)[P], S (&im)[P], int j, int t, const longlong2* sm) {
    constexpr bool fixed = T % (1 << SH) == 0 || (1 << SH) % T == 0;
    const int q = j * NP + t + (t >> SH);
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const longlong2 v = fixed ? sm[q + T * i + (T * i >> SH)] : sm[slot(j, t + T * i)];
      re[i] = from_bits(v.x);
      im[i] = from_bits(v.y);
    }
  }
  __device__ __forceinline__ static long long to_bits(S v) {
    if constexpr (E::kId == EngF64::kId) return __double_as_longlong(v);
    else return (long long)v;
  }
  __device__ __forceinline__ static S from_bits(long long b) {
    if constexpr (E::kId == EngF64::kId) return __longlong_as_double(b);
    else return (S)b;
  }

  template <int s>
  __device__ __forceinline__ static void run_passes(S (&re)[P], S (&im)[P], int j, int t, const TW* __restrict__ tw,
                                                    longlong2* sm) {
    constexpr int R = PL::R[s];
    pass<s>(re, im, t, tw, std::make_integer_sequence<int, P / R>{});
    if constexpr (s + 1 < NS) {
      if constexpr (s > 0) __syncthreads();  // previous readers of the buffer are done
      write_smem<s>(re, im, j, t, sm);
      __syncthreads();
      read_smem(re, im, j, t, sm);
      run_passes<s + 1>(re, im, j, t, tw, sm);
    }
  }

  // The passes of the CTA's binary64 transforms.  True if one of them may
  // overflow on the way (F64Range, on the first pass's outputs); then no output
  // is stored, and redo_ranged() follows.  The vote is the first exchange's
  // barrier, and nothing branches on it before the stores: a branch there keeps
  // the next pass's twiddle loads from moving above the barrier (N = 512 to 4096,
  // one transform: 2 to 6 % more time).
  __device__ __forceinline__ static bool run_voted(double (&re)[P], double (&im)[P], bool check, int j, int t,
                                                   const TW* __restrict__ tw, longlong2* sm) {
    pass<0>(re, im, t, tw, std::make_integer_sequence<int, P / PL::R[0]>{});
    const bool large = check && f64_exponent(re, im) > F64Range<N / PL::R[0]>::top;
    write_smem<0>(re, im, j, t, sm);
    const bool hold = __syncthreads_or(large);
    read_smem(re, im, j, t, sm);
    run_passes<1>(re, im, j, t, tw, sm);
    return hold;
  }

  // The CTA's transforms again from their inputs, those of large values scaled;
  // src and dst are this thread's transform.  Out of line: inlined it took the
  // kernels' registers (binary64, 1,500 transforms of 256 points 17.7 -> 20.6 us).
  __device__ __noinline__ static void redo_ranged(const double2* src, double2* dst, bool active, const TW* tw,
                                                  longlong2* sm, int* red) {
    const int tid = threadIdx.x, j = tid / T, t = tid - j * T;
    double re[P], im[P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const double2 v = active ? src[t + T * i] : make_double2(0.0, 0.0);
      re[i] = v.x;
      im[i] = v.y;
    }
    __syncthreads();  // the last readers of the exchange buffer and of `red` are done
    const bool scaled = fx_transform_max<T, TPB>(f64_exponent(re, im), tid, j, red) > F64Range<N>::top;
    if (scaled) f64_scale_down<F64Range<N>::down>(re, im);
    run_passes<0>(re, im, j, t, tw, sm);
    if (scaled) f64_scale_up<F64Range<N>::down>(re, im);
    if (!active) return;
    constexpr int RL = PL::R[NS - 1], BL = P / RL;
#pragma unroll
    for (int b = 0; b < BL; ++b)
#pragma unroll
      for (int m = 0; m < RL; ++m) dst[dest<NS - 1>(t, b, m)] = make_double2(re[b + BL * m], im[b + BL * m]);
  }
};

// Where the transforms of one CTA tile live.  IndexedTile (the uneven-batch
// kernel): transform j of the tile at element base[j], with the bases staged in
// shared memory by the caller.
struct IndexedTile {
  static constexpr bool REPEATS = false;
  const double2* __restrict__ in;
  double2* __restrict__ out;
  const long long* base;  // shared memory, one entry per transform of the tile
  long long tile0, count;
  __device__ __forceinline__ const double2* in_of(int j) const { return in + base[j]; }
  __device__ __forceinline__ double2* out_of(int j) const { return out + base[j]; }
  __device__ __forceinline__ const double2* in_elem(int, int jj, int e) const { return in + base[jj] + e; }
  __device__ __forceinline__ double2* out_elem(int, int jj, int e) const { return out + base[jj] + e; }
  __device__ __forceinline__ static double2 load(const double2* p) { return __ldg(p); }
};

// Tiles of an uneven batch for plans that do not stage their tile (each
// thread touches only its own transform): the thread's transform offset in a
// register, loaded ahead by the caller.
struct RegTile {
  static constexpr bool REPEATS = false;
  const double2* __restrict__ in;
  double2* __restrict__ out;
  long long off;  // this thread's transform
  long long tile0, count;
  __device__ __forceinline__ const double2* in_of(int) const { return in + off; }
  __device__ __forceinline__ double2* out_of(int) const { return out + off; }
  __device__ __forceinline__ const double2* in_elem(int, int, int e) const { return in + off + e; }
  __device__ __forceinline__ double2* out_elem(int, int, int e) const { return out + off + e; }
  __device__ __forceinline__ static double2 load(const double2* p) { return __ldg(p); }
};

// The on-chip repeat harness: the tile's transforms resident in shared
// memory (`buf`, TPB * N points, transformed in place), loaded with plain
// shared loads.
template <int N>
struct SmemTile {
  static constexpr bool REPEATS = true;  // outputs are inputs again, up to infinities
  double2* buf;
  long long tile0, count;  // tile0 = 0, count = TPB
  __device__ __forceinline__ const double2* in_of(int j) const { return buf + j * N; }
  __device__ __forceinline__ double2* out_of(int j) const { return buf + j * N; }
  __device__ __forceinline__ const double2* in_elem(int idx, int, int) const { return buf + idx; }
  __device__ __forceinline__ double2* out_elem(int idx, int, int) const { return buf + idx; }
  __device__ __forceinline__ static double2 load(const double2* p) { return *p; }
};

// One CTA tile: load raw points (binary64), convert, run the passes, convert
// back and store.  Engine-specific entry/exit.  Used by the uneven-batch
// kernel; the batched kernel below carries the same body.
template <class E, class PL, class Tile>
__device__ __forceinline__ void fft_tile(const Tile& tl, const typename E::TW* __restrict__ tw,
                                         unsigned char* smem_raw) {
  using EK = PlanEngine<E, PL>;
  using F = Fft<EK, PL>;
  using S = typename EK::S;
  constexpr int N = PL::N, TPB = PL::TPB;
  constexpr int P = F::P, T = F::T, NS = F::NS;
  longlong2* sm = reinterpret_cast<longlong2*>(smem_raw);

  const int tid = threadIdx.x;
  const int j = tid / T;
  const int t = tid - j * T;
  const long long tile0 = tl.tile0;
  const bool active = tile0 + j < tl.count;
  const long long tile_elems = (min((long long)TPB, tl.count - tile0)) * N;

  // ---- load raw binary64 points: point i of this thread is element t + T*i
  double2 raw[P];
  if constexpr (F::STAGED) {
    for (int idx = tid; idx < tile_elems; idx += F::THREADS) {
      const int jj = idx / N, e = idx - jj * N;
      const double2 v = Tile::load(tl.in_elem(idx, jj, e));
      sm[F::slot(jj, e)] = make_longlong2(__double_as_longlong(v.x), __double_as_longlong(v.y));
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const longlong2 v = sm[F::slot(j, t + T * i)];
      raw[i] = make_double2(__longlong_as_double(v.x), __longlong_as_double(v.y));
    }
  } else {
    // RegTile's threads past the tile hold the offset of a transform of the tile
    const double2* src = tl.in_of(j) + t;
#pragma unroll
    for (int i = 0; i < P; ++i)
      raw[i] = EK::kNatural || active ? Tile::load(src + T * i) : make_double2(0.0, 0.0);
  }

  S re[P], im[P];
  int K = 0, kshift = 0;
  bool slow = false, special = false;
  if constexpr (E::kId == EngF64::kId) {
#pragma unroll
    for (int i = 0; i < P; ++i) { re[i] = raw[i].x; im[i] = raw[i].y; }
  } else {
    // largest biased exponent of the transform, smallest of this thread
    constexpr bool TR = FxTrunc<N>::value;
    int em, emin;
    fx_exponent_range<P, TR>(raw, em, emin);
    em = fx_transform_max<T, TPB>(em, tid, j, reinterpret_cast<int*>(smem_raw + TPB * F::NP * 16));
    const FxScale sc = fx_size_scale<EK, N>(em);
    special = sc.special;
    K = sc.K;
    kshift = sc.kshift;
    slow = sc.slow;
    fx_convert_in<P, false, TR, FxFar<N>::value>(raw, re, im, sc.eref, emin);
  }

  if constexpr (F::STAGED) __syncthreads();  // staging buffer is reused by the passes
  // binary64: a transform of the CTA has to be redone (nothing is stored before);
  // a transform that one thread holds is scaled where it is
  bool hold = false, scaled = false, check = active;
  if constexpr (E::kId == EngF64::kId && Tile::REPEATS) {  // scaling does nothing for infinities and NaNs
#pragma unroll
    for (int i = 0; i < P; ++i) check = check && expo_of(hi_word(re[i])) < 0x7FF && expo_of(hi_word(im[i])) < 0x7FF;
  }
  if constexpr (E::kId == EngF64::kId && NS > 1) {
    hold = F::run_voted(re, im, check, j, t, tw, sm);
  } else {
    if constexpr (E::kId == EngF64::kId) {
      scaled = check && f64_exponent(re, im) > F64Range<N>::top;
      if (scaled) f64_scale_down<F64Range<N>::down>(re, im);
    }
    F::template run_passes<0>(re, im, j, t, tw, sm);
    if constexpr (E::kId == EngF64::kId) {
      if (scaled) f64_scale_up<F64Range<N>::down>(re, im);
    }
  }

  // ---- store: output m of butterfly b of the last pass is element dest(...)
  constexpr int RL = PL::R[NS - 1];
  constexpr int BL = P / RL;
  // Fixed point: the rare transforms whose outputs leave the normal range, or
  // whose inputs were not finite, take the slow conversion: a per-value select
  // where the output is staged or the size is small (FxTrunc; both measured
  // faster so), else one branch per thread between two store loops.
  auto value = [&](int i) -> double2 {
    if constexpr (E::kId == EngF64::kId) {
      return make_double2(re[i], im[i]);
    } else {
      return make_double2(fx_out<PL::OUT_HI_ZERO>((long long)re[i], kshift),
                          fx_out<PL::OUT_HI_ZERO>((long long)im[i], kshift));
    }
  };
  auto slow_value = [&](int i) -> double2 {
    if constexpr (E::kId == EngF64::kId) {
      return make_double2(re[i], im[i]);
    } else {
      const double qnan = __longlong_as_double(0x7FF8000000000000LL);
      return special ? make_double2(qnan, qnan)
                     : make_double2(fx_out_slow((long long)re[i], K), fx_out_slow((long long)im[i], K));
    }
  };
  const bool redo = E::kId != EngF64::kId && (slow || special);
  // Small sizes with at most 4 points per thread: the slow values replace the
  // fixed-point words in place (one branch; the words are few, so this costs
  // no registers), and the stores select the words or the fast conversion.
  constexpr bool IN_PLACE = E::kId != EngF64::kId && FxTrunc<N>::value && P <= 4;
  if constexpr (IN_PLACE) {
    if (redo) {
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const double2 v = slow_value(i);
        re[i] = __double_as_longlong(v.x);
        im[i] = __double_as_longlong(v.y);
      }
    }
  }
  auto stored = [&](int i) -> double2 {
    if constexpr (IN_PLACE) {
      return redo ? make_double2(__longlong_as_double(re[i]), __longlong_as_double(im[i])) : value(i);
    } else {
      return redo ? slow_value(i) : value(i);
    }
  };
  if constexpr (F::STAGED) {
    if constexpr (NS > 1) __syncthreads();
#pragma unroll
    for (int b = 0; b < BL; ++b)
#pragma unroll
      for (int m = 0; m < RL; ++m) {
        const double2 v = stored(b + BL * m);
        sm[F::slot(j, F::template dest<NS - 1>(t, b, m))] =
            make_longlong2(__double_as_longlong(v.x), __double_as_longlong(v.y));
      }
    __syncthreads();
    for (int idx = tid; idx < (hold ? 0 : tile_elems); idx += F::THREADS) {
      const int jj = idx / N, e = idx - jj * N;
      const longlong2 v = sm[F::slot(jj, e)];
      *tl.out_elem(idx, jj, e) = make_double2(__longlong_as_double(v.x), __longlong_as_double(v.y));
    }
  } else {
    if (active && !hold) {
      double2* dst = tl.out_of(j);
      if constexpr (FxTrunc<N>::value) {
#pragma unroll
        for (int b = 0; b < BL; ++b)
#pragma unroll
          for (int m = 0; m < RL; ++m)
            dst[F::template dest<NS - 1>(t, b, m)] = stored(b + BL * m);
      } else if (!redo) {
#pragma unroll
        for (int b = 0; b < BL; ++b) {
          double2* q = dst + F::template dest<NS - 1>(t, b, 0);
#pragma unroll
          for (int m = 0; m < RL; ++m) q[m * PL::span(NS - 1)] = value(b + BL * m);
        }
      } else {
#pragma unroll
        for (int b = 0; b < BL; ++b)
#pragma unroll
          for (int m = 0; m < RL; ++m) dst[F::template dest<NS - 1>(t, b, m)] = slow_value(b + BL * m);
      }
    }
  }
  if constexpr (E::kId == EngF64::kId && NS > 1) {
    if (hold) F::redo_ranged(tl.in_of(j), tl.out_of(j), active, tw, sm, reinterpret_cast<int*>(smem_raw + TPB * F::NP * 16));
  }
}


// The batched kernel: CTA b transforms transforms [b*TPB, b*TPB + TPB).
// in and out may be the same buffer (in place): a CTA reads only the tile it
// writes, and every load of that tile (registers, or the shared staging
// buffer) happens before its first store, which is what the __restrict__
// qualifiers rely on; the tests run every plan in place.
// Its body is fft_tile's with contiguous addressing written out: routed
// through fft_tile it computes the same results but compiled to code measured
// 2.5-4% slower at N=64 and N=512, so the two are kept separate and the tests
// check them against each other bit for bit.
template <class E, class PL>
__global__ void __launch_bounds__(Fft<E, PL>::THREADS, PL::MINB)
fft_fwd_kernel(const double2* __restrict__ in, double2* __restrict__ out, long long batch,
               const typename E::TW* __restrict__ tw, int* __restrict__ err, int prefetch) {
  (void)err;  // no waits in this kernel; the argument keeps one launch signature
  using EK = PlanEngine<E, PL>;
  using F = Fft<EK, PL>;
  using S = typename EK::S;
  constexpr int N = PL::N, TPB = PL::TPB;
  constexpr int P = F::P, T = F::T, NS = F::NS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  longlong2* sm = reinterpret_cast<longlong2*>(smem_raw);

  after_previous();
  allow_next();
  if constexpr (PL::PREFETCH) {
    if (threadIdx.x == 0 && prefetch && batch * (PL::N * 16) >= PL::PREFETCH_MIN_BYTES) {
      // the tile of the CTA that starts one full wave later, into L2
      unsigned nsm;
      asm("mov.u32 %0, %%nsmid;" : "=r"(nsm));
      const long long first = ((long long)blockIdx.x + (long long)nsm * PL::MINB) * TPB;
      if (first < batch) {
        const long long cnt = batch - first < TPB ? batch - first : TPB;
        const char* p = reinterpret_cast<const char*>(in + first * N);
        long long bytes = cnt * N * 16;
        while (bytes > 0) {  // pieces of at most 64 KiB; 16-byte aligned multiples of 16
          const unsigned b = bytes > 65536 ? 65536u : (unsigned)bytes;
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(b) : "memory");
          p += b;
          bytes -= b;
        }
      }
    }
  }

  const int tid = threadIdx.x;
  const int j = tid / T;
  const int t = tid - j * T;
  const long long tile0 = (long long)blockIdx.x * TPB;
  const long long tr = tile0 + j;
  const bool active = TPB == 1 || tr < batch;  // the grid has one CTA per tile
  const long long tile_elems = (min((long long)TPB, batch - tile0)) * N;

  // ---- load raw binary64 points: point i of this thread is element t + T*i
  double2 raw[P];
  if constexpr (F::STAGED) {
    const double2* src = in + tile0 * N;
    for (int idx = tid; idx < tile_elems; idx += F::THREADS) {
      const int jj = idx / N, e = idx - jj * N;
      const double2 v = load_point(src + idx);
      sm[F::slot(jj, e)] = make_longlong2(__double_as_longlong(v.x), __double_as_longlong(v.y));
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const longlong2 v = sm[F::slot(j, t + T * i)];
      raw[i] = make_double2(__longlong_as_double(v.x), __longlong_as_double(v.y));
    }
  } else {
    // threads past the batch load its last transform: no zero fill for
    // predicated loads (2 instructions a point at N >= 64), and no zeros, which
    // take the general conversion (1.5 us of a single transform of 16 points)
    const double2* src = in + (TPB == 1 || active ? tr : batch - 1) * N + t;
#pragma unroll
    for (int i = 0; i < P; ++i) raw[i] = load_point(src + T * i);
  }

  S re[P], im[P];
  int K = 0, kshift = 0;
  bool slow = false, special = false;
  if constexpr (E::kId == EngF64::kId) {
#pragma unroll
    for (int i = 0; i < P; ++i) { re[i] = raw[i].x; im[i] = raw[i].y; }
  } else {
    // largest biased exponent of the transform, smallest of this thread
    constexpr bool TR = FxTrunc<N>::value;
    int em, emin;
    fx_exponent_range<P, TR>(raw, em, emin);
    em = fx_transform_max<T, TPB>(em, tid, j, reinterpret_cast<int*>(smem_raw + TPB * F::NP * 16));
    const FxScale sc = fx_size_scale<EK, N>(em);
    special = sc.special;
    K = sc.K;
    kshift = sc.kshift;
    slow = sc.slow;
    fx_convert_in<P, PL::OUTLINE_SLOW_IN, TR, FxFar<N>::value>(raw, re, im, sc.eref, emin);
  }

  if constexpr (F::STAGED) __syncthreads();  // staging buffer is reused by the passes
  // binary64: a transform of the CTA has to be redone (nothing is stored before);
  // a transform that one thread holds is scaled where it is
  bool hold = false, scaled = false;
  if constexpr (E::kId == EngF64::kId && NS > 1) {
    hold = F::run_voted(re, im, active, j, t, tw, sm);
  } else {
    if constexpr (E::kId == EngF64::kId) {
      scaled = f64_exponent(re, im) > F64Range<N>::top;
      if (scaled) f64_scale_down<F64Range<N>::down>(re, im);
    }
    F::template run_passes<0>(re, im, j, t, tw, sm);
    if constexpr (E::kId == EngF64::kId) {
      if (scaled) f64_scale_up<F64Range<N>::down>(re, im);
    }
  }

  // ---- store: output m of butterfly b of the last pass is element dest(...)
  constexpr int RL = PL::R[NS - 1];
  constexpr int BL = P / RL;
  // Fixed point: the rare transforms whose outputs leave the normal range, or
  // whose inputs were not finite, take the slow conversion: a per-value select
  // where the output is staged or the size is small (FxTrunc; both measured
  // faster so), else one branch per thread between two store loops.
  auto value = [&](int i) -> double2 {
    if constexpr (E::kId == EngF64::kId) {
      return make_double2(re[i], im[i]);
    } else {
      return make_double2(fx_out<PL::OUT_HI_ZERO>((long long)re[i], kshift),
                          fx_out<PL::OUT_HI_ZERO>((long long)im[i], kshift));
    }
  };
  auto slow_value = [&](int i) -> double2 {
    if constexpr (E::kId == EngF64::kId) {
      return make_double2(re[i], im[i]);
    } else {
      const double qnan = __longlong_as_double(0x7FF8000000000000LL);
      return special ? make_double2(qnan, qnan)
                     : make_double2(fx_out_slow((long long)re[i], K), fx_out_slow((long long)im[i], K));
    }
  };
  const bool redo = E::kId != EngF64::kId && (slow || special);
  // Small sizes with at most 4 points per thread: the slow values replace the
  // fixed-point words in place (one branch; the words are few, so this costs
  // no registers), and the stores select the words or the fast conversion.
  constexpr bool IN_PLACE = E::kId != EngF64::kId && FxTrunc<N>::value && P <= 4;
  if constexpr (IN_PLACE) {
    if (redo) {
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const double2 v = slow_value(i);
        re[i] = __double_as_longlong(v.x);
        im[i] = __double_as_longlong(v.y);
      }
    }
  }
  auto stored = [&](int i) -> double2 {
    if constexpr (IN_PLACE) {
      return redo ? make_double2(__longlong_as_double(re[i]), __longlong_as_double(im[i])) : value(i);
    } else {
      return redo ? slow_value(i) : value(i);
    }
  };
  if constexpr (F::STAGED) {
    if constexpr (NS > 1) __syncthreads();
#pragma unroll
    for (int b = 0; b < BL; ++b)
#pragma unroll
      for (int m = 0; m < RL; ++m) {
        const double2 v = stored(b + BL * m);
        sm[F::slot(j, F::template dest<NS - 1>(t, b, m))] =
            make_longlong2(__double_as_longlong(v.x), __double_as_longlong(v.y));
      }
    __syncthreads();
    double2* dst = out + tile0 * N;
    for (int idx = tid; idx < (hold ? 0 : tile_elems); idx += F::THREADS) {
      const int jj = idx / N, e = idx - jj * N;
      const longlong2 v = sm[F::slot(jj, e)];
      dst[idx] = make_double2(__longlong_as_double(v.x), __longlong_as_double(v.y));
    }
  } else {
    if (TPB == 1 ? active : active && !hold) {
      double2* dst = out + tr * N;
      if constexpr (FxTrunc<N>::value) {
#pragma unroll
        for (int b = 0; b < BL; ++b)
#pragma unroll
          for (int m = 0; m < RL; ++m)
            dst[F::template dest<NS - 1>(t, b, m)] = stored(b + BL * m);
      } else if (!redo) {
#pragma unroll
        for (int b = 0; b < BL; ++b) {
          double2* q = dst + F::template dest<NS - 1>(t, b, 0);
#pragma unroll
          for (int m = 0; m < RL; ++m)
            if constexpr (E::kId == EngF64::kId && TPB == 1) store_point_if(q + m * PL::span(NS - 1), value(b + BL * m), !hold);
            else q[m * PL::span(NS - 1)] = value(b + BL * m);
        }
      } else {
#pragma unroll
        for (int b = 0; b < BL; ++b)
#pragma unroll
          for (int m = 0; m < RL; ++m) dst[F::template dest<NS - 1>(t, b, m)] = slow_value(b + BL * m);
      }
    }
  }
  if constexpr (E::kId == EngF64::kId && NS > 1) {
    if (hold) F::redo_ranged(in + tr * N, out + tr * N, active, tw, sm, reinterpret_cast<int*>(smem_raw + TPB * F::NP * 16));
  }
}

}  // namespace fftoc
