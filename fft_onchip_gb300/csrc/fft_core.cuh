// fftoc — batched forward complex FFTs (N = 8..4096) for GB300 (sm_103a).
//
// Device core shared by every engine.  A transform of N points is computed by
// T = N / P threads, each holding P points in registers.  Each pass of radix R
// is one Stockham step (the structure of the reference's radix-8 executor,
// includes/legacy8_fft.cuh:57-119): butterfly t' reads x[t' + m*N/R],
// multiplies input m by W_{R*p}^{k*m} (k = t' mod p, p = product of earlier
// radices), runs an R-point DFT and writes y[(t'-k)*R + k + m*p].  Passes are
// joined through shared memory; the first pass reads HBM and the last writes
// HBM, both coalesced (consecutive threads touch consecutive 16-byte points).
//
// Engines (arithmetic used inside the transform; input/output are always
// interleaved binary64 complex values):
//   EngF64 — IEEE binary64 (DFMA/DADD).
//   EngFx  — 64-bit block fixed point.  Each transform is scaled by a power of
//            two taken from its largest exponent so that no value can overflow
//            (headroom for the worst-case growth of N), adds are exact 64-bit
//            integer adds, and products use 32 x 32 -> 64 multiplies: on 30-bit
//            limbs for N <= 32 (EngFxT), on the natural 32-bit words from
//            N = 64 up (EngFxN).  The conversion back to binary64 rounds once
//            (cvt.rn.f64.s64).
#pragma once
#include <type_traits>
#include <cstdint>
#include <cuda_runtime.h>

#define FFTOC_HD __host__ __device__ __forceinline__

namespace fftoc {

// ---------------------------------------------------------------------------
// Plans: a transform of N points is split over T = N/P threads holding P
// points each, and computed in passes of radix R[0], R[1], ... (product N,
// every R dividing P).  T threads per transform, TPB transforms per CTA.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int ilog2c(int n) { return n <= 1 ? 0 : 1 + ilog2c(n / 2); }

template <int N_, int P_, int TPB_, int R0, int R1 = 1, int R2 = 1, int R3 = 1, int MINB_ = 1>
struct PlanT {
  static constexpr int N = N_;
  static constexpr int P = P_;
  static constexpr int TPB = TPB_;
  static constexpr int MINB = MINB_;  // minimum resident CTAs per SM (register budget)
  static constexpr bool PREFETCH = false;  // batched kernel: L2 prefetch one wave ahead (Prefetched<>)
  static constexpr long long PREFETCH_MIN_BYTES = 0;  // ... for batches of at least this much input
  static constexpr bool OUTLINE_SLOW_IN = false;  // batched kernel: rare input path out of line (OutlinedSlowIn<>)
  static constexpr bool IMAD_SPLIT = false;  // fixed point: low limbs by integer multiply-add (ImadSplit<>)
  static constexpr bool OUT_HI_ZERO = false;  // fixed point: zero test on the converted word (OutHiZero<>)
  static constexpr bool NO_STAGE = false;  // fewer than 8 threads per transform: direct HBM access (NoStage<>)
  static constexpr bool UNEVEN_DEFAULT = false;  // the uneven path's default plan for its size (UnevenDefault<>)
  static constexpr int SMALL_PER_SM = 0;  // the size's plan for small batches (SmallBatch<>)
  static constexpr int R[4] = {R0, R1, R2, R3};
  static constexpr int S = (R0 > 1) + (R1 > 1) + (R2 > 1) + (R3 > 1);
  static constexpr int T = N / P;
  static_assert(R0 * R1 * R2 * R3 == N, "radices must multiply to N");
  static_assert(P % R0 == 0 && P % R1 == 0 && P % R2 == 0 && P % R3 == 0, "every radix divides P");
  // span p of pass s (product of the radices before it)
  __host__ __device__ static constexpr int span(int s) {
    int p = 1;
    for (int i = 0; i < s; ++i) p *= R[i];
    return p;
  }
  // offset (in twiddle entries) of pass s's table; pass s holds (R-1)*p
  // entries, entry (m-1)*p + k = W_{R p}^{k m}.  Pass 0 has no twiddles.
  __host__ __device__ static constexpr int tw_offset(int s) {
    int off = 0;
    for (int i = 1; i < s; ++i) off += (R[i] - 1) * span(i);
    return off;
  }
  static constexpr int TW_COUNT = tw_offset(S);
};

// ---------------------------------------------------------------------------
// Engines
// ---------------------------------------------------------------------------
struct EngF64 {
  using S = double;
  using TW = double2;   // (cos, -sin) of the twiddle, or its tangent form (twiddled_sum)
  static constexpr int kId = 1;
  static constexpr bool kNatural = false;
  FFTOC_HD static S add(S a, S b) { return a + b; }
  FFTOC_HD static S sub(S a, S b) { return a - b; }
  FFTOC_HD static S add3(S a, S b, S c) { return (a + b) + c; }
  FFTOC_HD static S addsub(S a, S b, S c) { return (a + b) - c; }
  FFTOC_HD static S subadd(S a, S b, S c) { return (a - b) + c; }
  FFTOC_HD static S sub3(S a, S b, S c) { return (a - b) - c; }
  FFTOC_HD static void cmul(S& xr, S& xi, const TW w) {
    const double r = fma(xr, w.x, -xi * w.y);
    const double i = fma(xr, w.y, xi * w.x);
    xr = r;
    xi = i;
  }
  // The tangent form of w = c + j s (the FFT for fused multiply-add machines of
  // Linzer and Feig, 1993): w x = a y with y two multiply-adds,
  //   |s| <= |c|: a = c, b = s / c,  y = x + j b x,
  //   else:       a = s, b = -c / s, y = j x + j b (j x),
  // and A + w x, A - w x then four more: a radix-2 butterfly in 6 instructions
  // and two roundings per output instead of 8 and three.  Which form an entry
  // has follows from its place in the table (tangent_turned).
  FFTOC_HD static void twiddled_sum(S& ar, S& ai, S& xr, S& xi, const TW w, bool turned) {
    const double p = turned ? -xi : xr, q = turned ? xr : xi;
    const double yr = fma(-w.y, q, p), yi = fma(w.y, p, q);
    xr = fma(-w.x, yr, ar);
    xi = fma(-w.x, yi, ai);
    ar = fma(w.x, yr, ar);
    ai = fma(w.x, yi, ai);
  }
  // whether e^(-2 pi j i / n) is nearer to the imaginary axis; i < n, n >= 2
  // a power of two
  FFTOC_HD static bool tangent_turned(int i, int n) { return ((8u * (unsigned)i / (unsigned)n + 1u) & 2u) != 0; }
};

// Limbs of a fixed-point constant: v*2^60 = h*2^30 + l, 0 <= l < 2^30.
struct FxKC {
  int h, l;
};

// IMAD_SPLIT selects how the low limb of a split is formed (a logic op or an
// integer multiply-add: same value, different pipe); the plans choose the form
// that measured faster.
template <bool IMAD_SPLIT = false>
struct EngFxT {
  using S = long long;
  using TW = int4;      // (wr.h, wr.l, wi.h, wi.l): w*2^60 = h*2^30 + l, 0 <= l < 2^30
  using KC = FxKC;
  static constexpr int kId = 2;
  static constexpr bool kNatural = false;
  FFTOC_HD static S add(S a, S b) { return a + b; }
  FFTOC_HD static S sub(S a, S b) { return a - b; }
  // Three-operand sums as one PTX sequence each: the front end cannot share
  // partial sums between outputs, so ptxas can emit a fused 3-input add pair.
#ifdef __CUDA_ARCH__
  FFTOC_HD static S add3(S a, S b, S c) {
    S r;
    asm("add.s64 %0, %1, %2;\n\tadd.s64 %0, %0, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
  }
  FFTOC_HD static S addsub(S a, S b, S c) {
    S r;
    asm("add.s64 %0, %1, %2;\n\tsub.s64 %0, %0, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
  }
  FFTOC_HD static S subadd(S a, S b, S c) {
    S r;
    asm("sub.s64 %0, %1, %2;\n\tadd.s64 %0, %0, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
  }
  FFTOC_HD static S sub3(S a, S b, S c) {
    S r;
    asm("sub.s64 %0, %1, %2;\n\tsub.s64 %0, %0, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
  }
#else
  static S add3(S a, S b, S c) { return a + b + c; }
  static S addsub(S a, S b, S c) { return a + b - c; }
  static S subadd(S a, S b, S c) { return a - b + c; }
  static S sub3(S a, S b, S c) { return a - b - c; }
#endif
  // Limbs of a value, |x| < 2^61: x = xh*2^30 + xl, |xh| < 2^31, 0 <= xl < 2^30.
  FFTOC_HD static void split(S x, int& xh, int& xl) {
    xh = (int)(x >> 30);
#ifdef __CUDA_ARCH__
    if constexpr (IMAD_SPLIT) {  // lo32(x) - xh * 2^30 (mod 2^32)
      asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(xl) : "r"(xh), "r"(0xC0000000u), "r"((unsigned)x));
      return;
    }
#endif
    xl = (int)((unsigned)x & 0x3FFFFFFFu);
  }
  // a*b + c with a, b 32-bit and c 64-bit: one IMAD.WIDE (spelled out in PTX;
  // written as (long long)a * b + c the front end may emit a 64x64 multiply)
  FFTOC_HD static S madw(int a, int b, S c) {
#ifdef __CUDA_ARCH__
    S d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
#else
    return (S)a * (S)b + c;
#endif
  }
  // a*b with a, b 32-bit: one IMAD.WIDE without an addend
  FFTOC_HD static S mulw(int a, int b) {
#ifdef __CUDA_ARCH__
    S d;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
    return d;
#else
    return (S)a * (S)b;
#endif
  }
  // x * c for a real constant, |c| <= 1:
  //   x*c = xh*ch + (xh*cl + xl*ch) / 2^30 + xl*cl/2^60   (last term < 1, dropped)
  // |xh*cl| < 2^61, |xl*ch| <= 2^60, so the middle sum cannot overflow.  The
  // middle sum is shifted without a rounding constant (floor): the product is
  // within 2 units of the exact value, and a chain that opens with a plain
  // multiply measured 2-4 % faster than one that opens with a 64-bit addend.
  FFTOC_HD static S mulc(S x, KC k) {
    int xh, xl;
    split(x, xh, xl);
    const long long m = madw(xl, k.h, mulw(xh, k.l));
    return madw(xh, k.h, m >> 30);
  }
  // (xr + i xi) * (wr + i wi); each middle sum has four terms of magnitude
  // < 2^61 or <= 2^60, so |m| < 1.5 * 2^62.
  FFTOC_HD static void cmul_limbs(S& xr, S& xi, int wrh, int wrl, int wih, int wil) {
    int rh, rl, ih, il;
    split(xr, rh, rl);
    split(xi, ih, il);
    // negate the twiddle limbs (|wih| <= 2^30, 0 <= wil < 2^30), never the
    // data limbs (ih may be -2^31)
    const int nwih = -wih, nwil = -wil;
    const long long mr = madw(il, nwih, madw(ih, nwil, madw(rl, wrh, mulw(rh, wrl))));
    const long long mi = madw(il, wrh, madw(ih, wrl, madw(rl, wih, mulw(rh, wil))));
    xr = madw(ih, nwih, madw(rh, wrh, mr >> 30));
    xi = madw(ih, wrh, madw(rh, wih, mi >> 30));
  }
  FFTOC_HD static void cmul(S& xr, S& xi, const int4 w) { cmul_limbs(xr, xi, w.x, w.y, w.z, w.w); }
  FFTOC_HD static void cmulk(S& xr, S& xi, KC c, KC s) { cmul_limbs(xr, xi, c.h, c.l, s.h, s.l); }
};
using EngFx = EngFxT<false>;

// Fixed point on the natural 32-bit words (transforms of N >= 64).  A value is
// split as x = xh * 2^32 + xl with xl its low word read as signed, so a split
// costs one instruction (the low word's sign carried into the high word).
//
// Twiddles are held as w * 2^62 = wh * 2^32 + wl, and a product takes three
// real products instead of four:
//   k1 = wr (xr + xi),  yr = k1 - xi (wr + wi),  yi = k1 + xr (wi - wr),
// the sums and differences of w's parts from the table.  It comes at quarter
// scale, x * w / 4, where the middle sum's high word is its share of the
// result with no funnel shift, or at full scale for two more instructions a
// component.  Transforms that have to give up low bits to the growth of N
// anyway do so in their first passes with twiddles (FxPasses): the input is
// converted at 53 bits for every N, and the last pass has at least the bits
// that a conversion at the final scale from the start would leave.
// The kernels are bound by the integer pipes.  Per warp and SM quadrant a
// 32 x 32 -> 64 multiply takes four cycles of the FMA-heavy pipe and two of
// the ALU (both measured by mixing it with ALU instructions), every other
// integer instruction two cycles of one of them, so fewer and narrower
// instructions are what counts: a product is 9 multiplies and about 9 others
// at quarter scale, against 12 and about 17 with the 30-bit limbs of EngFxT
// (hardware counters over a kernel of products alone: 18.7 against 29).
// With the slots and exponent range of fft_kernel.cuh, 1 GiB of input, on one
// GB300: N = 512 430 -> 371 us (5.0 -> 5.8 TB/s), N = 4096 626 -> 576 us,
// N = 1024 (82 MB) 47.1 -> 41.0 us.
struct EngFxN {
  using S = long long;
  using TW = int4;  // limbs (h, l) of wr and of wi - wr; those of -(wr + wi) in an int2 table behind
  static constexpr int kId = 2;
  static constexpr bool kNatural = true;
  FFTOC_HD static S add(S a, S b) { return a + b; }
  FFTOC_HD static S sub(S a, S b) { return a - b; }
  FFTOC_HD static S add3(S a, S b, S c) { return EngFx::add3(a, b, c); }
  FFTOC_HD static S addsub(S a, S b, S c) { return EngFx::addsub(a, b, c); }
  FFTOC_HD static S subadd(S a, S b, S c) { return EngFx::subadd(a, b, c); }
  FFTOC_HD static S sub3(S a, S b, S c) { return EngFx::sub3(a, b, c); }
  FFTOC_HD static void split(S x, int& xh, int& xl) {
    xl = (int)(unsigned)x;
    xh = (int)((unsigned long long)x >> 32) + (int)((unsigned)x >> 31);
  }
  // a * b, 32 x 32 -> 64.  Sums of products are written as plain 64-bit
  // additions of these: the assembler then fuses each addition into a
  // multiply-add where that is cheaper.  Spelled out as mad.wide chains the
  // same product took 25 instructions instead of 19.
  FFTOC_HD static S mul(int a, int b) { return EngFx::mulw(a, b); }
  // x * w, or x * w / 4 (QUARTER); |xr + j xi| <= 2^61.5: the middle sums stay
  // below (sqrt(5) + 1 + sqrt(1/2)) * 2^61 < 2^63.
  template <bool QUARTER>
  FFTOC_HD static void cmul(S& xr, S& xi, const int4 w, const int2 c) {
    int rh, rl, ih, il, sh, sl;
    split(xr, rh, rl);
    split(xi, ih, il);
    split(xr + xi, sh, sl);
    const S m = mul(sl, w.x) + mul(sh, w.y), h = mul(sh, w.x);
    const S mr = mul(il, c.x) + mul(ih, c.y) + m;
    const S mi = mul(rl, w.z) + mul(rh, w.w) + m;
    const S hr = mul(ih, c.x) + h, hi = mul(rh, w.z) + h;
    if constexpr (QUARTER) {
      xr = hr + (mr >> 32);
      xi = hi + (mi >> 32);
    } else {
      xr = (S)((unsigned long long)hr << 2) + (mr >> 30);
      xi = (S)((unsigned long long)hi << 2) + (mi >> 30);
    }
  }
  // x * sqrt(1/2) = x + x * (sqrt(1/2) - 1), full scale
  FFTOC_HD static S mulh(S x) {
    constexpr FxKC V = {-1257966796, -102865788};
    int xh, xl;
    split(x, xh, xl);
    const S m = mul(xl, V.h) + mul(xh, V.l);
    return mul(xh, V.h) + x + (m >> 32);
  }
  // (r, i) -> (c r + s i, c i - s r), c = cos(pi/8), s = sin(pi/8), full scale:
  // with t = s (r + i), c r + s i = r + (t + (c - s - 1) r) and
  // c i - s r = i - (t + (1 - c - s) i); constants v as v * 2^64 = h * 2^32 + l,
  // l signed.  |r + j i| <= 2^59.5 keeps the middle sums below 2^63.
  FFTOC_HD static void rot8(S& r, S& i) {
    constexpr FxKC S8 = {1643612827, -1163556025}, E = {-1970547745, -641423873}, F = {-1316677908, -1326431372};
    int rh, rl, ih, il, sh, sl;
    split(r, rh, rl);
    split(i, ih, il);
    split(r + i, sh, sl);
    const S m = mul(sl, S8.h) + mul(sh, S8.l), h = mul(sh, S8.h);
    const S mr = mul(rl, E.h) + mul(rh, E.l) + m;
    const S mi = mul(il, F.h) + mul(ih, F.l) + m;
    r = r + mul(rh, E.h) + h + (mr >> 32);
    i = i - (mul(ih, F.h) + h + (mi >> 32));
  }
};

// Smallest N on the natural words; below it the kernels stream at the HBM
// rate (EngFxT) and their register budgets are full.
constexpr int kNaturalMinN = 64;

// constants of the DFT kernels, per engine
template <class E> struct Konst;
// Fixed-point limbs of sqrt(1/2), cos(pi/8) and sin(pi/8): v*2^60 = h*2^30 + l, 0 <= l < 2^30.
template <bool B> struct Konst<EngFxT<B>> {
  FFTOC_HD static FxKC h() { return {759250124, 1067312712}; }
  FFTOC_HD static FxKC nh() { return {-759250125, 6429112}; }
  FFTOC_HD static FxKC c8() { return {992008094, 424059668}; }
  FFTOC_HD static FxKC s8() { return {410903206, 732584116}; }
  FFTOC_HD static FxKC nc8() { return {-992008095, 649682156}; }
  FFTOC_HD static FxKC ns8() { return {-410903207, 341157708}; }
};

// A plan whose batched kernel also prefetches, into L2, the tile of the CTA
// that starts one full wave (SMs x MINB CTAs) later, for batches of at least
// MIN_MIB MiB of input (below that the prefetch measured slower at some sizes:
// N = 64 by 16 % at 64 MiB, N = 4096 by 1-2 % up to 256 MiB).
template <class PL, int MIN_MIB = 0>
struct Prefetched : PL {
  static constexpr bool PREFETCH = true;
  static constexpr long long PREFETCH_MIN_BYTES = (long long)MIN_MIB << 20;
};

// A plan whose batched kernel converts the rare transforms that leave the
// fast binary64 -> fixed-point input path through an out-of-line function
// (otherwise the compiler may if-convert that path into the fast one).
template <class PL>
struct OutlinedSlowIn : PL {
  static constexpr bool OUTLINE_SLOW_IN = true;
};

// A plan whose fixed-point splits form the low limb with an integer
// multiply-add instead of a mask (moves work from the ALU pipe to the FMA pipe).
template <class PL>
struct ImadSplit : PL {
  static constexpr bool IMAD_SPLIT = true;
};

// A plan whose output conversion tests the converted value's high word for
// zero instead of the 64-bit integer (one compare less per value).
template <class PL>
struct OutHiZero : PL {
  static constexpr bool OUT_HI_ZERO = true;
};

// A plan with fewer than 8 threads per transform that loads and stores HBM
// directly instead of staging its tile through shared memory.  With T
// threads per transform each warp access still covers whole 32-byte sectors
// for T >= 2; it pays off where the staging round trip costs more than the
// spread of the access (measured: T = 4).
template <class PL>
struct NoStage : PL {
  static constexpr bool NO_STAGE = true;
};

// The plan the uneven-batch path uses for its size while the size's plan
// choice is the library default (its persistent kernels measured faster
// with it than with the batched default).
template <class PL>
struct UnevenDefault : PL {
  static constexpr bool UNEVEN_DEFAULT = true;
};

// The plan of batches of up to PER_SM transforms per SM while the size's plan
// choice is the library default.  Such grids take about as long as one CTA, so
// these plans have fewer points per thread (shorter chains, more warps to
// share the FP64 pipe's conversions) or more registers than full SMs allow.
template <class PL, int PER_SM>
struct SmallBatch : PL {
  static constexpr int SMALL_PER_SM = PER_SM;
};

// The engine a plan's kernels compute with: the fixed-point engine in the
// plan's split form, or E unchanged.
template <class E, class PL>
using PlanEngine = typename std::conditional<
    E::kId != EngFx::kId, E,
    typename std::conditional<(PL::N >= kNaturalMinN), EngFxN,
                              typename std::conditional<PL::IMAD_SPLIT, EngFxT<true>, E>::type>::type>::type;

// ---------------------------------------------------------------------------
// Small forward DFTs on registers.  re[i], im[i] at compile-time indices
// base + stride*m, in place, natural order.
// ---------------------------------------------------------------------------
template <class E, int B, int ST, int PP>
FFTOC_HD void dft2(typename E::S (&re)[PP], typename E::S (&im)[PP]) {
  using S = typename E::S;
  const S ar = re[B], ai = im[B], br = re[B + ST], bi = im[B + ST];
  re[B] = E::add(ar, br); im[B] = E::add(ai, bi);
  re[B + ST] = E::sub(ar, br); im[B + ST] = E::sub(ai, bi);
}

// 4-point DFT of (x0, x1, x2, x3): with t = x1 + x3 and u = x1 - x3,
//   y0 = x0 + x2 + t, y2 = x0 + x2 - t, y1 = x0 - x2 - i*u, y3 = x0 - x2 + i*u,
// every output one three-operand sum.
template <class E>
FFTOC_HD void dft4_core(typename E::S x0r, typename E::S x0i, typename E::S x1r, typename E::S x1i,
                        typename E::S x2r, typename E::S x2i, typename E::S x3r, typename E::S x3i,
                        typename E::S& y0r, typename E::S& y0i, typename E::S& y1r, typename E::S& y1i,
                        typename E::S& y2r, typename E::S& y2i, typename E::S& y3r, typename E::S& y3i) {
  using S = typename E::S;
  const S tr = E::add(x1r, x3r), ti = E::add(x1i, x3i);
  const S ur = E::sub(x1r, x3r), ui = E::sub(x1i, x3i);
  y0r = E::add3(x0r, x2r, tr);
  y0i = E::add3(x0i, x2i, ti);
  y2r = E::addsub(x0r, x2r, tr);
  y2i = E::addsub(x0i, x2i, ti);
  y1r = E::subadd(x0r, x2r, ui);
  y1i = E::sub3(x0i, x2i, ur);
  y3r = E::sub3(x0r, x2r, ui);
  y3i = E::subadd(x0i, x2i, ur);
}

template <class E, int B, int ST, int PP>
FFTOC_HD void dft4(typename E::S (&re)[PP], typename E::S (&im)[PP]) {
  dft4_core<E>(re[B], im[B], re[B + ST], im[B + ST], re[B + 2 * ST], im[B + 2 * ST], re[B + 3 * ST], im[B + 3 * ST],
               re[B], im[B], re[B + ST], im[B + ST], re[B + 2 * ST], im[B + 2 * ST], re[B + 3 * ST], im[B + 3 * ST]);
}

// 8-point DFT: a_m = x_m + x_{m+4}, b_m = (x_m - x_{m+4}) W8^m; even outputs
// are DFT4(a), odd outputs DFT4(b).  W8^1 and W8^3 are real-constant
// products (sqrt(1/2)); W8^2 = -i is folded into the odd DFT4's signs.
template <class E, int B, int ST, int PP>
FFTOC_HD void dft8(typename E::S (&re)[PP], typename E::S (&im)[PP]) {
  using S = typename E::S;
  using K = Konst<E>;
  S ar[4], ai[4], br[4], bi[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    ar[m] = E::add(re[B + m * ST], re[B + (m + 4) * ST]);
    ai[m] = E::add(im[B + m * ST], im[B + (m + 4) * ST]);
    br[m] = E::sub(re[B + m * ST], re[B + (m + 4) * ST]);
    bi[m] = E::sub(im[B + m * ST], im[B + (m + 4) * ST]);
  }
  // b1 *= (1 - i)/sqrt2 ; b3 *= (-1 - i)/sqrt2
  const S b1r = E::mulc(E::add(br[1], bi[1]), K::h());
  const S b1i = E::mulc(E::sub(bi[1], br[1]), K::h());
  const S b3r = E::mulc(E::sub(bi[3], br[3]), K::h());
  const S b3i = E::mulc(E::add(br[3], bi[3]), K::nh());
  // even outputs X0, X2, X4, X6
  dft4_core<E>(ar[0], ai[0], ar[1], ai[1], ar[2], ai[2], ar[3], ai[3], re[B], im[B], re[B + 2 * ST], im[B + 2 * ST],
               re[B + 4 * ST], im[B + 4 * ST], re[B + 6 * ST], im[B + 6 * ST]);
  // odd outputs X1, X3, X5, X7: DFT4(b0, b1', b2', b3') with b2' = -i*b2 = (b2i, -b2r)
  {
    const S tr = E::add(b1r, b3r), ti = E::add(b1i, b3i);
    const S ur = E::sub(b1r, b3r), ui = E::sub(b1i, b3i);
    re[B + ST] = E::add3(br[0], bi[2], tr);
    im[B + ST] = E::subadd(bi[0], br[2], ti);
    re[B + 5 * ST] = E::addsub(br[0], bi[2], tr);
    im[B + 5 * ST] = E::sub3(bi[0], br[2], ti);
    re[B + 3 * ST] = E::subadd(br[0], bi[2], ui);
    im[B + 3 * ST] = E::addsub(bi[0], br[2], ur);
    re[B + 7 * ST] = E::sub3(br[0], bi[2], ui);
    im[B + 7 * ST] = E::add3(bi[0], br[2], ur);
  }
}

// 16-point DFT as 4 x 4: with n = 4*n1 + n2 and k = k1 + 4*k2,
//   X[k1 + 4 k2] = sum_n2 W4^(n2 k2) * (W16^(n2 k1) * sum_n1 x[4 n1 + n2] W4^(n1 k1)):
// four DFT4s over n1, the nine non-trivial W16^(n2 k1), four DFT4s over n2,
// and a transposition of the outputs (register renaming).
template <class E, int B, int ST, int PP>
FFTOC_HD void dft16(typename E::S (&re)[PP], typename E::S (&im)[PP]) {
  using S = typename E::S;
  using K = Konst<E>;
  // y[n2][k1] at B + (n2 + 4 k1) ST
  dft4<E, B, 4 * ST, PP>(re, im);
  dft4<E, B + ST, 4 * ST, PP>(re, im);
  dft4<E, B + 2 * ST, 4 * ST, PP>(re, im);
  dft4<E, B + 3 * ST, 4 * ST, PP>(re, im);
  auto at = [](int n2, int k1) { return B + (n2 + 4 * k1) * ST; };
  S r, i;
  // W16^1 = (c8, -s8)
  r = re[at(1, 1)]; i = im[at(1, 1)]; E::cmulk(r, i, K::c8(), K::ns8()); re[at(1, 1)] = r; im[at(1, 1)] = i;
  // W16^2 = (1 - i)/sqrt2, at (1, 2) and (2, 1)
  r = re[at(1, 2)]; i = im[at(1, 2)];
  re[at(1, 2)] = E::mulc(E::add(r, i), K::h()); im[at(1, 2)] = E::mulc(E::sub(i, r), K::h());
  r = re[at(2, 1)]; i = im[at(2, 1)];
  re[at(2, 1)] = E::mulc(E::add(r, i), K::h()); im[at(2, 1)] = E::mulc(E::sub(i, r), K::h());
  // W16^3 = (s8, -c8), at (1, 3) and (3, 1)
  r = re[at(1, 3)]; i = im[at(1, 3)]; E::cmulk(r, i, K::s8(), K::nc8()); re[at(1, 3)] = r; im[at(1, 3)] = i;
  r = re[at(3, 1)]; i = im[at(3, 1)]; E::cmulk(r, i, K::s8(), K::nc8()); re[at(3, 1)] = r; im[at(3, 1)] = i;
  // W16^4 = -i, at (2, 2)
  r = re[at(2, 2)]; i = im[at(2, 2)]; re[at(2, 2)] = i; im[at(2, 2)] = E::sub(S(0), r);
  // W16^6 = (-1 - i)/sqrt2, at (2, 3) and (3, 2)
  r = re[at(2, 3)]; i = im[at(2, 3)];
  re[at(2, 3)] = E::mulc(E::sub(i, r), K::h()); im[at(2, 3)] = E::mulc(E::add(r, i), K::nh());
  r = re[at(3, 2)]; i = im[at(3, 2)];
  re[at(3, 2)] = E::mulc(E::sub(i, r), K::h()); im[at(3, 2)] = E::mulc(E::add(r, i), K::nh());
  // W16^9 = (-c8, s8), at (3, 3)
  r = re[at(3, 3)]; i = im[at(3, 3)]; E::cmulk(r, i, K::nc8(), K::s8()); re[at(3, 3)] = r; im[at(3, 3)] = i;
  // DFT4 over n2 for each k1: inputs at B + (4 k1 + n2) ST, outputs X[k1 + 4 k2] at B + (4 k1 + k2) ST
  dft4<E, B, ST, PP>(re, im);
  dft4<E, B + 4 * ST, ST, PP>(re, im);
  dft4<E, B + 8 * ST, ST, PP>(re, im);
  dft4<E, B + 12 * ST, ST, PP>(re, im);
  S xr[16], xi[16];
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
      xr[k1 + 4 * k2] = re[B + (4 * k1 + k2) * ST];
      xi[k1 + 4 * k2] = im[B + (4 * k1 + k2) * ST];
    }
#pragma unroll
  for (int k = 0; k < 16; ++k) { re[B + k * ST] = xr[k]; im[B + k * ST] = xi[k]; }
}

// The 4-, 8- and 16-point DFTs of EngFxN.  The factors -i and -1 are folded
// into the signs of the sums; the constant products are mulh and rot8.
//
// 4-point DFT of (x0, x1, x2, x3) with x2 replaced by -i x2 (MI2), x3 by -i x3
// (MI3) or by -x3 (NEG3), outputs to y0..y3.
template <bool MI2, bool MI3, bool NEG3, class S>
FFTOC_HD void fxn_dft4(S x0r, S x0i, S x1r, S x1i, S x2r, S x2i, S x3r, S x3i, S& y0r, S& y0i, S& y1r, S& y1i, S& y2r,
                       S& y2i, S& y3r, S& y3i) {
  S tr, ti, ur, ui;  // x1 + x3, x1 - x3
  if constexpr (MI3) {
    tr = x1r + x3i; ti = x1i - x3r; ur = x1r - x3i; ui = x1i + x3r;
  } else if constexpr (NEG3) {
    tr = x1r - x3r; ti = x1i - x3i; ur = x1r + x3r; ui = x1i + x3i;
  } else {
    tr = x1r + x3r; ti = x1i + x3i; ur = x1r - x3r; ui = x1i - x3i;
  }
  S pr, pi, qr, qi;  // x0 + x2, x0 - x2
  if constexpr (MI2) {
    pr = x0r + x2i; pi = x0i - x2r; qr = x0r - x2i; qi = x0i + x2r;
  } else {
    pr = x0r + x2r; pi = x0i + x2i; qr = x0r - x2r; qi = x0i - x2i;
  }
  y0r = pr + tr; y0i = pi + ti;
  y2r = pr - tr; y2i = pi - ti;
  y1r = qr + ui; y1i = qi - ur;
  y3r = qr - ui; y3i = qi + ur;
}

template <bool MI2, bool MI3, bool NEG3, int B, int ST, int PP>
FFTOC_HD void fxn_dft4_at(long long (&re)[PP], long long (&im)[PP]) {
  fxn_dft4<MI2, MI3, NEG3>(re[B], im[B], re[B + ST], im[B + ST], re[B + 2 * ST], im[B + 2 * ST], re[B + 3 * ST],
                           im[B + 3 * ST], re[B], im[B], re[B + ST], im[B + ST], re[B + 2 * ST], im[B + 2 * ST],
                           re[B + 3 * ST], im[B + 3 * ST]);
}

// Sums and differences of x_m and x_{m+4}; W8 = (1 - i)/sqrt2 and W8^3 = -i W8
// on the odd half, whose inputs 2 and 3 then carry a factor -i each.
template <int B, int ST, int PP>
FFTOC_HD void fxn_dft8(long long (&re)[PP], long long (&im)[PP]) {
  using S = long long;
  S ar[4], ai[4], br[4], bi[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    ar[m] = re[B + m * ST] + re[B + (m + 4) * ST];
    ai[m] = im[B + m * ST] + im[B + (m + 4) * ST];
    br[m] = re[B + m * ST] - re[B + (m + 4) * ST];
    bi[m] = im[B + m * ST] - im[B + (m + 4) * ST];
  }
  const S b1r = EngFxN::mulh(br[1] + bi[1]), b1i = EngFxN::mulh(bi[1] - br[1]);
  const S b3r = EngFxN::mulh(br[3] + bi[3]), b3i = EngFxN::mulh(bi[3] - br[3]);
  fxn_dft4<false, false, false>(ar[0], ai[0], ar[1], ai[1], ar[2], ai[2], ar[3], ai[3], re[B], im[B], re[B + 2 * ST],
                                im[B + 2 * ST], re[B + 4 * ST], im[B + 4 * ST], re[B + 6 * ST], im[B + 6 * ST]);
  fxn_dft4<true, true, false>(br[0], bi[0], b1r, b1i, br[2], bi[2], b3r, b3i, re[B + ST], im[B + ST], re[B + 3 * ST],
                              im[B + 3 * ST], re[B + 5 * ST], im[B + 5 * ST], re[B + 7 * ST], im[B + 7 * ST]);
}

// dft16's 4 x 4 form.  Of the factors W16^(n2 k1): W^1 = rot8; W^2 = (1 - i)/sqrt2;
// W^3 (r, i) = (p, -q) with (p, q) = rot8(i, r); W^4 = -i; W^6 = -i W^2; W^9 = -W^1.
template <int B, int ST, int PP>
FFTOC_HD void fxn_dft16(long long (&re)[PP], long long (&im)[PP]) {
  using S = long long;
  fxn_dft4_at<false, false, false, B, 4 * ST, PP>(re, im);
  fxn_dft4_at<false, false, false, B + ST, 4 * ST, PP>(re, im);
  fxn_dft4_at<false, false, false, B + 2 * ST, 4 * ST, PP>(re, im);
  fxn_dft4_at<false, false, false, B + 3 * ST, 4 * ST, PP>(re, im);
  // y[n2][k1] at B + (n2 + 4 k1) ST
  auto at = [](int n2, int k1) { return B + (n2 + 4 * k1) * ST; };
  auto w1 = [&](int i) {
    S r = re[i], q = im[i];
    EngFxN::rot8(r, q);
    re[i] = r;
    im[i] = q;
  };
  auto w2 = [&](int i) {
    const S r = re[i], q = im[i];
    re[i] = EngFxN::mulh(r + q);
    im[i] = EngFxN::mulh(q - r);
  };
  auto w3 = [&](int i) {
    S q = im[i], r = re[i];
    EngFxN::rot8(q, r);
    re[i] = q;
    im[i] = -r;
  };
  w1(at(1, 1));
  w2(at(2, 1));
  w3(at(3, 1));
  w2(at(1, 2));
  w2(at(3, 2));  // times -i below; (2, 2) too
  w3(at(1, 3));
  w2(at(2, 3));  // times -i below
  w1(at(3, 3));  // times -1 below
  fxn_dft4_at<false, false, false, B, ST, PP>(re, im);
  fxn_dft4_at<false, false, false, B + 4 * ST, ST, PP>(re, im);
  fxn_dft4_at<true, true, false, B + 8 * ST, ST, PP>(re, im);
  fxn_dft4_at<true, false, true, B + 12 * ST, ST, PP>(re, im);
  S xr[16], xi[16];
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
      xr[k1 + 4 * k2] = re[B + (4 * k1 + k2) * ST];
      xi[k1 + 4 * k2] = im[B + (4 * k1 + k2) * ST];
    }
#pragma unroll
  for (int k = 0; k < 16; ++k) { re[B + k * ST] = xr[k]; im[B + k * ST] = xi[k]; }
}

// The DFTs of EngF64.  FP64 instructions issue at 1/64 of the FP32 rate, so
// these count them: every constant product is a multiply-add of the sum behind
// it, with a twiddle c (1 - j t) as x - j t x and c in the next sum.  144
// instructions for 16 points and 52 for 8, against 160 and 56 with the
// products by themselves.  Each has the radix-2 step over m and m + R/2 apart
// (f64_sums, or with twiddles EngF64::twiddled_sum), then this step.  16411
// transforms of 256 points 195 -> 174 us, 64 MiB of 64 to 4096 points 9 to 12 %
// less time; errors against long double are 2 to 4 % smaller at every size.
// Inside, values reach sqrt(2) times those of the plain products, as they do
// in W8 = H (1 - j): transforms that this could make overflow are scaled
// (F64Range).  The step takes the
// sums a_m at B + m ST and differences b_m at B + (m + R/2) ST, m < R/2, to
// the R outputs in natural order.
template <int R, int B, int ST, int PP>
FFTOC_HD void f64_sums(double (&re)[PP], double (&im)[PP]) {
#pragma unroll
  for (int m = 0; m < R / 2; ++m) {
    double &ar = re[B + m * ST], &ai = im[B + m * ST], &br = re[B + (m + R / 2) * ST], &bi = im[B + (m + R / 2) * ST];
    const double sr = ar + br, si = ai + bi;
    br = ar - br;
    bi = ai - bi;
    ar = sr;
    ai = si;
  }
}

// y0, y2 = P +- c u and y1, y3 = Q -+ j c v, the second half of a 4-point DFT
// whose odd inputs' sum and difference are c u and c v.
FFTOC_HD void f64_outputs(double pr, double pi, double qr, double qi, double ur, double ui, double vr, double vi,
                          double c, double (&yr)[4], double (&yi)[4]) {
  yr[0] = fma(c, ur, pr);
  yi[0] = fma(c, ui, pi);
  yr[2] = fma(-c, ur, pr);
  yi[2] = fma(-c, ui, pi);
  yr[1] = fma(c, vi, qr);
  yi[1] = fma(-c, vr, qi);
  yr[3] = fma(-c, vi, qr);
  yi[3] = fma(c, vr, qi);
}

template <int R, int B, int ST, int PP>
FFTOC_HD void f64_finish(double (&re)[PP], double (&im)[PP]) {
  constexpr double H = 0.70710678118654752440, C = 0.92387953251128675613;  // sqrt(1/2), cos(pi/8)
  constexpr double T = 0.41421356237309504880;                              // tan(pi/8)
  if constexpr (R == 4) {
    const double a0r = re[B], a0i = im[B], a1r = re[B + ST], a1i = im[B + ST];
    const double b0r = re[B + 2 * ST], b0i = im[B + 2 * ST], b1r = re[B + 3 * ST], b1i = im[B + 3 * ST];
    re[B] = a0r + a1r; im[B] = a0i + a1i;
    re[B + 2 * ST] = a0r - a1r; im[B + 2 * ST] = a0i - a1i;
    re[B + ST] = b0r + b1i; im[B + ST] = b0i - b1r;
    re[B + 3 * ST] = b0r - b1i; im[B + 3 * ST] = b0i + b1r;
  } else if constexpr (R == 8) {
    double ar[4], ai[4], br[4], bi[4], yr[4], yi[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      ar[m] = re[B + m * ST]; ai[m] = im[B + m * ST];
      br[m] = re[B + (m + 4) * ST]; bi[m] = im[B + (m + 4) * ST];
    }
    dft4_core<EngF64>(ar[0], ai[0], ar[1], ai[1], ar[2], ai[2], ar[3], ai[3], re[B], im[B], re[B + 2 * ST],
                      im[B + 2 * ST], re[B + 4 * ST], im[B + 4 * ST], re[B + 6 * ST], im[B + 6 * ST]);
    // odd outputs: W8^1 b1 = H (1 - j) b1, W8^3 b3 = H (-1 - j) b3
    const double xr = br[1] + bi[1], xi = bi[1] - br[1], zr = bi[3] - br[3], zi = br[3] + bi[3];  // zi: negated
    f64_outputs(br[0] + bi[2], bi[0] - br[2], br[0] - bi[2], bi[0] + br[2], xr + zr, xi - zi, xr - zr, xi + zi, H, yr,
                yi);
#pragma unroll
    for (int q = 0; q < 4; ++q) { re[B + (2 * q + 1) * ST] = yr[q]; im[B + (2 * q + 1) * ST] = yi[q]; }
  } else if constexpr (R == 16) {
    // columns: y[k1][n2], the 4-point DFT over n1 of the inputs n2 + 4 n1
    double yr[4][4], yi[4][4], xr[4][4], xi[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int a = B + n * ST, c = B + (n + 4) * ST, b = B + (n + 8) * ST, d = B + (n + 12) * ST;
      yr[0][n] = re[a] + re[c]; yi[0][n] = im[a] + im[c];
      yr[2][n] = re[a] - re[c]; yi[2][n] = im[a] - im[c];
      yr[1][n] = re[b] + im[d]; yi[1][n] = im[b] - re[d];
      yr[3][n] = re[b] - im[d]; yi[3][n] = im[b] + re[d];
    }
    // rows: the 4-point DFTs over n2 of W16^(n2 k1) y[k1][n2]
    dft4_core<EngF64>(yr[0][0], yi[0][0], yr[0][1], yi[0][1], yr[0][2], yi[0][2], yr[0][3], yi[0][3], xr[0][0],
                      xi[0][0], xr[0][1], xi[0][1], xr[0][2], xi[0][2], xr[0][3], xi[0][3]);
    {  // k1 = 1: W = C (1 - j T), H (1 - j), C (T - j)
      const double sr = yr[1][2] + yi[1][2], si = yi[1][2] - yr[1][2];
      const double er = fma(T, yi[1][1], yr[1][1]), ei = fma(-T, yr[1][1], yi[1][1]);
      const double fr = fma(T, yr[1][3], yi[1][3]), fi = fma(T, yi[1][3], -yr[1][3]);
      f64_outputs(fma(H, sr, yr[1][0]), fma(H, si, yi[1][0]), fma(-H, sr, yr[1][0]), fma(-H, si, yi[1][0]), er + fr,
                  ei + fi, er - fr, ei - fi, C, xr[1], xi[1]);
    }
    {  // k1 = 2: W = H (1 - j), -j, H (-1 - j)
      const double er = yr[2][1] + yi[2][1], ei = yi[2][1] - yr[2][1];
      const double fr = yi[2][3] - yr[2][3], fi = yr[2][3] + yi[2][3];  // fi: negated
      f64_outputs(yr[2][0] + yi[2][2], yi[2][0] - yr[2][2], yr[2][0] - yi[2][2], yi[2][0] + yr[2][2], er + fr, ei - fi,
                  er - fr, ei + fi, H, xr[2], xi[2]);
    }
    {  // k1 = 3: W = C (T - j), H (-1 - j), C (-1 + j T)
      const double sr = yi[3][2] - yr[3][2], si = yr[3][2] + yi[3][2];  // si: negated
      const double er = fma(T, yr[3][1], yi[3][1]), ei = fma(T, yi[3][1], -yr[3][1]);
      const double fr = fma(T, yi[3][3], yr[3][3]), fi = fma(-T, yr[3][3], yi[3][3]);  // both negated
      f64_outputs(fma(H, sr, yr[3][0]), fma(-H, si, yi[3][0]), fma(-H, sr, yr[3][0]), fma(H, si, yi[3][0]), er - fr,
                  ei - fi, er + fr, ei + fi, C, xr[3], xi[3]);
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) {
        re[B + (k1 + 4 * k2) * ST] = xr[k1][k2];
        im[B + (k1 + 4 * k2) * ST] = xi[k1][k2];
      }
  }
}

template <class E, int R, int B, int ST, int PP>
FFTOC_HD void dft(typename E::S (&re)[PP], typename E::S (&im)[PP]) {
  if constexpr (E::kNatural && R == 4) fxn_dft4_at<false, false, false, B, ST, PP>(re, im);
  else if constexpr (E::kNatural && R == 8) fxn_dft8<B, ST, PP>(re, im);
  else if constexpr (E::kNatural && R == 16) fxn_dft16<B, ST, PP>(re, im);
  else if constexpr (E::kId == EngF64::kId && R > 1) {
    f64_sums<R, B, ST, PP>(re, im);
    f64_finish<R, B, ST, PP>(re, im);
  }
  else if constexpr (R == 2) dft2<E, B, ST, PP>(re, im);
  else if constexpr (R == 4) dft4<E, B, ST, PP>(re, im);
  else if constexpr (R == 8) dft8<E, B, ST, PP>(re, im);
  else if constexpr (R == 16) dft16<E, B, ST, PP>(re, im);
}

// ---------------------------------------------------------------------------
// Shared-memory layout: element e of a transform lives at 16-byte slot
// e ^ ((e >> SW) & 7).  Writes of the first pass go at stride R (=2^SW) points
// per thread; the XOR keeps 8 consecutive threads on 8 distinct bank groups.
// ---------------------------------------------------------------------------
template <int SW> FFTOC_HD int swz(int e) { return e ^ ((e >> SW) & 7); }

}  // namespace fftoc
