// Host-side check of the natural-word fixed-point engine (EngFxN, the plans of
// N >= 64), compiled as host code: its products against long double, up to the
// largest magnitudes they take; its 4-, 8- and 16-point DFTs against the DFT
// in long double; and whole plans (the kernel's pass structure over an array)
// at the largest input scale.  Prints "name value" lines.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "fft_kernel.cuh"

using namespace fftoc;
typedef long double ld;
static const ld kPi = 3.141592653589793238462643383279502884L;

static void limbs62(ld v, int* h, int* l) {
  const long long q = llroundl(v * 4611686018427387904.0L);
  *l = (int)(unsigned)q;
  *h = (int)((q - *l) >> 32);
}
static void twiddle(long long k, long long n, int4* w, int2* c) {
  const ld a = cosl(2 * kPi * k / n), b = -sinl(2 * kPi * k / n);
  limbs62(a, &w->x, &w->y);
  limbs62(b - a, &w->z, &w->w);
  limbs62(-a - b, &c->x, &c->y);
}

// A value for a component: random, or an edge (words of all ones and zeros, the
// largest magnitudes).
static long long pick(std::mt19937_64& g, long long lim) {
  switch (g() % 8) {
    case 0: return lim;
    case 1: return -lim;
    case 2: return (lim & ~0xFFFFFFFFLL) | (g() & 1 ? 0x7FFFFFFFLL : 0x80000000LL);
    case 3: return -((lim & ~0xFFFFFFFFLL) | (g() & 1 ? 0x7FFFFFFFLL : 0x80000000LL));
    case 4: return (long long)(g() % 7) - 3;
    default: return (long long)(g() % (2 * (unsigned long long)lim + 1)) - lim;
  }
}

template <bool QUARTER>
static double check_cmul(std::mt19937_64& g) {
  double worst = 0;
  for (int t = 0; t < 400000; ++t) {
    const long long n = 4096, k = t < 4096 ? t : (long long)(g() % n);
    int4 w;
    int2 c;
    twiddle(k, n, &w, &c);
    const ld a = cosl(2 * kPi * k / n), b = -sinl(2 * kPi * k / n);
    long long xr, xi;
    if (t & 1) {  // on the circle of the largest modulus
      const ld top = powl(2, 61.5L), p = 2 * kPi * (ld)(g() >> 11) / 9007199254740992.0L;
      xr = (long long)(top * cosl(p));
      xi = (long long)(top * sinl(p));
    } else {
      xr = pick(g, 1LL << 61);
      xi = pick(g, 1LL << 61);
    }
    const ld f = QUARTER ? 0.25L : 1.0L, er = ((ld)xr * a - (ld)xi * b) * f, ei = ((ld)xr * b + (ld)xi * a) * f;
    EngFxN::cmul<QUARTER>(xr, xi, w, c);
    const double d = (double)fmaxl(fabsl(er - xr), fabsl(ei - xi));
    if (!(d <= worst)) worst = d;
  }
  return worst;
}
static double check_mulh(std::mt19937_64& g) {
  double worst = 0;
  for (int t = 0; t < 400000; ++t) {
    const long long x = pick(g, 1LL << 62);
    const double d = (double)fabsl((ld)x * sqrtl(0.5L) - (ld)EngFxN::mulh(x));
    if (!(d <= worst)) worst = d;
  }
  return worst;
}
static double check_rot8(std::mt19937_64& g) {
  const ld c = cosl(kPi / 8), s = sinl(kPi / 8);
  const long long lim = (long long)(powl(2, 59.5L));  // largest modulus
  double worst = 0;
  for (int t = 0; t < 400000; ++t) {
    long long r, i;
    if (t & 1) {  // on the circle of the largest modulus
      const ld a = 2 * kPi * (ld)(g() >> 11) / 9007199254740992.0L;
      r = (long long)(lim * cosl(a));
      i = (long long)(lim * sinl(a));
    } else {
      r = pick(g, (long long)(powl(2, 59.0L)));
      i = pick(g, (long long)(powl(2, 59.0L)));
    }
    const ld er = c * r + s * i, ei = c * i - s * r;
    EngFxN::rot8(r, i);
    const double d = (double)fmaxl(fabsl(er - r), fabsl(ei - i));
    if (!(d <= worst)) worst = d;
  }
  return worst;
}

template <int R>
static double check_dft(std::mt19937_64& g) {  // worst error of an output, in units of the last place
  double worst = 0;
  const long long lim = 1LL << 55;
  for (int t = 0; t < 20000; ++t) {
    long long re[R], im[R];
    ld xr[R], xi[R];
    for (int i = 0; i < R; ++i) {
      xr[i] = re[i] = pick(g, lim);
      xi[i] = im[i] = pick(g, lim);
    }
    dft<EngFxN, R, 0, 1, R>(re, im);
    for (int k = 0; k < R; ++k) {
      ld sr = 0, si = 0;
      for (int j = 0; j < R; ++j) {
        const ld c = cosl(2 * kPi * (j * k % R) / R), s = -sinl(2 * kPi * (j * k % R) / R);
        sr += xr[j] * c - xi[j] * s;
        si += xr[j] * s + xi[j] * c;
      }
      const double d = (double)fmaxl(fabsl(sr - re[k]), fabsl(si - im[k]));
      if (!(d <= worst)) worst = d;
    }
  }
  return worst;
}

// One butterfly of pass s, with radix R, on an array.
template <int R>
static void one(const long long* xr, const long long* xi, long long* yr, long long* yi, int N, int p, int t, int s,
                bool quarter) {
  long long re[R], im[R];
  const int k = t % p;
  for (int m = 0; m < R; ++m) {
    re[m] = xr[t + m * (N / R)];
    im[m] = xi[t + m * (N / R)];
    if (s == 0) continue;
    if (m == 0) {
      re[0] >>= quarter ? 2 : 0;
      im[0] >>= quarter ? 2 : 0;
    } else {
      int4 w;
      int2 c;
      twiddle((long long)k * m, (long long)R * p, &w, &c);
      if (quarter) EngFxN::cmul<true>(re[m], im[m], w, c);
      else EngFxN::cmul<false>(re[m], im[m], w, c);
    }
  }
  dft<EngFxN, R, 0, 1, R>(re, im);
  for (int m = 0; m < R; ++m) {
    yr[(t - k) * R + k + m * p] = re[m];
    yi[(t - k) * R + k + m * p] = im[m];
  }
}
static void transform(std::vector<long long>& xr, std::vector<long long>& xi, const int* radix, int passes, int quarters) {
  const int N = (int)xr.size();
  std::vector<long long> yr(N), yi(N);
  int p = 1;
  for (int s = 0; s < passes; ++s) {
    for (int t = 0; t < N / radix[s]; ++t) switch (radix[s]) {
        case 2: one<2>(&xr[0], &xi[0], &yr[0], &yi[0], N, p, t, s, s <= quarters); break;
        case 4: one<4>(&xr[0], &xi[0], &yr[0], &yi[0], N, p, t, s, s <= quarters); break;
        case 8: one<8>(&xr[0], &xi[0], &yr[0], &yi[0], N, p, t, s, s <= quarters); break;
        default: one<16>(&xr[0], &xi[0], &yr[0], &yi[0], N, p, t, s, s <= quarters);
      }
    xr.swap(yr);
    xi.swap(yi);
    p *= radix[s];
  }
}
static void fft_ld(std::vector<ld>& r, std::vector<ld>& i) {  // recursive, radix 2
  const size_t n = r.size();
  if (n == 1) return;
  std::vector<ld> ar(n / 2), ai(n / 2), br(n / 2), bi(n / 2);
  for (size_t k = 0; k < n / 2; ++k) {
    ar[k] = r[2 * k]; ai[k] = i[2 * k]; br[k] = r[2 * k + 1]; bi[k] = i[2 * k + 1];
  }
  fft_ld(ar, ai);
  fft_ld(br, bi);
  for (size_t k = 0; k < n / 2; ++k) {
    const ld c = cosl(2 * kPi * k / n), s = -sinl(2 * kPi * k / n);
    const ld tr = br[k] * c - bi[k] * s, ti = br[k] * s + bi[k] * c;
    r[k] = ar[k] + tr; i[k] = ai[k] + ti; r[k + n / 2] = ar[k] - tr; i[k + n / 2] = ai[k] - ti;
  }
}

// Whole plans at the input scale of the kernels (53 bits): random values, every
// component at the largest magnitude, and tones (whose energy meets in one
// output, the largest growth).  Worst error over the transforms, relative to
// the root mean square of the outputs.
static double check_plan(std::mt19937_64& g, const int* radix, int passes) {
  int N = 1;
  for (int s = 0; s < passes; ++s) N *= radix[s];
  const int quarters = N <= 512 ? 0 : N <= 2048 ? 1 : 2;
  const ld down = powl(4, quarters);
  double worst = 0;
  for (int t = 0; t < 6; ++t) {
    std::vector<long long> xr(N), xi(N);
    std::vector<ld> er(N), ei(N);
    const int f = t == 1 ? 0 : t == 2 ? 1 : (int)(g() % N);
    for (int i = 0; i < N; ++i) {
      const ld top = 9007199254740991.0L;  // 2^53 - 1
      ld a, b;
      if (t == 0) {
        a = b = top;
      } else if (t < 4) {  // a tone of the largest modulus: both components full at 45 degrees
        a = roundl(top * sqrtl(2) * cosl(2 * kPi * (ld)((long long)f * i % N) / N + kPi / 4));
        b = roundl(top * sqrtl(2) * sinl(2 * kPi * (ld)((long long)f * i % N) / N + kPi / 4));
        a = fmaxl(-top, fminl(top, a));
        b = fmaxl(-top, fminl(top, b));
      } else {
        a = (long long)(g() >> 10) - (1LL << 53);
        b = (long long)(g() >> 10) - (1LL << 53);
      }
      xr[i] = (long long)a; xi[i] = (long long)b;
      er[i] = a; ei[i] = b;
    }
    transform(xr, xi, radix, passes, quarters);
    fft_ld(er, ei);
    ld num = 0, den = 0;
    for (int i = 0; i < N; ++i) {
      const ld dr = er[i] / down - xr[i], di = ei[i] / down - xi[i];
      num += dr * dr + di * di;
      den += (er[i] * er[i] + ei[i] * ei[i]) / (down * down);
    }
    const double e = (double)sqrtl(num / den);
    if (!(e <= worst)) worst = e;
  }
  return worst;
}

// fx_in_far against fx_in over its domain: normal values from the transform's
// largest exponent (zero distance) to far below it.  Returns the mismatches.
static long long check_in_far(std::mt19937_64& g) {
  long long bad = 0;
  for (int t = 0; t < 1000000; ++t) {
    const int em = 1 + (int)(g() % 2046), below = (int)(g() % (t & 1 ? 70 : 2046));
    const int eref = em + (t % 3 == 0 ? 5 : 0);  // 53 and 48 input bits
    const int e = em - below < 1 ? 1 : em - below;
    const unsigned long long bits = g();
    const unsigned hw = ((unsigned)(bits >> 32) & 0x800FFFFFu) | ((unsigned)e << 20);
    const unsigned lw = t % 5 == 0 ? 0u : (unsigned)bits;
    if (fx_in_far(hw, lw, eref) != fx_in<false>(hw, lw, eref)) ++bad;
  }
  return bad;
}

int main() {
  std::mt19937_64 g(20240607);
  printf("in_far_mismatch %lld\n", check_in_far(g));
  printf("cmul_quarter_units %.4f\n", check_cmul<true>(g));
  printf("cmul_units %.4f\n", check_cmul<false>(g));
  printf("mulh_units %.4f\n", check_mulh(g));
  printf("rot8_units %.4f\n", check_rot8(g));
  printf("dft2_units %.4f\n", check_dft<2>(g));
  printf("dft4_units %.4f\n", check_dft<4>(g));
  printf("dft8_units %.4f\n", check_dft<8>(g));
  printf("dft16_units %.4f\n", check_dft<16>(g));
  const int plans[][4] = {{8, 8}, {16, 4}, {16, 8}, {8, 8, 2}, {16, 16}, {8, 8, 4}, {8, 8, 8}, {16, 16, 2}, {16, 16, 4},
                          {8, 8, 8, 2}, {16, 8, 8}, {16, 16, 8}, {8, 8, 8, 4}, {16, 16, 16}, {8, 8, 8, 8}};
  double worst = 0;
  for (const int* r : plans) {
    int s = 0;
    while (s < 4 && r[s] > 1) ++s;
    const double e = check_plan(g, r, s);
    if (!(e <= worst)) worst = e;
    fprintf(stderr, "%d %d %d %d: %.3e\n", r[0], r[1], r[2], r[3], e);
  }
  printf("plans_rel %.3e\n", worst);
  return 0;
}
